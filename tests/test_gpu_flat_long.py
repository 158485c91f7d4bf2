"""score_batch over flat atoms whose groups are cut in two (atoms in a row without a gap,
longer than any residue) or not cut at gaps (scattered atoms against a small antigen), at the
edges of both rules, against the f64 oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _atoms(pkg, rng, xyz):
    at = np.zeros(len(xyz), pkg.GPU_ATOM)
    at["x"], at["y"], at["z"] = xyz.T.astype(np.float32)
    at["q"] = rng.uniform(-0.8, 0.8, len(xyz))
    at["r_min_half"], at["epsilon"] = 1.9, 0.1
    at["hydrophobic"] = rng.integers(0, 2, len(xyz))
    return at


@pytest.mark.parametrize("kind", ["line", "bent", "scattered", "half"])
@pytest.mark.parametrize("n_ag", [1, 640, 641, 3000])
@pytest.mark.parametrize("n_ab", [1, 7, 8, 14, 15, 256, 263, 300])
def test_long_and_scattered_groups(ctx, oracle, pkg, n_ab, n_ag, kind):
    """1e-5 of the sum of the terms' sizes: f32 pair terms (a few 2^-24 each), compensated sums."""
    rng = np.random.default_rng(n_ab + n_ag)
    half = 4.0 * n_ag ** (1.0 / 3.0)
    ag = _atoms(pkg, rng, rng.uniform(-half, half, (n_ag, 3)))
    antigen = pkg.AtomCloud(ag["x"], ag["y"], ag["z"], ag["q"], ag["r_min_half"], ag["epsilon"],
                            ag["hydrophobic"].astype(np.uint8))
    n_cand = 3
    i = np.arange(n_ab)
    if kind == "line":      # 14 atoms reach over 12 A from the 5th on
        one = np.stack([3.8 * i - 1.9 * n_ab, 0 * i, 0 * i], 1)
    elif kind == "bent":    # the 14th atom alone lies at 12 A from the first
        one = np.stack([12.0 / 13.0 * i - 6.0 / 13.0 * n_ab, 0 * i, 0 * i], 1)
    elif kind == "half":    # residue-like runs of 4 atoms, on the edge of the rule's count
        one = np.stack([9.0 * (i // 4), 1.2 * (i % 4), 0 * i], 1) - [4.5 * (n_ab // 4), 0, 0]
    else:
        one = rng.uniform(-half - 8, half + 8, (n_ab, 3))
    xyz = (one[None] + rng.uniform(-2, 2, (n_cand, 1, 3))).reshape(-1, 3)
    at = _atoms(pkg, rng, xyz)
    off = np.arange(n_cand + 1, dtype=np.int64) * n_ab
    want = oracle.score_batch64(antigen.to_gpu_atoms(), at, off)
    e, size = ctx.score_batch_f64(antigen, at, n_ab, with_abs=True)
    assert np.all(np.abs(e - want) <= 1e-5 * size + 1e-9)
    plain = ctx.score_batch_ragged(antigen, at, off)
    assert np.all(np.abs(plain - want) <= 1e-5 * size + 1e-9)
    assert ctx.last_pair_count() == oracle.count_pairs(antigen.to_gpu_atoms(), at)
