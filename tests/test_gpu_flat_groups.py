"""score_batch over flat atoms where the kernel's groups change shape: candidates of 1, 14,
15, 255, 256, 257 and 600 atoms (the group's and the chunk's edges), atoms all in one spot
or all far apart, uniform and ragged calls alike, against the f64 oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spread", [0.0, 1.0, 12.0])
@pytest.mark.parametrize("n_ab", [1, 14, 15, 255, 256, 257, 600])
def test_flat_groups(ctx, oracle, pkg, n_ab, spread):
    """1e-5 of the sum of the terms' sizes: f32 pair terms (a few 2^-24 each), compensated sums."""
    W = pkg.workloads
    rng = np.random.default_rng(n_ab)
    ag_aa, ag_ca, radius = W._globule_antigen(60, W.rng_for(3))
    ag_pos, _ = oracle.build_residues(ag_ca, ag_aa)
    antigen = pkg.AtomCloud.from_slots(ag_aa, ag_pos)
    n_cand = 3
    at = np.zeros(n_cand * n_ab, pkg.GPU_ATOM)
    xyz = W.sphere_points(1, radius + 3.0, np.zeros(3), rng) + rng.uniform(-1, 1, (n_cand * n_ab, 3)) * spread
    at["x"], at["y"], at["z"] = xyz.T.astype(np.float32)
    at["q"] = rng.uniform(-0.8, 0.8, n_cand * n_ab)
    at["r_min_half"], at["epsilon"] = 1.9, 0.1
    at["hydrophobic"] = rng.integers(0, 2, n_cand * n_ab)
    off = np.arange(n_cand + 1, dtype=np.int64) * n_ab
    e, size = ctx.score_batch_f64(antigen, at, n_ab, with_abs=True)
    want = oracle.score_batch64(antigen.to_gpu_atoms(), at, off)
    assert np.all(np.abs(e - want) <= 1e-5 * size + 1e-9)
    assert np.array_equal(ctx.score_batch_ragged(antigen, at, off, with_abs=True)[0], e)
    plain = ctx.score_batch_f64(antigen, at, n_ab)  # the instance without the terms' sizes
    assert np.all(np.abs(plain - want) <= 1e-5 * size + 1e-9)
    assert np.array_equal(ctx.score_batch_ragged(antigen, at, off), plain)
    assert np.array_equal(ctx.score_batch(antigen, at, n_ab), plain.astype(np.float32))
    f, ef = ctx.forces_allatom(antigen, at, off)
    assert np.all(np.abs(ef - want) <= 1e-5 * size + 1e-9) and np.all(np.isfinite(f))
