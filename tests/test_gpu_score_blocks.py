"""The score kernels' walk over the antigen's blocks of 32 atoms: antigens at the edges of a
block and of the rule that starts from the group's x-slab (128 blocks), candidates deep in,
at the rim and out of reach on every side, against the f64 oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_ag", [1, 31, 32, 33, 4095, 4096, 4097, 9000])
def test_antigen_blocks(ctx, oracle, pkg, n_ag):
    """1e-5 of the sum of the terms' sizes: f32 pair terms (a few 2^-24 each), compensated sums."""
    rng = np.random.default_rng(n_ag)
    half = np.array([60.0, 9.0, 9.0])  # a long box: slabs of the grid leave most of it out

    def atoms(n, xyz):
        at = np.zeros(n, pkg.GPU_ATOM)
        at["x"], at["y"], at["z"] = xyz.T.astype(np.float32)
        at["q"] = rng.uniform(-0.8, 0.8, n)
        at["r_min_half"], at["epsilon"] = 1.9, 0.1
        at["hydrophobic"] = rng.integers(0, 2, n)
        return at

    ag = atoms(n_ag, rng.uniform(-half, half, (n_ag, 3)))
    antigen = pkg.AtomCloud(ag["x"], ag["y"], ag["z"], ag["q"], ag["r_min_half"], ag["epsilon"],
                            ag["hydrophobic"].astype(np.uint8))
    centres = np.array([[0, 0, 0], [55, 8, 0], [-68, 0, 3], [68, -5, 0], [90, 0, 0], [-90, 0, 0], [0, 40, 0], [20, 0, -17]], float)
    at = atoms(8 * 10, np.repeat(centres, 10, 0) + rng.uniform(-2.0, 2.0, (80, 3)))
    off = np.arange(9, dtype=np.int64) * 10
    e, size = ctx.score_batch_f64(antigen, at, 10, with_abs=True)
    want = oracle.score_batch64(antigen.to_gpu_atoms(), at, off)
    assert np.all(np.abs(e - want) <= 1e-5 * size + 1e-9)
    assert np.all(e[4:7] == 0.0) and (n_ag < 4000 or np.all(e[:4] != 0.0))
