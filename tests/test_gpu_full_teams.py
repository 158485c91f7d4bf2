"""The full all-atom energy of the resident state against the f64 oracle where the scoring
kernel's warp teams change shape (populations on both sides of the team rule, candidates
of one residue, a dense antigen whose residues queue several segments of atoms), and the
division by a constant that the energy uses."""
import ctypes

import numpy as np
import pytest


def _dense(W, n, radius, seed):
    rng = W.rng_for(seed)
    d = rng.normal(size=(n, 3))
    d *= radius * (rng.random((n, 1)) ** (1 / 3)) / np.linalg.norm(d, axis=1, keepdims=True)
    return W.random_sequence(n, rng), d.astype(np.float32)


@pytest.mark.gpu
@pytest.mark.parametrize("n_ag,radius,n_cand,n_res", [(300, 22.0, 3, 1), (300, 22.0, 64, 20), (300, 22.0, 118, 20),
                                                      (300, 22.0, 119, 20), (900, 9.0, 4, 5)])
def test_full_energy_teams(ctx, oracle, pkg, n_ag, radius, n_cand, n_res):
    """1e-5 of the sum of the terms' sizes: f32 pair terms (a few 2^-24 each), compensated
    sums."""
    W = pkg.workloads
    ag_aa, ag_ca = _dense(W, n_ag, radius, 11)
    ag_pos, _ = oracle.build_residues(ag_ca, ag_aa)
    rng = np.random.default_rng(5)
    aa = W.random_sequence(n_cand * n_res, rng)
    pos, chi = oracle.build_residues(W.sphere_points(n_cand * n_res, radius + 4.0, np.zeros(3), rng), aa)
    ctx.clear_antigens()
    ctx.add_antigen(ag_aa, ag_pos)
    ctx.state_upload(aa, chi, pos, uniform_n_res=n_res)
    got = ctx.score_state(full=True)
    A = oracle.Antigen(ag_aa, ag_pos)
    want, scale = A.score_slots64(aa, pos, n_res, full=True, with_abs=True)
    assert np.array_equal(got, ctx.score_state(full=True))
    assert np.all(np.abs(got - want) <= 1e-5 * scale + 1e-9)


def test_constant_division_is_exact():
    """div_by of csrc/score.cuh (q = r y, one correction by the exact remainder) equals the
    IEEE quotient for its divisors, on random and edge floats of the range it is used in."""
    m = ctypes.CDLL("libm.so.6")
    m.fmaf.restype, m.fmaf.argtypes = ctypes.c_float, [ctypes.c_float] * 3
    rng = np.random.default_rng(1)
    r = np.concatenate([np.exp(rng.uniform(np.log(1e-7), np.log(15.9), 4000)), [0.5, 9.0, 2.9, 1.0, 0.25]]).astype(np.float32)
    for d in np.float32([3.15, 3.5, 3.7, 3.9, 0.35]):
        y = np.float32(1.0) / d
        for x in r:
            q = x * y
            got = np.float32(m.fmaf(m.fmaf(-float(d), float(q), float(x)), float(y), float(q)))
            assert got == x / d
