"""Metropolis launches that take over the residues' lists of earlier launches (their own and
the gradient steps') follow the same trajectory, bit for bit, as launches that build every
list anew: an antigen added between the calls makes all kept lists stale."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_ag,radius,n_res,n_cand", [(300, 22.0, 20, 8), (300, 22.0, 40, 3), (400, 11.0, 12, 150)])
def test_kept_lists(pkg, n_ag, radius, n_res, n_cand):
    """(400 residues in 11 A: lists that overflow with any wide skin.)"""
    W = pkg.workloads
    got = []
    for stale in (False, True):
        rng = W.rng_for(40)
        d = rng.normal(size=(n_ag, 3))
        d *= radius * (rng.random((n_ag, 1)) ** (1 / 3)) / np.linalg.norm(d, axis=1, keepdims=True)
        ag_aa, ag_ca = W.random_sequence(n_ag, rng), d.astype(np.float32)
        aa = W.random_sequence(n_cand * n_res, rng)
        ca = W.sphere_points(n_cand * n_res, radius + 2.0, np.zeros(3), rng)
        with pkg.GpuContext.create(0, pkg.Params.defaults(shell_radius=radius, backbone_move_p=0.2, seed=9)) as ctx:
            ag_pos = ctx.build_residues(ag_ca, ag_aa)[0]
            ctx.add_antigen(ag_aa, ag_pos)
            pos, chi = ctx.build_residues(ca, aa)
            ctx.state_upload(aa, chi, pos, uniform_n_res=n_res)
            for call in range(4):
                if stale:
                    ctx.add_antigen(ag_aa[:5], ag_pos[:5])
                mc = call != 1
                ctx.diffuse(3, step0=3 * call, with_noise=mc, with_mc=mc, temps=np.full(3, 1.5, np.float32))
            got.append(ctx.state_download() + (ctx.mc_stats(),))
    for a, b in zip(*got):
        assert np.array_equal(a, b)
