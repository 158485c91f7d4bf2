"""The launch shapes picked by the state's size give the trajectories and energies of an
explicit shape bit for bit, on both sides of each size limit and for a population that
grows and shrinks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_cand,n_res", [(1, 1), (204, 20), (205, 20), (1638, 20), (1639, 20)])
def test_default_shapes(pkg, n_cand, n_res):
    W = pkg.workloads
    rng = np.random.default_rng(n_cand)
    got = []
    for explicit in (False, True):
        with pkg.GpuContext.create(0, pkg.Params.defaults(shell_radius=26.0)) as ctx:
            if explicit:
                ctx.set_launch_cfg()  # the lane-group form
            ags = [W._globule_antigen(n, W.rng_for(21 + n)) for n in (60, 90)]
            for aa, ca, _ in ags:
                ctx.add_antigen(aa, ctx.build_residues(ca, aa)[0])
            rng = np.random.default_rng(n_cand)
            aa = W.random_sequence(n_cand * n_res, rng)
            pos, chi = ctx.build_residues(W.sphere_points(n_cand * n_res, 18.0, np.zeros(3), rng), aa)
            agid = (np.arange(n_cand) % 2).astype(np.int32)
            for cands in (min(3, n_cand), n_cand):
                m = cands * n_res
                ctx.state_upload(aa[:m], chi[:m], pos[:m], uniform_n_res=n_res, antigen_id=agid[:cands])
                for b in range(3):
                    e, top = ctx.block(10, 10 * b, k=min(8, cands), n_segments=2)
            shape = ctx.launch_cfg().as_dict()
            got.append((e, top, ctx.state_download()[2]))
    assert shape["cg_flat"] == 0
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])
    assert np.array_equal(got[0][2], got[1][2])
