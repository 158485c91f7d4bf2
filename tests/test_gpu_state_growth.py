"""A selection that repeats candidates makes the state larger than its upload: every
per-residue buffer (the Verlet lists among them) has to grow with it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _population(pkg, ctx, n_cand, n_res, seed=31):
    W = pkg.workloads
    rng = W.rng_for(seed)
    ag_aa, ag_ca, _ = W._globule_antigen(80, rng)
    ctx.add_antigen(ag_aa, ctx.build_residues(ag_ca, ag_aa)[0])
    aa = W.random_sequence(n_cand * n_res, rng)
    pos, chi = ctx.build_residues(W.sphere_points(n_cand * n_res, 18.0, np.zeros(3), rng), aa)
    return aa, chi, pos


@pytest.mark.parametrize("lane_groups", [False, True])
@pytest.mark.parametrize("n_cand,n_res,copies", [(3, 7, 5), (8, 20, 64), (2, 40, 9)])
def test_growing_selection(pkg, n_cand, n_res, copies, lane_groups):
    """Metropolis and gradient steps (launches that keep the residues' lists for the next
    one) on a selection of many copies, bit for bit those of a fresh upload of the same
    residues with the same candidate ids."""
    idx = (np.arange(copies) * 7 + 1) % n_cand
    got = []
    for select in (True, False):
        with pkg.GpuContext.create(0, pkg.Params.defaults(shell_radius=18.0, seed=4, backbone_move_p=0.1)) as ctx:
            if lane_groups:
                ctx.set_launch_cfg()
            aa, chi, pos = _population(pkg, ctx, n_cand, n_res)
            if select:
                ctx.state_upload(aa, chi, pos, uniform_n_res=n_res)
                ctx.state_select(idx)
            else:
                r = (idx[:, None] * n_res + np.arange(n_res)).ravel()
                ctx.state_upload(aa[r], chi[r], pos[r], uniform_n_res=n_res, cand_id=idx)
            for call in range(4):
                mc = call != 1
                ctx.diffuse(4, step0=4 * call, with_noise=mc, with_mc=mc, temps=np.full(4, 1.5, np.float32))
            e, top = ctx.block(10, 0, k=min(8, copies))
            got.append(ctx.state_download() + (ctx.mc_stats(), e, top))
    for a, b in zip(*got):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("grow", ["upload", "select"])
def test_no_state_without_its_buffers(pkg, grow):
    """An allocation that fails while the state grows leaves either the old state or none:
    the calls that follow are refused, and a later upload works."""
    L = pkg.lib()
    failed = 0
    try:
        for k in range(64):
            with pkg.GpuContext.create(0, pkg.Params.defaults(shell_radius=18.0)) as ctx:
                aa, chi, pos = _population(pkg, ctx, 12, 5)
                ctx.state_upload(aa[:15], chi[:15], pos[:15], uniform_n_res=5)
                ctx.diffuse(2)
                L.binder_debug_fail_alloc(k)
                try:
                    if grow == "upload":
                        ctx.state_upload(aa, chi, pos, uniform_n_res=5)
                    else:
                        ctx.state_select(np.arange(12) % 3)
                except pkg.BinderError as e:
                    assert e.status == 3  # BINDER_ERR_OOM
                    failed += 1
                    L.binder_debug_fail_alloc(-1)
                    assert ctx.state_info()[0] in ((0,) if grow == "upload" else (0, 3))
                    if ctx.state_info()[0] == 0:
                        for call in (lambda: ctx.diffuse(2), lambda: ctx.diffuse(2, with_mc=True), ctx.score_state,
                                     ctx.state_download, lambda: ctx.state_select([0])):
                            with pytest.raises(pkg.BinderError) as ei:
                                call()
                            assert ei.value.status == 7  # BINDER_ERR_STATE
                    ctx.state_upload(aa, chi, pos, uniform_n_res=5)
                    assert np.array_equal(ctx.state_download()[2], pos)
                    ctx.diffuse(2)
                else:
                    L.binder_debug_fail_alloc(-1)
                    break
    finally:
        L.binder_debug_fail_alloc(-1)
    assert failed >= (5 if grow == "upload" else 10) and failed < 63
