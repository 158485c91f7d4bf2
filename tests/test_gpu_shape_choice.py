"""Launch shapes follow the state's size until the caller sets or tunes them, and then stay."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SMALL = dict(score_warps=16, score_ctas_per_sm=2, cg_warps=4, cg_lanes=8, cg_order=3, score_order=1, cg_queue=0, cg_flat=4)
MIDDLE = dict(SMALL, cg_flat=8)
LARGE = dict(MIDDLE, cg_warps=8, cg_queue=1)


def _upload(pkg, ctx, total):
    """One residue per candidate, as many as asked."""
    aa = np.zeros(total, np.uint8)
    ca = np.zeros((total, 3), np.float32)
    ca[:, 0] = 15.0
    pos, chi = ctx.build_residues(ca, aa)
    ctx.state_upload(aa, chi, pos, uniform_n_res=1)


def _context(pkg):
    ctx = pkg.GpuContext.create(0, pkg.Params.defaults(shell_radius=15.0))
    W = pkg.workloads
    aa, ca, _ = W._globule_antigen(40, W.rng_for(2))
    ctx.add_antigen(aa, ctx.build_residues(ca, aa)[0])
    return ctx


def test_shape_by_size(pkg):
    with _context(pkg) as ctx:
        for total, want in ((1, SMALL), (4095, SMALL), (4096, MIDDLE), (32767, MIDDLE), (32768, LARGE), (7, SMALL)):
            _upload(pkg, ctx, total)
            assert ctx.launch_cfg().as_dict() == want, total
        ctx.state_select(np.zeros(4096, np.int32))
        assert ctx.launch_cfg().as_dict() == MIDDLE


@pytest.mark.parametrize("how", ["set", "tune"])
def test_chosen_shape_stays(pkg, how):
    with _context(pkg) as ctx:
        _upload(pkg, ctx, 64)
        if how == "set":
            ctx.set_launch_cfg(score_warps=4, cg_warps=2)
        else:
            ctx.autotune(reps=1)
        chosen = ctx.launch_cfg().as_dict()
        for total in (5000, 40000, 3):
            _upload(pkg, ctx, total)
            assert ctx.launch_cfg().as_dict() == chosen
