"""An enqueued block's pending selection is not left behind on a buffer that a failed
allocation of the next block has released."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_allocation_failure_with_a_selection_pending(pkg):
    W = pkg.workloads
    L = pkg.lib()
    rng = W.rng_for(12)
    try:
        with pkg.GpuContext.create(0, pkg.Params.defaults(shell_radius=18.0)) as ctx:
            ag_aa, ag_ca, _ = W._globule_antigen(60, rng)
            ctx.add_antigen(ag_aa, ctx.build_residues(ag_ca, ag_aa)[0])
            aa = W.random_sequence(100 * 6, rng)
            pos, chi = ctx.build_residues(W.sphere_points(600, 16.0, np.zeros(3), rng), aa)
            ctx.state_upload(aa, chi, pos, uniform_n_res=6)
            want = ctx.block(5, 0, k=50)
            ctx.state_upload(aa, chi, pos, uniform_n_res=6)
            ctx.block_async(5, 0, k=4)
            L.binder_debug_fail_alloc(0)
            with pytest.raises(pkg.BinderError) as ei:
                ctx.block_async(5, 5, k=64)
            assert ei.value.status == 3  # BINDER_ERR_OOM
            L.binder_debug_fail_alloc(-1)
            ctx.synchronize()
            assert np.array_equal(ctx.score_state(), want[0])
            ctx.state_upload(aa, chi, pos, uniform_n_res=6)
            e, top = ctx.block(5, 0, k=50)
            assert np.array_equal(e, want[0]) and np.array_equal(top, want[1])
    finally:
        L.binder_debug_fail_alloc(-1)
