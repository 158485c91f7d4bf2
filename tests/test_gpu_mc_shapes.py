"""Langevin + Metropolis steps at the edges of the Metropolis kernel's shapes: the
shared-memory sizes (32, 64, 128 residues), the 16- and the 8-warp instances, and an
interface cutoff that reaches beyond the residues' lists.  Bit for bit against the CPU
oracle, as tests/test_gpu_mc.py (the default accumulation's decisions could only differ
where u lands within ~1e-15 of exp(-dE/T))."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STEPS = [0, 1, 2, 3, 4]


@pytest.mark.parametrize("acc", [0, 1])
@pytest.mark.parametrize("n_res,n_cand,iface_sq", [(1, 5, 64.0), (2, 149, 64.0), (31, 4, 400.0), (32, 149, 64.0),
                                                   (33, 3, 64.0), (64, 3, 400.0), (64, 149, 64.0), (65, 2, 64.0),
                                                   (127, 2, 64.0), (128, 2, 64.0)])
def test_mc_shapes_bit_exact(ctx, oracle, pkg, acc, n_res, n_cand, iface_sq):
    cfg = pkg.workloads.config1(n_cand=max(1, (n_cand * n_res + 19) // 20))
    ag_aa, ag_ca = cfg["antigens"][0]
    ag_pos, _ = oracle.build_residues(ag_ca, ag_aa)
    kw = dict(shell_radius=cfg["shell"][0], seed=77, accumulate=acc, mutation_p=0.3, rotamer_move_p=0.5,
              backbone_move_p=0.15, iface_cutoff_sq=iface_sq)
    ctx.clear_antigens()
    ctx.set_params(pkg.Params.defaults(**kw))
    ctx.add_antigen(ag_aa, ag_pos)
    A = oracle.Antigen(ag_aa, ag_pos)
    op = oracle.OrcParams.defaults(**kw)
    total = n_cand * n_res
    aa = cfg["pop"].aa[:total].copy()
    aa[::9] = pkg.ONE_LETTER.index("C")  # several Cys per candidate: the ordered part of the sweep
    pos, chi = oracle.build_residues(cfg["pop"].ca[:total], aa)
    cid = np.arange(n_cand, dtype=np.uint32) * 3 + 1
    temps = np.array([oracle.temperature(s * 100, 600) for s in STEPS], np.float32)
    ctx.state_upload(aa, chi, pos, uniform_n_res=n_res, cand_id=cid)
    ctx.diffuse(len(STEPS), step0=0, with_noise=True, with_mc=True, temps=temps)
    g_aa, g_chi, g_pos = ctx.state_download()
    g_stats = ctx.mc_stats()
    o_stats = np.zeros((n_cand, 4), np.int64)
    for s, t in zip(STEPS, temps):
        A.step(op, aa, chi, pos, n_res, cid, s, t, True, True, stats=o_stats)
    assert o_stats[:, 0].sum() + o_stats[:, 2].sum() > 0
    assert np.array_equal(g_stats, o_stats)
    assert np.array_equal(g_aa, aa)
    assert np.array_equal(g_chi, chi)
    assert np.array_equal(g_pos, pos)
