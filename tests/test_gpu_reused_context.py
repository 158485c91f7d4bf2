"""What one call leaves in a context (lists, work bands, buffers) does not show in the next:
the same calls in a fresh context give the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _antigens(pkg, ctx):
    W = pkg.workloads
    for n in (60, 300):
        aa, ca, _ = W._globule_antigen(n, W.rng_for(n))
        ctx.add_antigen(aa, ctx.build_residues(ca, aa)[0])


@pytest.mark.parametrize("lane_groups", [False, True])
def test_gradient_steps_on_lists_of_fv_steps(pkg, lane_groups):
    """The Fv steps leave lists with skins up to 8 A, wider than the gradient steps build."""
    W = pkg.workloads
    got = []
    with pkg.GpuContext.create(0) as ctx:
        if lane_groups:
            ctx.set_launch_cfg()
        _antigens(pkg, ctx)
        _, ag_ca, _ = W._globule_antigen(300, W.rng_for(300))
        fv = W.config_fv(ag_ca, n_cand=3, seed=4)
        chains = []
        for c in ("heavy", "light"):
            aa, ca, cdr = fv[c]
            pos, chi = ctx.build_residues(ca, aa)
            chains.append((aa, chi, pos, (cdr > 0).astype(np.uint8)))
        ctx.set_params(pkg.Params.defaults(shell_radius=fv["target_radius"], backbone_move_p=0.2))
        ctx.fv_upload(*chains, antigen_id=1, cand_id=np.arange(3, dtype=np.uint32))
        ctx.fv_run(4)
        start = ctx.state_download()
        ctx.diffuse(6)
        got.append(ctx.state_download())
        ctx.diffuse(6, step0=6, with_noise=True)
        got.append(ctx.state_download())
    n_h, n_l = (len(c[0]) // 3 for c in chains)
    n_res = np.tile(np.int32([n_h, n_l]), 3)
    ids = np.repeat(np.arange(3, dtype=np.uint32), 2)
    with pkg.GpuContext.create(0) as ctx:
        if lane_groups:
            ctx.set_launch_cfg()
        _antigens(pkg, ctx)
        ctx.set_params(pkg.Params.defaults(shell_radius=fv["target_radius"], backbone_move_p=0.2))
        ctx.state_upload(*start, n_res=n_res, antigen_id=np.ones(6, np.int32), cand_id=ids)
        for k, noise in ((0, False), (6, True)):
            ctx.diffuse(6, step0=k, with_noise=noise)
            for a, b in zip(ctx.state_download(), got[k // 6]):
                assert np.array_equal(a, b)


def test_states_of_other_shapes(pkg):
    """States that grow, shrink and keep their residue count with other candidates."""
    W = pkg.workloads
    shapes = [(40, 20), (25, 12), (80, 10), (20, 40), (3, 1), (40, 20)]  # 800, 300, 800, 800, 3, 800 residues

    def one(ctx, i):
        n_cand, n_res = shapes[i]
        r = np.random.default_rng(100 + i)
        aa = W.random_sequence(n_cand * n_res, r)
        pos, chi = ctx.build_residues(W.sphere_points(n_cand * n_res, 22.0, np.zeros(3), r), aa)
        ctx.state_upload(aa, chi, pos, uniform_n_res=n_res, antigen_id=(np.arange(n_cand) % 2).astype(np.int32))
        first = ctx.score_state()
        e, top = ctx.block(10, 0, k=3, n_segments=2)
        ctx.diffuse(3, 10, with_noise=True, with_mc=True)
        return (first, e, top, ctx.score_state(full=True), ctx.mc_energy()) + ctx.state_download()

    with pkg.GpuContext.create(0) as used:
        _antigens(pkg, used)
        for i in range(len(shapes)):
            a = one(used, i)
            with pkg.GpuContext.create(0) as fresh:
                _antigens(pkg, fresh)
                for x, y in zip(a, one(fresh, i)):
                    assert np.array_equal(x, y), i


@pytest.mark.parametrize("n_cand,n_res", [(4, 5), (130, 20)])
def test_full_energy_by_slabs(ctx, oracle, pkg, n_cand, n_res):
    """The resident state's energies against an antigen of more than 128 blocks of 32 atoms
    in a long box, whose groups look at their x-slab of the grid only: warp teams and single
    warps, candidates inside, at the ends and out of reach.  1e-5 of the sum of the terms'
    sizes: f32 pair terms (a few 2^-24 each), compensated sums."""
    W = pkg.workloads
    rng = np.random.default_rng(17)
    half = np.array([90.0, 14.0, 14.0])
    ag_aa = W.random_sequence(900, rng)
    ag_pos, _ = oracle.build_residues(rng.uniform(-half, half, (900, 3)).astype(np.float32), ag_aa)
    assert pkg.tables().n_atoms[ag_aa].sum() > 4096
    aa = W.random_sequence(n_cand * n_res, rng)
    ca = rng.uniform(-half - 12, half + 12, (n_cand * n_res, 3)).astype(np.float32)
    ca[0] = (140.0, 0.0, 0.0)
    ca[1] = (-140.0, 0.0, 0.0)
    pos, chi = oracle.build_residues(ca, aa)
    ctx.clear_antigens()
    ctx.set_params(pkg.Params.defaults())
    ctx.add_antigen(ag_aa, ag_pos)
    ctx.state_upload(aa, chi, pos, uniform_n_res=n_res)
    A = oracle.Antigen(ag_aa, ag_pos)
    for full in (False, True):
        got = ctx.score_state(full=full)
        want, scale = A.score_slots64(aa, pos, n_res, full=full, with_abs=True)
        assert np.all(np.abs(got - want) <= 1e-5 * scale + 1e-9)
