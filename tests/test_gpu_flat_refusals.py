"""A flat call that is refused or fails leaves the context as it was: the last scored batch
stays what binder_last_pair_count counts, or there is none."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

OOM, NAN, GRID, STATE = 3, 5, 6, 7


def _cloud(pkg, ctx, n_res, seed):
    W = pkg.workloads
    rng = W.rng_for(seed)
    aa, ca, _ = W._globule_antigen(n_res, rng)
    return pkg.AtomCloud.from_slots(aa, ctx.build_residues(ca, aa)[0])


def _batch(cloud, n_cand, n_ab, seed):
    rng = np.random.default_rng(seed)
    a = cloud.to_gpu_atoms()[rng.integers(0, len(cloud), n_cand * n_ab)]
    for k in "xyz":
        a[k] += rng.normal(scale=3.0, size=len(a)).astype(np.float32)
    return a, np.arange(n_cand + 1, dtype=np.int64) * n_ab


def _call(ctx, kind, ag, atoms, off):
    if kind == "uniform":
        return ctx.score_batch_f64(ag, atoms, int(off[1]))
    if kind == "ragged":
        return ctx.score_batch_ragged(ag, atoms, off)
    return ctx.forces_allatom(ag, atoms, off)[1]


def _set_antigen(pkg, ctx, ag):
    c = ag._c()
    assert pkg.lib().binder_set_antigen_atoms(ctx._h, C.byref(c)) == 0


@pytest.mark.parametrize("kind", ["uniform", "ragged", "forces"])
@pytest.mark.parametrize("first", ["uniform", "ragged"])
@pytest.mark.parametrize("bad", ["nan", "box"])
def test_refused_antigen(pkg, first, kind, bad):
    with pkg.GpuContext.create(0) as ctx:
        good = _cloud(pkg, ctx, 30, 1)
        atoms, off = _batch(good, 6, 11, 2)
        e = _call(ctx, first, good, atoms, off)
        pairs = ctx.last_pair_count()
        wrong = _cloud(pkg, ctx, 30, 3)
        wrong.x = wrong.x.copy()
        wrong.x[4] = np.nan if bad == "nan" else 1e8
        if bad == "box":
            wrong.y = wrong.y.copy()
            wrong.y[5] = -1e8
        others, o_off = _batch(good, 9, 17, 4)
        with pytest.raises(pkg.BinderError) as ei:
            _call(ctx, kind, wrong, others, o_off)
        assert ei.value.status == (NAN if bad == "nan" else GRID)
        with pytest.raises(pkg.BinderError) as ei:  # no antigen
            ctx.last_pair_count()
        assert ei.value.status == STATE
        _set_antigen(pkg, ctx, good)
        assert ctx.last_pair_count() == pairs
        assert np.array_equal(_call(ctx, first, good, atoms, off), e)


@pytest.mark.parametrize("kind", ["uniform", "ragged", "forces"])
@pytest.mark.parametrize("same_antigen", [True, False])
def test_failed_allocation(pkg, kind, same_antigen):
    """Each device allocation of a larger call fails in turn: no batch to count afterwards
    unless the earlier one is untouched, and the call works when repeated."""
    L = pkg.lib()
    failed = 0
    try:
        for k in range(64):
            with pkg.GpuContext.create(0) as ctx:
                good = _cloud(pkg, ctx, 30, 1)
                ag = good if same_antigen else _cloud(pkg, ctx, 60, 3)
                atoms, off = _batch(good, 6, 11, 2)
                more, m_off = _batch(good, 900, 17, 4)
                want = _call(ctx, kind, ag, more[:17], m_off[:2])[0]
                _call(ctx, "uniform", good, atoms, off)
                pairs = ctx.last_pair_count()
                L.binder_debug_fail_alloc(k)
                try:
                    e = _call(ctx, kind, ag, more, m_off)
                except pkg.BinderError as err:
                    assert err.status == OOM
                    failed += 1
                    L.binder_debug_fail_alloc(-1)
                    _set_antigen(pkg, ctx, good)
                    try:
                        assert ctx.last_pair_count() == pairs
                    except pkg.BinderError as err:
                        assert err.status == STATE
                    assert _call(ctx, kind, ag, more, m_off)[0] == want
                else:
                    L.binder_debug_fail_alloc(-1)
                    assert e[0] == want
                    break
    finally:
        L.binder_debug_fail_alloc(-1)
    assert 1 <= failed < 63
