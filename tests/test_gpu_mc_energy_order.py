"""The double Metropolis energy of a residue is a function of its Calpha, its amino acid and
the antigen alone, bit for bit: not of the residues evaluated beside it, nor of whether its
antigen Calphas come from a list, a scan, or unstaged memory.

Calphas half an Angstrom apart make terms of 1e9..1e11 kcal/mol beside terms of a few, so
that another order of the sum shows in the logged float energy changes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CLUSTERS = 12


def _antigen(pkg, far):
    """Calphas along z in CLUSTERS groups of 4..26 around the residues' places, 0.5 A from
    them at least; ascending in z, so that every grid lists them in the same order.  far:
    that many more beyond reach."""
    z = [9.0 * c + s * (0.5 + 0.013 * c + 0.2 * i) for c in range(CLUSTERS) for i in range(2 + c) for s in (-1, 1)]
    z = np.concatenate([np.sort(z), 400.0 + 0.5 * np.arange(far)])
    ca = np.stack([np.zeros_like(z), np.zeros_like(z), z], 1).astype(np.float32)
    return pkg.workloads.random_sequence(len(z), pkg.workloads.rng_for(5)), ca


def _log(pkg, far, cell, alone):
    """{(candidate id, residue): (amino acid, action, logged dE)} of one step of mutations."""
    W = pkg.workloads
    n_id = 24
    with pkg.GpuContext.create(0, pkg.Params.defaults(step=0.0, mutation_p=1.0, rotamer_move_p=0.0, backbone_move_p=0.0,
                                                      ca_cell=cell, seed=3)) as ctx:
        ag_aa, ag_ca = _antigen(pkg, far)
        ctx.add_antigen(ag_aa, ctx.build_residues(ag_ca, ag_aa)[0])
        aa = W.random_sequence(n_id * CLUSTERS, W.rng_for(6))
        ca = np.zeros((n_id * CLUSTERS, 3), np.float32)
        ca[:, 2] = 9.0 * np.tile((np.arange(CLUSTERS) * 5 + 11) % CLUSTERS, n_id)  # the largest cluster first
        pos, chi = ctx.build_residues(ca, aa)
        if alone:  # the first residue of every candidate only
            first = np.arange(n_id) * CLUSTERS
            ctx.state_upload(aa[first], chi[first], pos[first], uniform_n_res=1)
        else:
            ctx.state_upload(aa, chi, pos, uniform_n_res=CLUSTERS)
        ctx.mc_log(1 << 16)
        ctx.diffuse(1, 0, with_mc=True, temps=np.ones(1, np.float32))
        log = ctx.mc_log_fetch()
    return {(int(t["cand"]), int(t["residue"])): (int(t["aa"]), int(t["action"]), t["delta_e"].tobytes()) for t in log}


def test_energy_order(pkg):
    ref = _log(pkg, 0, 10.0, False)
    assert len(ref) == 24 * CLUSTERS
    alone = _log(pkg, 0, 10.0, True)
    assert alone == {k: ref[k] for k in alone} and len(alone) == 24
    # a grid too fine for lists: every energy is a scan
    assert _log(pkg, 0, 1.2, False) == ref
    # an antigen too large to be staged: lists and scans of global memory
    assert _log(pkg, 1000, 10.0, False) == ref
    assert _log(pkg, 1000, 1.2, False) == ref
