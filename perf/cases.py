"""The work a user of the library has it do, as cases that can be timed and compared.

Every case goes through the Python binding's public entry points (the C ABI behind
them) on host arrays, as a design program calls them: inputs and results are host
memory, the population of a search is uploaded by the call that starts it and its
results are read back.  Sizes are those of the repository's own workloads
(workloads.py): a 16-residue peptide with 64 x 12-residue antibodies up to 300-800
residue globules with 1024-4096 antibodies.

listed() holds the fixed cases, draw() gives more of the same ranges, prepare() the
inputs and the context a program keeps, run() one pass, work() what the pass cannot
do without, exact() the energies and forces in 64 bits.
"""
import math

import numpy as np
import torch

import __graft_entry__

pkg = __graft_entry__.load_package()
wl = pkg.workloads

SURVIVORS = 64    # survivors of phase 1 (diffusion.rs: the population phase 2 keeps)
BLOCK_STEPS = 10  # gradient steps between two scorings

# Sizes of a case: n_cand candidates of res_min..res_max residues (uniform when equal)
# against n_ag antigens of ag_min..ag_max residues; steps: Langevin / Metropolis /
# refinement / training steps or Fv iterations of the pass.


def _case(kind, n_cand, res_min, res_max, ag_min, ag_max=None, n_ag=1, steps=0, **more):
    return dict(kind=kind, n_cand=n_cand, res_min=res_min, res_max=res_max, ag_min=ag_min,
                ag_max=ag_min if ag_max is None else ag_max, n_ag=n_ag, steps=steps, **more)


def listed():
    return [
        # The drop-in GpuContext::score_batch at the size of a short peptide run: a new
        # set of poses every call, so that launches, copies and latency count.
        dict(_case("score", 64, 12, 12, 16), name="score_peptide"),
        # The same call at the size of a search population against a protein.
        dict(_case("score", 1024, 20, 20, 300), name="score_population"),
        # All-atom forces (the energy's gradient) of ragged candidates: a host program's
        # own minimiser calls it once per step.
        dict(_case("forces", 1024, 10, 30, 300), name="forces_ragged"),
        # A whole phase-1 search pass, population resident on the GPU: upload, 20 enqueued
        # blocks (10 gradient steps, all-atom score, top 64), results and population back.
        # Launch shapes tuned once in advance, as a program with many runs does.
        dict(_case("phase1", 1024, 20, 20, 300, steps=200, tuned=True), name="phase1_population"),
        # The batched form: 8 antigens of 50-800 residues and 4096 ragged candidates in one
        # state, launch shapes as the library picks them.
        dict(_case("phase1", 4096, 10, 30, 50, 800, n_ag=8, steps=50, tuned=False), name="phase1_batched"),
        # The same search with the population in (pinned) host memory: every block uploads
        # it and writes the moved residues back (binder_block_io).
        dict(_case("block_io", 1024, 20, 20, 300, steps=200), name="block_io_population"),
        # The whole run_allatom: 200 gradient steps on 1024 candidates, 600 Langevin +
        # Metropolis steps on the 64 survivors, final ranking.
        dict(_case("run", 1024, 20, 20, 300, steps=600), name="run_allatom"),
        # Annealed Metropolis steps of a whole population in contact (the reference's
        # uniform proposal): training-set generation and annealing studies.
        dict(_case("anneal", 1024, 20, 20, 300, steps=60, learned=False), name="anneal_population"),
        # The same steps with the learned proposal (network evaluated in every step).
        dict(_case("anneal", 1024, 20, 20, 300, steps=60, learned=True), name="anneal_learned"),
        # Training of the proposal network: minibatches of 8192 logged moves.
        dict(_case("train", 8192, 1, 1, 300, steps=20), name="train_proposal"),
        # Post-search refinement of the 64 results: 60 minimisation steps, affinity
        # maturation, structure validation.
        dict(_case("refine", 64, 20, 20, 300, steps=60), name="refine_results"),
        # The Fv two-chain engine: 32 heavy / light pairs of about 120 + 107 residues.
        dict(_case("fv", 32, 12, 9, 300, steps=20), name="fv_pairs"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["score", "forces", "phase1", "block_io", "run", "anneal", "train", "refine", "fv"])
    ag = _log_int(rng, 16, 400)
    if kind in ("score", "forces"):
        lo = rng.randint(6, 30)
        hi = lo if kind == "score" else min(40, lo + rng.randint(0, 15))
        return _case(kind, _log_int(rng, 16, 2048), lo, hi, ag)
    if kind == "phase1":
        n_ag = rng.randint(1, 6)
        lo = rng.randint(8, 24)
        hi = lo if n_ag == 1 else lo + rng.randint(0, 10)
        return _case(kind, max(_log_int(rng, 48, 3000), 8 * n_ag), lo, hi, max(16, ag // 2), ag + 50, n_ag=n_ag,
                     steps=10 * rng.randint(2, 6), tuned=False)
    if kind == "block_io":
        lo = rng.randint(8, 28)
        return _case(kind, _log_int(rng, 48, 1500), lo, lo, ag, steps=10 * rng.randint(3, 12))
    if kind == "run":
        lo = rng.randint(8, 28)
        return _case(kind, _log_int(rng, 64, 1024), lo, lo, ag, steps=rng.randint(60, 400))
    if kind == "anneal":
        lo = rng.randint(8, 40)
        learned = rng.random() < 0.5
        return _case(kind, _log_int(rng, 32, 1024), lo, lo, ag, steps=rng.randint(8, 30), learned=learned)
    if kind == "train":
        return _case(kind, _log_int(rng, 128, 8192), 1, 1, ag, steps=rng.randint(3, 12))
    if kind == "refine":
        lo = rng.randint(8, 30)
        return _case(kind, _log_int(rng, 8, 128), lo, lo, ag, steps=rng.randint(10, 60))
    return _case("fv", _log_int(rng, 4, 32), rng.randint(6, 16), rng.randint(6, 11), max(ag, 50),
                 steps=rng.randint(3, 12))


# ---- inputs -------------------------------------------------------------------------
def _antigens(case, rng):
    """(amino acids, Calpha trace, shell radius) per antigen: an extended peptide up to 24
    residues, else a compact globule of the workloads' density."""
    sizes = np.exp(np.linspace(math.log(case["ag_min"]), math.log(case["ag_max"]), case["n_ag"])).round().astype(int)
    out = []
    for n in sizes:
        aa = wl.random_sequence(int(n), rng)
        if n <= 24:
            out.append((aa, wl.peptide_trace(int(n)), 12.0))
            continue
        radius = 22.0 * (int(n) / 300.0) ** (1.0 / 3.0)
        out.append((aa, wl.globule_trace(int(n), radius, rng, tries=16), radius + 4.0))
    return out


def _population(case, ags, rng, same_sequence=False):
    """Antibodies with Calphas on their antigen's shell: n_res, antigen ids, aa, Calphas.
    Lengths and sequences, which set the sizes of the outputs, are the same for every seed."""
    n = case["n_cand"]
    shape = np.random.default_rng(n)
    n_res = shape.integers(case["res_min"], case["res_max"] + 1, size=n).astype(np.int32)
    ag_id = (np.arange(n) % len(ags)).astype(np.int32)
    if same_sequence:
        aa = np.tile(wl.random_sequence(case["res_min"], shape), n)
    else:
        aa = wl.random_sequence(int(n_res.sum()), shape)
    who = np.repeat(ag_id, n_res)
    d = rng.normal(size=(len(aa), 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    centre = np.stack([wl.ca_center(ca) for _, ca, _ in ags])[who]
    shell = np.array([s for _, _, s in ags])[who]
    return n_res, ag_id, aa, (centre + shell[:, None] * d).astype(np.float32)


def _flat_atoms(aa, pos):
    """GpuAtom records of slot-layout residues, and each residue's atom count."""
    return pkg.AtomCloud.from_slots(aa, pos).to_gpu_atoms(), pkg.tables().n_atoms[aa]


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.from_numpy(a).dtype, pin_memory=torch.cuda.is_available())
    t.numpy()[...] = a
    return t.numpy()


def _score_inputs(case, seed, ctx):
    rng = np.random.default_rng(seed)
    ags = _antigens(case, rng)
    ag_aa, ag_ca, _ = ags[0]
    ag_pos, _ = ctx.build_residues(ag_ca, ag_aa)
    n_res, _, aa, ca = _population(case, ags, rng, same_sequence=case["kind"] == "score")
    pos, _ = ctx.build_residues(ca, aa)
    atoms, n_at = _flat_atoms(aa, pos)
    off = np.concatenate([[0], np.cumsum(np.add.reduceat(n_at, np.concatenate([[0], np.cumsum(n_res)[:-1]])))])
    return pkg.AtomCloud.from_slots(ag_aa, ag_pos), atoms, off.astype(np.int64)


def _search_context(case, rng):
    """A context with the case's antigens added, and their host data."""
    ags = _antigens(case, rng)
    ctx = pkg.GpuContext.create(0, pkg.Params.defaults(shell_radius=float(ags[-1][2]), seed=int(rng.integers(1 << 30))))
    for aa, ca, _ in ags:
        pos, _ = ctx.build_residues(ca, aa)
        ctx.add_antigen(aa, pos)
    return ctx, ags


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("score", "forces"):
        ctx = pkg.GpuContext.create(0)
        antigen, atoms, off = _score_inputs(case, seed, ctx)
        atoms = _pinned(atoms.view(np.float32)).view(pkg.GPU_ATOM)
        return dict(case=case, ctx=ctx, antigen=antigen, atoms=atoms, off=off, n_ab=int(off[1]))
    rng = np.random.default_rng(seed)
    ctx, ags = _search_context(case, rng)
    st = dict(case=case, ctx=ctx, temps=pkg.learned.annealing(max(1, case["steps"]), max(1, case["steps"])))
    if kind == "train":
        # logged moves around the antigen: mutations (action < 20) and rotamer moves
        n, batch = 16 * case["n_cand"], case["n_cand"]
        t = np.zeros(n, pkg.MC_TUPLE)
        _, _, _, ca = _population(dict(case, n_cand=n), ags, rng)
        t["x"], t["y"], t["z"] = ca[:, 0], ca[:, 1], ca[:, 2]
        t["aa"] = rng.integers(0, 20, n)
        t["action"] = np.where(rng.random(n) < 0.9, rng.integers(0, 20, n), 20 + rng.integers(0, 3, n))
        t["delta_e"] = rng.laplace(0.0, 1.0, n)
        ctx.mlp_set_tuples(t)
        st.update(params=pkg.mlp_init_params(int(rng.integers(1 << 30))), batch=batch, seed=int(rng.integers(1 << 30)))
        return st
    if kind == "fv":
        fv = wl.config_fv(ags[0][1], case["n_cand"], case["res_min"], case["res_max"], seed=seed)
        chains = []
        for c in ("heavy", "light"):
            aa, ca, cdr = fv[c]
            pos, chi = ctx.build_residues(ca, aa)
            chains.append((aa, chi, pos, (cdr > 0).astype(np.uint8)))
        ctx.set_params(pkg.Params.defaults(shell_radius=fv["target_radius"], seed=ctx.params.seed))
        return dict(st, heavy=chains[0], light=chains[1], cand_id=np.arange(case["n_cand"], dtype=np.uint32))
    n_res, ag_id, aa, ca = _population(case, ags, rng)
    pos, chi = ctx.build_residues(ca, aa)
    if kind in ("anneal", "refine"):  # a population the gradient steps brought into contact
        ctx.state_upload(aa, chi, pos, n_res=n_res, antigen_id=ag_id)
        ctx.diffuse(200)
        aa, chi, pos = ctx.state_download()
    st.update(aa=_pinned(aa), chi=_pinned(chi), pos=_pinned(pos), n_res=n_res, ag_id=ag_id)
    kept = int(n_res[:min(SURVIVORS, len(n_res))].sum()) if kind == "run" else len(aa)  # run: the ranked results
    st["back"] = (_pinned(np.zeros(kept, np.uint8)), _pinned(np.zeros((kept, 4), np.float32)),
                  _pinned(np.zeros((kept, pkg.SLOTS, 3), np.float32)))
    if case.get("learned"):
        p = pkg.mlp_init_params(int(rng.integers(1 << 30)))
        p[pkg.MLP_OFF["w3"]:pkg.MLP_OFF["b3"]] *= 4.0  # outputs of a few kcal/mol, as after training
        ctx.mlp_set_params(p)
        ctx.set_proposal(True)
    if kind == "phase1" and case["tuned"]:
        ctx.state_upload(st["aa"], st["chi"], st["pos"], n_res=n_res, antigen_id=ag_id)
        ctx.autotune()
    if kind == "block_io":
        n = case["n_cand"]
        st.update(w_e=_pinned(np.zeros(n)), w_top=_pinned(np.zeros(min(SURVIVORS, n), np.int32)))
    return st


# ---- one pass -------------------------------------------------------------------------
def run(s):
    case, ctx = s["case"], s["ctx"]
    kind, steps = case["kind"], case["steps"]
    if kind == "score":
        return ctx.score_batch(s["antigen"], s["atoms"], s["n_ab"])
    if kind == "forces":
        return ctx.forces_allatom(s["antigen"], s["atoms"], s["off"])
    if kind == "train":
        ctx.mlp_set_params(s["params"])
        losses = ctx.mlp_train(steps, batch=s["batch"], seed=s["seed"])
        return losses, ctx.mlp_get_params()
    if kind == "fv":
        ctx.fv_upload(s["heavy"], s["light"], cand_id=s["cand_id"])
        e = ctx.fv_run(steps)
        return e, ctx.fv_download()
    if kind == "block_io":
        # one phase-1 pass of a program that keeps its population in host memory
        w_aa, w_chi, w_pos = s["back"]
        w_aa[:], w_chi[:], w_pos[:] = s["aa"], s["chi"], s["pos"]
        for _ in range(steps // BLOCK_STEPS):
            ctx.block_io(w_aa, w_chi, w_pos, BLOCK_STEPS, len(s["w_top"]), n_res=s["n_res"], antigen_id=s["ag_id"],
                         out_e=s["w_e"], out_top=s["w_top"])
        return s["w_e"], s["w_top"], w_aa, w_chi, w_pos
    ctx.state_upload(s["aa"], s["chi"], s["pos"], n_res=s["n_res"], antigen_id=s["ag_id"])
    k = min(SURVIVORS, case["n_cand"])
    if kind == "phase1":
        for b in range(steps // BLOCK_STEPS):
            ctx.block_async(BLOCK_STEPS, b * BLOCK_STEPS, k)
        return ctx.block_fetch(k, n_segments=case["n_ag"]) + ctx.state_download(*s["back"])
    if kind == "run":
        found = ctx.run_allatom(pkg.RunCfg.defaults(phase2_steps=steps, survivors=k, top_n=k))
        return found + ctx.state_download(*s["back"])
    if kind == "anneal":
        ctx.diffuse(steps, 0, with_noise=True, with_mc=True, temps=s["temps"])
        return (ctx.mc_energy(), ctx.mc_stats()) + ctx.state_download(*s["back"])
    # refine
    e_min = ctx.minimize(steps)
    matured = ctx.affinity_maturation()
    return (e_min,) + matured + ctx.validate() + ctx.state_download(*s["back"])


# ---- what a pass cannot do without ------------------------------------------------------
# Flops of one pair inside the 10 A cutoff: 24 for the all-atom energy, 36 with the
# force, 29 for the Calpha-level force, 20 for a Calpha energy.
ATOMS = 8.0  # heavy atoms of a residue, on average


def _near(ag_res):
    """Antigen residues within 10 A of a point 4 A outside a globule of ag_res residues."""
    if ag_res <= 24:
        return min(ag_res, 5.0)
    R, a = 22.0 * (ag_res / 300.0) ** (1.0 / 3.0), 10.0
    d = R + 4.0
    lens = math.pi * (R + a - d) ** 2 * (d * d + 2 * d * (a + R) - 3 * (a - R) ** 2) / (12 * d)
    return lens * ag_res / (4.0 / 3.0 * math.pi * R ** 3)


def work(case):
    kind, steps, n = case["kind"], max(1, case["steps"]), case["n_cand"]
    res = n * (case["res_min"] + case["res_max"]) / 2.0
    ag = case["n_ag"] * math.sqrt(case["ag_min"] * case["ag_max"])
    near = _near(ag / case["n_ag"])
    score = res * ATOMS * near * ATOMS * 24.0
    cg = res * near * 29.0
    state = res * (14 * 12 + 16 + 1)  # positions, chi, amino acid
    ag_bytes = ag * ATOMS * 30
    if kind == "score":
        return {"bytes": res * ATOMS * 32 + ag_bytes + 4 * n, "flops": score}
    if kind == "forces":
        return {"bytes": res * ATOMS * 44 + ag_bytes + 8 * n, "flops": 1.5 * score}
    if kind == "train":
        par = pkg.MLP_N_PARAMS
        return {"bytes": steps * n * 32 + 8 * par, "flops": 6.0 * steps * n * par}
    if kind == "phase1":
        return {"bytes": 2 * state + ag_bytes + 8 * n, "flops": steps * cg + steps / BLOCK_STEPS * score}
    if kind == "block_io":
        blocks = steps / BLOCK_STEPS
        return {"bytes": blocks * (2 * state + 8 * n) + ag_bytes, "flops": steps * cg + blocks * score}
    # a Metropolis step of n residues: the force, about 0.15 n moves of two energies and
    # 0.04 n backbone moves of n / 2 energies
    def mc(c, length):
        return c * length * (near * 29.0 + (0.3 + 0.02 * length) * near * 20.0)
    if kind == "run":
        surv = min(SURVIVORS, n)
        return {"bytes": state * (1 + surv / n) + ag_bytes, "flops": 200 * cg + 20 * score + steps * mc(surv, case["res_min"])}
    if kind == "anneal":
        net = 2.0 * 0.11 * res * pkg.MLP_N_PARAMS if case["learned"] else 0.0
        return {"bytes": 2 * state + ag_bytes + 40 * n, "flops": steps * (mc(n, case["res_min"]) + net)}
    if kind == "refine":
        # minimisation, then 19 other amino acids at about half of the positions
        return {"bytes": 2 * state + ag_bytes + 24 * n, "flops": steps * (cg + 1.2 * score) + 10 * 1.2 * score}
    heavy, light = 99 + case["res_min"], 94 + case["res_max"]
    both = heavy + light
    pair = heavy * light * ATOMS * ATOMS * 0.1 * 24.0
    return {"bytes": 2 * n * both * 185 + ag_bytes, "flops": steps * n * (
        mc(1, heavy) + mc(1, light) + both * ATOMS * near * ATOMS * 29.0 + pair)}


# ---- 64-bit results ---------------------------------------------------------------------
def exact(case, seed):
    """Energies (and forces) of the flat-atom calls by brute force in 64 bits; the pair set
    is the reference's, whose cutoff test takes r^2 in f32.  None for the searches, whose
    trajectories are not defined beyond their f32 steps."""
    if case["kind"] not in ("score", "forces"):
        return None
    with pkg.GpuContext.create(0) as ctx:
        ag, atoms, off = _score_inputs(case, seed, ctx)
    dev = "cuda" if torch.cuda.is_available() else "cpu"

    def put(a, dtype=torch.float64):
        return torch.from_numpy(np.ascontiguousarray(a)).to(dev).to(dtype)

    A32 = torch.stack([put(v, torch.float32) for v in (ag.x, ag.y, ag.z)])
    aq, arm, aep, ahy = (put(v) for v in (ag.charge, ag.r_min_half, ag.epsilon, ag.hydrophobic))
    b32 = torch.stack([put(atoms[v], torch.float32) for v in ("x", "y", "z")])
    bq, brm, bep, bhy = (put(atoms[v]) for v in ("q", "r_min_half", "epsilon", "hydrophobic"))
    n = len(atoms)
    e_atom = torch.zeros(n, dtype=torch.float64, device=dev)
    force = torch.zeros((n, 3), dtype=torch.float64, device=dev)
    rows = max(1, (1 << 25) // max(1, A32.shape[1]))
    for i in range(0, n, rows):
        j = slice(i, min(n, i + rows))
        d32 = b32[:, j, None] - A32[:, None, :]
        r32 = d32[0] * d32[0] + d32[1] * d32[1] + d32[2] * d32[2]
        near = (r32 <= 100.0) & (r32 >= 0.25)
        d = b32[:, j, None].double() - A32[:, None, :].double()
        r2 = torch.where(near, (d * d).sum(0), torch.ones((), dtype=torch.float64, device=dev))
        s6 = ((brm[j, None] + arm) ** 2 / r2) ** 3
        eps = torch.sqrt(bep[j, None] * aep)
        coul = 332.0 * bq[j, None] * aq / torch.sqrt(r2)
        hyd = torch.where((r32 < 36.0) & (bhy[j, None] > 0.5) & (ahy > 0.5), -0.5, 0.0)
        e = eps * s6 * (s6 - 2.0) + coul + hyd
        e_atom[j] = torch.where(near, e, torch.zeros_like(e)).sum(1)
        sc = torch.where(near, (12.0 * eps * s6 * (s6 - 1.0) + coul) / r2, torch.zeros_like(e))
        force[j] = (sc * d).sum(2).T
    energy = torch.from_numpy(np.add.reduceat(e_atom.cpu().numpy(), off[:-1]))
    if case["kind"] == "score":
        return energy
    return force.cpu(), energy
