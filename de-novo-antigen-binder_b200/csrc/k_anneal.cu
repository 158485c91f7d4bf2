// k_anneal.cu — allatom_diffusion_step with its Metropolis moves (diffusion.rs:290-463)
// on the GPU: one CTA per candidate, the candidate's residues and its antigen's
// Calphas resident in shared memory for all n_steps of the launch.
//
// Per step, in the reference's order:
//  1. Langevin: coarse-grained force, restraint, noise, 2 A clamp, rigid
//     translation (diffusion.rs:306-339), then the interface test (any antigen
//     Calpha within sqrt(iface_cutoff_sq), :343-351) and the residue's mutation /
//     rotamer draw, all by one group of GL lanes per residue.  The force comes from
//     the residue's Verlet list: its in-cutoff entries in list order are the
//     reference's pairs in its order; the group compacts them, evaluates one pair per
//     lane and folds the terms in that order by shuffles -- the reference's
//     sequential sum, held by every lane.  Meanwhile idle warps draw the backbone
//     moves.
//  2. Mutation / rotamer sweep (:354-399).  A move at residue r changes only
//     residue r's atoms, and the Calpha-level energy of r depends only on r's
//     Calpha and amino acid; residues interact only through the disulfide term.
//     So every proposal, its rejection rebuild and both Calpha energies are computed
//     in parallel (builds on the last warps, energies on the others, together with
//     the energies the first backbone move starts from); then warp 0 decides: the
//     moves that involve a Cys in residue order, updating the disulfide energy, the
//     others -- which leave it unchanged -- each by a lane with the disulfide energy
//     of its turn: the reference's sequential sweep, exactly.
//  3. Backbone phi/psi sweep (:403-418): sequential over the attempted moves;
//     per move the downstream atoms rotated by all threads (Rodrigues,
//     allatom.rs:397-479), the Calpha energies of residues r+1..n by all warps, the
//     decision by warp 0; a rejected move is undone by the opposite rotation, as in
//     the reference, and the energies it disturbed are recomputed only if another
//     move follows in the same step.
//
// What bounds it: the chain of dependent latencies of a step (one candidate's work is
// tiny), so every phase is arranged to be short and few (four barriers a step -- the
// second among the energy warps only unless a Cys moves -- four more per backbone move and
// one after a rejected one) and many candidates share an SM.  64 x 20 residues, 300-residue
// antigen, 600 steps: 13.4 ms before (42 k cycles a step: lane-0 FP64 folds of every
// energy, one thread scanning for Cys pairs, side chains built from divergent constant
// tables and local memory, nine barriers), 9.5 ms so arranged, 9.1 ms with the lists kept
// between launches and the skins below; 1024 x 20 residues, 60 steps: 7.9, 4.2, 4.1 ms.
// What is left is about 6.5 cycles per dependent instruction (2.5 of fixed latency, 1 of
// shared memory, 0.8 of branches, 0.7 of instruction fetch) and the other warps' waits for
// the one that decides: the code is kept small -- one copy of each exponential, pair term and scan, no
// unrolling (178 -> 122 KB) -- because several warps in different phases of unrolled code
// waited for instructions more than for anything else (a 1024-candidate launch 5.5 -> 4.3 ms).
//
// Accumulation: ACC = float reproduces the reference's f32 sums bit for bit (terms
// staged and added in antigen order by one lane); ACC = double sums the same f32 pair
// terms in double in one fixed order (EL below) and takes the Metropolis test on the
// double energy difference.
#include <type_traits>

#include "cg_list.cuh"
#include "geom.cuh"
#include "kernels.h"
#include "mlp_tile.cuh"

namespace binder {

cudaError_t anneal_init_tables() { return geom_init_tables(); }

// log1p of the environment counts for the in-kernel features (the same host table
// as the feature kernel's); copied to shared memory by each learned-proposal CTA
__device__ float g_an_log1p[MLP_COUNT_CAP + 1];
cudaError_t anneal_init_mlp_table(const float* t) {
    return cudaMemcpyToSymbol(g_an_log1p, t, sizeof(float) * (MLP_COUNT_CAP + 1));
}

constexpr int AN_WARPS = 8;
constexpr int AN_THREADS = AN_WARPS * 32;
constexpr int STAGE_CAP = 64;                        // staged in-cutoff terms per warp (ACC = float)
constexpr int HIT_CAP = 96;                          // in-cutoff entries a warp's scan holds (ACC = double)
// Skins of the residues' lists: a residue's first, and the most a residue that outruns its
// list gets (twice the last).  600 steps of 64 candidates and the rest of run_allatom: 12.35
// ms with at most 4 A, 12.8 with 5, 12.6 with 3 (longer lists cost every step, shorter ones
// more builds).  Fv chains take wide ones from the start (7.5 ms for 32 pairs x 20 steps
// with 4 and 8 A, 7.9 with 2 and 5): their backbone moves swing 60 residues at a time, and
// an energy inside the skin costs a fifth of a scan.
template <bool FV>
constexpr float AN_SKIN = FV ? 4.0f : 2.0f;
template <bool FV>
constexpr float AN_SKIN_MAX = FV ? 8.0f : 4.0f;
constexpr int MASK_WORDS = ANNEAL_MAX_RES / 32;      // residue bit masks of a candidate
constexpr int AN_IN = 32;                            // in-cutoff entries of the force a residue holds per round
constexpr int AG_STAGE_MAX = 1024;                   // antigen Calphas staged in shared memory
constexpr int CELL_STAGE_MAX = 4096;                 // Calpha-grid cells staged in shared memory
enum : int { MV_NONE = 0, MV_ROT = 1, MV_MUT = 2 };
enum : int { SEL_KEEP = 0, SEL_PROP = 1, SEL_REJ = 2, SEL_SIDE = 4 };  // SEL_SIDE: only the side chain was built
enum : int { IS_DVALID = 0, IS_DECISION = 1, IS_CYSMV = 2, IS_NMV = 4, IS_NTASK = 5 };

// What the Calpha energies read of the antigen: its Calphas in list (grid) order.
struct AnEnv {
    const float4* pos;
    const uint8_t* aa;
    int n, np;  // antigen Calphas, Fv: partner residues
};

// Fixed part of a CTA's shared memory: candidates of up to RT residues, W warps, ACC
// double or float (F32), with the learned proposal (LRN) or one chain of an Fv pair
// (FV).  Everything the step touches lies at a compile-time offset: with offsets read
// from the parameter bank each first access of a phase waited for a constant load.  The
// staged antigen follows it (an_tail_bytes).
template <int RT_, int W_, bool F32_, bool LRN_, bool FV_>
struct AnSmem {
    static constexpr int RT = RT_, W = W_;
    static constexpr bool F32 = F32_, LRN = LRN_, FV = FV_;
    float4 pos[RT * SLOT_STRIDE], prop[RT * SLOT_STRIDE], rej[RT * SLOT_STRIDE];  // state, proposals, rejections
    float4 trig[2 * RT];                      // sin/cos of chi1..4
    float4 chi[RT];                           // degrees
    float4 bb_trig[RT];                       // cos, sin of the torsion step and of its negation
    float4 cgcentre[RT];                      // list centre, skin
    float4 sct[N_AA * SC_MAX];                // bond, sin, cos of the angle, the reference atoms' bits
    float4 ca_atom[N_AA], res[N_AA];          // Calpha atom: charge, r_min_half, eps, hyd; residue-level parameters
    float4 stage[F32 ? W * STAGE_CAP : 1];    // F32: in-cutoff Calpha-energy terms
    float4 ptq[FV ? RT : 1], ptp[FV && F32 ? RT : 1];  // Fv: the partner's Calpha atoms (x, y, z, q | prm)
    float4 pcq[FV ? RT : 1], pcp[FV ? RT : 1];  // and residue-level bodies (AgView::ca_pq / ca_prm layout)
    float2 scf[N_AA * SC_MAX];                // sin, cos of the fixed dihedral
    float2 rott[N_AA * 20 + 4];               // rotamer sin/cos, then 4 x (0, 1)
    float2 hits[F32 ? 1 : W * HIT_CAP];       // in-cutoff (r^2, index)
    double c_cur[RT], c_old[RT], c_new[RT];   // Calpha energies (exact f32 values when F32)
    double lhr[RT];                           // log Hastings ratio of the move (network path)
    double d_turn[RT];                        // disulfide energy at the move's turn, then (log) its energy change
    double dscal;                             // disulfide energy of the current state
    AgView ag;
    AnEnv env;
    float u_acc[RT], bb_u[RT];
    int aa[RT], kind[RT], new_aa[RT], new_rot[RT], sel[RT], bb_phi[RT], cgnl[RT];
    int task[2 * RT];                         // 2 r + (0 proposal / energy before, 1 rejection / after) of the moves
    int rot[RT], mvl[RT];                     // rotamer index of the state (-1 unknown), residues with a move
    uint32_t dz[RT];                          // the move's choice draw
    int topo_n[N_AA], sc_n[N_AA], rot_n[N_AA], ca_hb[N_AA];
    unsigned attw[2 * MASK_WORDS];            // backbone attempts (two: a fast warp may draw the next step's
                                              // while a slow one still reads)
    unsigned cysw[MASK_WORDS], mxw[MASK_WORDS];  // Cys residues, moves that involve a Cys
    int iscal[8];
    float lg1p[LRN ? MLP_COUNT_CAP + 1 : 1];  // the log1p count table
    float mbias[LRN ? MLP_BIASES : 1];        // the network's biases b1 | b2 | b3
    __align__(16) unsigned char tile[LRN ? MT_BYTES : 16];  // the network tile
    __align__(16) uint16_t cglist[RT * CG_LIST_MAX];  // Verlet lists of the Langevin force
    uint8_t ptaa[RT], dirty[RT];              // dirty: the list was built in this launch
    unsigned char cysid[W][RT];               // Cys residues of a warp's disulfide sum
};
// Entries of each staged x / y / z array: room for the pad, a multiple of 4.
__host__ __device__ inline int anneal_xyz_len(int G) { return G > 0 ? (G + 4) & ~3 : 0; }
// The staged antigen: Calphas in CG-grid order (x, y, z, residue charge | residue-level
// epsilon, sigma, hydrophobic), F32 also the Calpha atoms in residue order (x, y, z, q |
// prm; x, y, z arrays), cell starts, amino acids in grid order.
__host__ __device__ inline size_t an_tail_bytes(int G, int C, bool f32) {
    return (size_t)G * (f32 ? 64 : 32) + (f32 ? (size_t)anneal_xyz_len(G) * 12 : 0) + (size_t)C * 4 + (size_t)G;
}
template <class L>
__device__ __forceinline__ L& an_smem() {
    extern __shared__ __align__(16) unsigned char an_smem_raw[];
    return *reinterpret_cast<L*>(an_smem_raw);
}

// hbond_energy (energy.rs:32-39) with the Metropolis-path exponential
__device__ __noinline__ float hbond_mc(float r_sq) {
    if (r_sq > HB_CUTOFF_SQ) return 0.0f;
    const float r = xsqrt(r_sq);
    const float z = xdiv(xsub(r, HB_R0), HB_SIGMA);
    return xmul(-HB_DEPTH, mc_exp(xmul(xmul(-0.5f, z), z)));
}

// Add staged Calpha-energy terms in order (lj; coulomb; hydrophobic; hbond per pair).
template <class ACC>
__device__ __forceinline__ void fold_terms(const float4* stage, int cnt, ACC& e) {
    for (int j = 0; j < cnt; ++j) {
        const float4 v = stage[j];
        const unsigned fl = __float_as_uint(v.w);
        e += (ACC)v.x;
        if (fl & 1u) e += (ACC)v.y;
        if (fl & 2u) e -= (ACC)0.5f;
        if (fl & 4u) e += (ACC)v.z;
    }
}

// The staged terms of one in-cutoff pair (r_sq passed the reference's cutoff test):
// lj; coulomb (flag 1); hydrophobic (flag 2); hbond (flag 4) -- residue_contribution_
// allatom's per-pair arithmetic (diffusion.rs:425-463).  b = the residue's Calpha
// (q, r_min_half, epsilon, hydrophobic), bhb its H-bond role.
__device__ __forceinline__ float4 ca_pair_terms(const float4& b, int bhb, const float4& a, const float4& ap,
                                                float r_sq) {
    float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
    unsigned fl = 0;
    const float r_ij = xadd(b.y, ap.x);
    const float eps = xsqrt(xmul(b.z, ap.y));
    const float r2 = xdiv(xmul(r_ij, r_ij), r_sq);
    const float r6 = xmul(xmul(r2, r2), r2);
    t.x = xmul(eps, xsub(xmul(r6, r6), xmul(2.0f, r6)));
    if (b.x != 0.0f && a.w != 0.0f) {
        t.y = xdiv(xmul(xmul(COULOMB_K, b.x), a.w), xsqrt(r_sq));
        fl |= 1u;
    }
    if (b.w == 1.0f && ap.z == 1.0f && r_sq < HYDRO_CUTOFF_SQ) fl |= 2u;
    const int ahb = s_hb_role[(int)ap.w];
    if (((bhb & 1) && (ahb & 2)) || ((bhb & 2) && (ahb & 1))) {
        t.z = hbond_mc(r_sq);
        fl |= 4u;
    }
    t.w = __uint_as_float(fl);
    return t;
}

// residue_contribution_allatom (diffusion.rs:425-463) of a Calpha at `ca` of amino
// acid `aa`, by one warp: lanes evaluate 32 antigen Calphas at a time (index
// order), in-cutoff terms are compacted into the warp's stage in that order and
// lane 0 adds them in the reference's order.  Result valid in lane 0.
template <class ACC>
__device__ __noinline__ ACC warp_contribution(const float4* __restrict__ agq, const float4* __restrict__ agp, int nag, F3 ca,
                                 int aa, float4* stage) {
    const int lane = threadIdx.x & 31;
    const float4 b = s_ca_atom[aa];  // q, r_min_half, epsilon, hydrophobic
    const int bhb = s_hb_role[s_ca_type[aa]];
    ACC e = 0;
    int cnt = 0;
    for (int base = 0; base < nag; base += 32) {
        const int i = base + lane;
        bool in = false;
        float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
        if (i < nag) {
            const float4 a = agq[i];
            const float r_sq = xdist2(xsub(ca.x, a.x), xsub(ca.y, a.y), xsub(ca.z, a.z));
            in = !(r_sq > CUTOFF_SQ || r_sq < MIN_R_SQ);
            if (in) t = ca_pair_terms(b, bhb, a, agp[i], r_sq);
        }
        const unsigned m = __ballot_sync(0xffffffffu, in);
        if (in) stage[cnt + __popc(m & ((1u << lane) - 1u))] = t;
        cnt += __popc(m);
        if (cnt > STAGE_CAP - 32) {  // flush before the stage can overflow
            __syncwarp();
            if (lane == 0) fold_terms(stage, cnt, e);
            __syncwarp();
            cnt = 0;
        }
    }
    __syncwarp();
    if (lane == 0) fold_terms(stage, cnt, e);
    __syncwarp();
    return e;
}

// The same for a staged antigen whose Calpha coordinates are also kept as x / y / z
// arrays (ax, ay, az; 8-byte aligned, entry nag a +1e30 pad when nag is odd).  Lane
// l tests Calphas base + 2l and base + 2l + 1 with one packed f32x2 computation (the
// same roundings as xdist2), 64 Calphas per warp step, and stages each in-cutoff
// Calpha's (r^2, index) in index order; the pair terms of everything staged are then
// computed one entry per lane (in place) and lane 0 adds them in order -- so the
// term code runs once per 32 in-cutoff Calphas instead of once per scan step.
template <class ACC>
__device__ __noinline__ ACC warp_contribution_pairs(const float* __restrict__ ax, const float* __restrict__ ay,
                                       const float* __restrict__ az, const float4* __restrict__ agq,
                                       const float4* __restrict__ agp, int nag, F3 ca, int aa, float4* stage) {
    static_assert(STAGE_CAP >= 64, "one step stages up to 64 entries");
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const float4 b = s_ca_atom[aa];
    const int bhb = s_hb_role[s_ca_type[aa]];
    const uint64_t cx = f2_pack(ca.x, ca.x), cy = f2_pack(ca.y, ca.y), cz = f2_pack(ca.z, ca.z);
    ACC e = 0;
    int cnt = 0;
    auto terms_and_fold = [&]() {  // the staged entries' terms, in place, then their sum in order
        __syncwarp();
        for (int k = lane; k < cnt; k += 32) {
            const float4 v = stage[k];
            const int i = __float_as_int(v.y);
            stage[k] = ca_pair_terms(b, bhb, agq[i], agp[i], v.x);
        }
        __syncwarp();
        if (lane == 0) fold_terms(stage, cnt, e);
        __syncwarp();
        cnt = 0;
    };
    for (int base = 0; base < nag; base += 64) {
        const int i = base + 2 * lane;
        bool in0 = false, in1 = false;
        float r0 = 0.0f, r1 = 0.0f;
        if (i < nag) {
            const uint64_t dx = f2_sub(cx, *(const uint64_t*)&ax[i]);
            const uint64_t dy = f2_sub(cy, *(const uint64_t*)&ay[i]);
            const uint64_t dz = f2_sub(cz, *(const uint64_t*)&az[i]);
            f2_dist2(dx, dy, dz, r0, r1);
            in0 = !(r0 > CUTOFF_SQ || r0 < MIN_R_SQ);
            in1 = i + 1 < nag && !(r1 > CUTOFF_SQ || r1 < MIN_R_SQ);
        }
        const unsigned m0 = __ballot_sync(0xffffffffu, in0), m1 = __ballot_sync(0xffffffffu, in1);
        const int n_step = __popc(m0) + __popc(m1);
        if (cnt + n_step > STAGE_CAP) terms_and_fold();
        const int at = cnt + __popc(m0 & lt) + __popc(m1 & lt);  // Calphas before base + 2 * lane
        if (in0) stage[at] = make_float4(r0, __int_as_float(i), 0.f, 0.f);
        if (in1) stage[at + (in0 ? 1 : 0)] = make_float4(r1, __int_as_float(i + 1), 0.f, 0.f);
        cnt += n_step;
    }
    terms_and_fold();
    return e;
}

// residue_contribution_allatom summed in double, order free: the pair of two Calphas
// within the cutoff, of amino acids with the Calpha atoms a and b (charge, r_min_half,
// eps, hyd) and H-bond roles -- ca_pair_terms' operations.
__device__ __noinline__ double ca_pair_sum(const float4 b, int bhb, const float4 a, int ahb, float r_sq) {
    const float r_ij = xadd(b.y, a.y);
    const float eps = xsqrt(xmul(b.z, a.z));
    const float r2 = xdiv(xmul(r_ij, r_ij), r_sq);
    const float r6 = xmul(xmul(r2, r2), r2);
    double e = (double)xmul(eps, xsub(xmul(r6, r6), xmul(2.0f, r6)));
    if (b.x != 0.0f && a.x != 0.0f) e += (double)xdiv(xmul(xmul(COULOMB_K, b.x), a.x), xsqrt(r_sq));
    if (b.w == 1.0f && a.w == 1.0f && r_sq < HYDRO_CUTOFF_SQ) e -= 0.5;
    if (((bhb & 1) && (ahb & 2)) || ((bhb & 2) && (ahb & 1))) e += (double)hbond_mc(r_sq);
    return e;
}

// The double sum of a Calpha energy: the in-cutoff Calphas numbered in list (grid) order
// (Fv: then the partner chain's), number h added to partial sum h % EL, and the partial
// sums folded in a fixed order.  List and scan, alone or beside other tasks, give the same
// bits (a Calpha's number does not depend on how it was found), so a run does not depend on
// the lists that earlier launches left.
constexpr int EL = 8;  // lanes per Calpha energy, a partial sum each
struct ScanSum {
    double e;  // partial sum lane % EL
    int n;     // Calphas within the cutoff
};

// A Calpha at `ca` of amino acid `aa` against all antigen Calphas, in double, by one warp:
// two tests per lane and step, the in-cutoff ones queued and their terms evaluated 32 at a
// time.
template <class L>
__device__ __noinline__ ScanSum warp_scan_energy(F3 ca, int aa, float2* hits) {
    L& S = an_smem<L>();
    const float4* pos = S.env.pos;
    const uint8_t* ag_aa = S.env.aa;
    const int n = S.env.n, lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const float4 b = S.ca_atom[aa];
    const int bhb = S.ca_hb[aa];
    ScanSum sum = {0.0, 0};
    int cnt = 0;
#pragma unroll 1
    for (int base = 0; base < n; base += 64) {
        const int i0 = base + lane, i1 = i0 + 32;
        const float4 a0 = pos[min(i0, n - 1)], a1 = pos[min(i1, n - 1)];
        const float r0 = xdist2(xsub(ca.x, a0.x), xsub(ca.y, a0.y), xsub(ca.z, a0.z));
        const float r1 = xdist2(xsub(ca.x, a1.x), xsub(ca.y, a1.y), xsub(ca.z, a1.z));
        const bool in0 = i0 < n && !(r0 > CUTOFF_SQ || r0 < MIN_R_SQ);
        const bool in1 = i1 < n && !(r1 > CUTOFF_SQ || r1 < MIN_R_SQ);
        const unsigned m0 = __ballot_sync(0xffffffffu, in0), m1 = __ballot_sync(0xffffffffu, in1);
        const int c0 = cnt + __popc(m0);
        if (in0) hits[cnt + __popc(m0 & lt)] = make_float2(r0, __int_as_float(i0));
        if (in1) hits[c0 + __popc(m1 & lt)] = make_float2(r1, __int_as_float(i1));
        cnt = c0 + __popc(m1);
        const bool last = base + 64 >= n;
        if (cnt > 32 || last) {  // room for the next step's 64, or the end
            __syncwarp();
            int done = 0;
#pragma unroll 1
            for (; done + (last ? 0 : 31) < cnt; done += 32) {
                double t = 0.0;
                if (done + lane < cnt) {
                    const float2 h = hits[done + lane];
                    const int a = ag_aa[__float_as_int(h.y)];
                    t = ca_pair_sum(b, bhb, S.ca_atom[a], S.ca_hb[a], h.x);
                }
                __syncwarp();
#pragma unroll
                for (int o = 0; o < 32; o += EL) sum.e += __shfl_sync(0xffffffffu, t, (lane & (EL - 1)) + o);
            }
            sum.n += min(done, cnt);
            if (!last) {  // the rest, fewer than 32, to the front
                cnt -= done;
                const float2 h = hits[done + lane];
                __syncwarp();
                if (lane < cnt) hits[lane] = h;
            }
        }
    }
    return sum;
}

// disulfide_energy (allatom.rs:155-180) over the SG atoms (topology atom 5) of the
// residues in the bit mask cysw, pairs in residue order, by one warp: the lanes list the
// Cys residues, test 32 pairs at a time and the in-range terms are subtracted in order
// (the result is on every lane).  sweep: residues take their slots as the sweep sees
// them (their proposal when accepted, their rejection rebuild when rejected, else the state)
// and residue `sub` (>= 0) its proposal; else every residue is read from the state.
template <class L, class ACC>
__device__ __noinline__ ACC warp_disulfide(bool sweep, int words, int sub) {
    L& S = an_smem<L>();
    const int lane = threadIdx.x & 31;
    ACC e = 0;
    int k = 0;
    unsigned char* ids = S.cysid[threadIdx.x >> 5];
    __syncwarp();
#pragma unroll 1
    for (int w = 0; w < words; ++w) {
        const unsigned m = S.cysw[w];
        if (m >> lane & 1u) ids[k + __popc(m & ((1u << lane) - 1u))] = (unsigned char)(w * 32 + lane);
        k += __popc(m);
    }
    if (k < 2) return e;
    __syncwarp();
    auto sg = [&](int j) -> float4 {
        const int s = sweep ? (j == sub ? (int)SEL_PROP : S.sel[j] & 3) : (int)SEL_KEEP;
        return (s == SEL_PROP ? S.prop : s == SEL_REJ ? S.rej : S.pos)[j * SLOT_STRIDE + 5];
    };
    int i = 0, left = lane;  // this lane's pair: (i, i + 1 + left)
    const int pairs = k * (k - 1) / 2;
#pragma unroll 1
    for (int p0 = 0; p0 < pairs; p0 += 32, left += 32) {
        float t = 0.0f;
        bool in = false;
        if (p0 + lane < pairs) {
            while (left >= k - 1 - i) {
                left -= k - 1 - i;
                ++i;
            }
            const float4 pi = sg(ids[i]), pj = sg(ids[i + 1 + left]);
            const float d = xsqrt(xdist2(xsub(pi.x, pj.x), xsub(pi.y, pj.y), xsub(pi.z, pj.z)));
            in = !(d > 4.0f);
            if (in) {
                const float z = xdiv(xsub(d, 2.05f), 0.4f);
                t = xmul(4.0f, mc_exp(xmul(xmul(-0.5f, z), z)));
            }
        }
        for (unsigned m = __ballot_sync(0xffffffffu, in); m; m &= m - 1) e -= (ACC)__shfl_sync(0xffffffffu, t, __ffs(m) - 1);
    }
    return e;
}

// The exponentials and trigonometry of the step, one copy each: inlined at every use
// their double-precision code was most of the kernel's instruction footprint.
__device__ __noinline__ bool accept_exact(float de, float temp, float u, double) { return u < mc_exp(xdiv(-de, temp)); }
__device__ __noinline__ bool accept_exact(double de, float temp, float u, double lhr) {
    return (double)u < exp(lhr == 0.0 ? -de / (double)temp : -de / (double)temp + lhr);
}
__device__ __noinline__ float4 torsion_trig(float delta) {  // cos, sin of delta and of -delta
    const float ca = mc_cos(delta), sa = mc_sin(delta);
    return make_float4(ca, sa, ca, -sa);
}
__device__ __noinline__ U4 step_draw(uint64_t seed, uint32_t cand, uint32_t step, uint32_t stream, uint32_t r) {
    return rng_draw(seed, cand, step, stream, r);
}

// Metropolis-Hastings (diffusion.rs:368, 385, 414-415) with the log proposal ratio lhr
// = log q(reverse) - log q(forward), 0 for the uniform proposal: accept when de <= 0 or
// u < exp(-dE/T + lhr) (for lhr = 0 the plain criterion).  The exponential is first
// taken in fast f32, whose argument x + l is off by less than 1e-6 (|x| + |l|): below
// -17 with that margin it is smaller than any nonzero u (u is 0 or at least 2^-24 =
// e^-16.6); with |x| + |l| < 64 the value is off by less than 1e-4 of itself, so a u
// further away is decided.  The others (about one in 10^4) take the exact test (ACC =
// float: the reference's f32 one).
template <class ACC>
__device__ __noinline__ bool mh_accept(ACC de, float temp, float u, double lhr) {
    if (lhr == 0.0 && de <= (ACC)0) return true;
    const float x = __fdividef(-(float)de, temp), l = (float)lhr, size = fabsf(x) + fabsf(l);
    if (x + l + 1e-6f * size < -17.0f && u > 0.0f) return false;
    if (size < 64.0f) {
        const float pr = __expf(x + l);
        if (u < pr * 0.9999f) return true;
        if (u > pr * 1.0001f) return false;
    }
    return lhr == 0.0 ? accept_exact(de, temp, u, 0.0) : accept_exact((double)de, temp, u, lhr);
}

// ---- learned proposal -------------------------------------------------------------
// Features of the tile rows: row i = residue mvl[base + i]; the one-hot of its amino
// acid for a rotamer query, none for a mutation query (the network's mutation
// outputs then depend on the environment alone, the same before and after the
// move); one warp per row (8 rows, 8 warps).  The environment counts come from the
// residue's Verlet list when it still covers the Calpha, else from all Calphas.
template <class L>
__device__ __forceinline__ void an_tile_features(const L& S, const MlpTile& T, const int* rows_of, int base, int rows) {
    const float4* agq = S.env.pos;
    const uint8_t* ag_aa = S.env.aa;
    const float* lg1p = S.lg1p;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int i = warp; i < MT_ROWS; i += AN_WARPS) {
        int* cnt = T.cnt + i * MLP_SHELLS * N_AA;
        __nv_bfloat16* x = T.x + i * MT_XS;
        if (i >= rows) {
            for (int j = lane; j < MLP_K1; j += 32) x[j] = __float2bfloat16_rn(0.0f);
            continue;
        }
        const int r = rows_of[base + i];
        for (int j = lane; j < MLP_SHELLS * N_AA; j += 32) cnt[j] = 0;
        __syncwarp();
        const float4 ca = S.pos[r * SLOT_STRIDE + 1];
        const float4 cc = S.cgcentre[r];
        const int nl = S.cgnl[r];
        const float mx = ca.x - cc.x, my = ca.y - cc.y, mz = ca.z - cc.z;
        if (nl <= CG_LIST_MAX && mx * mx + my * my + mz * mz <= (cc.w - 0.01f) * (cc.w - 0.01f)) {
            const uint16_t* list = S.cglist + (size_t)r * CG_LIST_MAX;
            for (int j = lane; j < nl; j += 32) {
                const int k = list[j];
                const float4 q = agq[k];
                const float r2 = xdist2(xsub(ca.x, q.x), xsub(ca.y, q.y), xsub(ca.z, q.z));
                if (r2 < 100.0f) atomicAdd(&cnt[mlp_shell(r2) * N_AA + ag_aa[k]], 1);
            }
        } else {
            mlp_count_env(agq, ag_aa, S.env.n, ca.x, ca.y, ca.z, cnt);
        }
        __syncwarp();
        const int a = S.kind[r] == MV_MUT ? -1 : S.aa[r];
        for (int j = lane; j < MLP_K1; j += 32) {
            float v = 0.0f;
            if (j < N_AA) v = j == a ? 1.0f : 0.0f;
            else if (j < MLP_IN) v = lg1p[min(cnt[j - N_AA], MLP_COUNT_CAP)];
            x[j] = __float2bfloat16_rn(v);
        }
    }
}

// Choice among n options (n <= 32) with probabilities softmax(-y / tp), by one
// warp, lane k holding option k: FP64 weights w_k = exp((min y - y[k]) / tp) (the
// largest is 1) and the inverse CDF on u = dz / 2^32 over their prefix sums (for
// equal outputs exactly urange(dz, n): the prefix sums are then exact integers).
// inv_tp = 1 / tp.  Returns the option (all lanes).  Its log probability is never
// needed: a move's Hastings ratio is a difference of two logits of the same softmax.
__device__ int warp_sample(const float* y, int n, double inv_tp, uint32_t dz) {
    const int lane = threadIdx.x & 31;
    const float yl = lane < n ? y[lane] : INFINITY;
    float ymin = yl;
#pragma unroll
    for (int o = 16; o; o >>= 1) ymin = fminf(ymin, __shfl_xor_sync(0xffffffffu, ymin, o));
    double cum = lane < n ? exp(((double)ymin - (double)yl) * inv_tp) : 0.0;  // inclusive prefix sum in lane order
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double v = __shfl_up_sync(0xffffffffu, cum, o);
        if (lane >= o) cum += v;
    }
    const double total = __shfl_sync(0xffffffffu, cum, 31);
    const double target = (double)dz * (1.0 / 4294967296.0) * total;
    const unsigned hit = __ballot_sync(0xffffffffu, lane < n && target < cum);
    return hit ? __ffs(hit) - 1 : n - 1;
}

// The residue a move leaves: which = SEL_PROP builds the proposal, SEL_REJ the state
// after a rejection (rebuild_side_chain with the old chi, or mutate_residue back to
// the old amino acid around the same Calpha; allatom.rs:244-384), by four lanes of a
// warp (all lanes call; live: the four lanes have a build).  The two kinds differ only
// in the backbone the side chain is built on (the current one, or the ideal one around
// the Calpha), so the builds of a warp share the side-chain loop (quad_side_chain).
// Atoms go straight into the row of prop / rej, the programs are the CTA's shared copy.
// A side-chain-only build writes the side chain's slots only (SEL_SIDE: the others stay
// as they are).
template <class L>
__device__ __forceinline__ void build_move(L& S, int r, int which, bool live) {
    const int q = threadIdx.x & 3;
    const int oa = S.aa[r];
    const int kind = S.kind[r];
    const int na = S.new_aa[r];
    const bool side_only = kind == MV_ROT || na == oa;  // side chain rebuilt on the current backbone
    const float4* cur = S.pos + (size_t)r * SLOT_STRIDE;
    float4* out = (which == SEL_PROP ? S.prop : S.rej) + (size_t)r * SLOT_STRIDE;
    const int a = which == SEL_PROP ? na : oa;
    const float2* trig = (const float2*)(S.trig + 2 * r);
    if (which == SEL_PROP) {
        const int rot = kind == MV_ROT ? S.new_rot[r] : 0;
        trig = S.rott + (kind == MV_ROT || S.rot_n[a] > 0 ? (a * 5 + rot) * 4 : N_AA * 20);
    }
    int n_bb = 4 + (a != GLY ? 1 : 0);  // N, CA, C, O[, CB]
    const int n_at = S.topo_n[a];
    const float4* bb = cur;
    if (live && !side_only) {  // ideal backbone around the Calpha with the new (or, rejected, the old) residue
        F3 at[5];
        n_bb = ideal_backbone(f3(cur[1]), a, at);
#pragma unroll
        for (int k = 0; k < 5; ++k)
            if ((k & 3) == q && k < n_bb) out[k] = make_float4(at[k].x, at[k].y, at[k].z, 0.f);
        for (int k = n_at + q; k < SLOT_STRIDE; k += 4) out[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        bb = out;
    }
    quad_side_chain(S.sct + a * SC_MAX, S.scf + a * SC_MAX, trig, bb, out, n_bb, live ? S.sc_n[a] : 0);
}

// rodrigues (allatom.rs:467-479)
__device__ __forceinline__ float4 rodrigues(float4 p, F3 o, F3 ax, float ca, float sa) {
    const F3 v = {xsub(p.x, o.x), xsub(p.y, o.y), xsub(p.z, o.z)};
    const float dot = xadd(xadd(xmul(v.x, ax.x), xmul(v.y, ax.y)), xmul(v.z, ax.z));
    const F3 cx = cross3(ax, v);
    const float omc = xsub(1.0f, ca);
    const float rx = xadd(xadd(xmul(v.x, ca), xmul(cx.x, sa)), xmul(xmul(ax.x, dot), omc));
    const float ry = xadd(xadd(xmul(v.y, ca), xmul(cx.y, sa)), xmul(xmul(ax.y, dot), omc));
    const float rz = xadd(xadd(xmul(v.z, ca), xmul(cx.z, sa)), xmul(xmul(ax.z, dot), omc));
    return make_float4(xadd(rx, o.x), xadd(ry, o.y), xadd(rz, o.z), p.w);
}

// Rotate the atoms a phi (about N-CA through CA: residue r's atoms after CA and all
// later residues) or psi move (about CA-C through C: residue r's O and all later
// residues) moves, by the angle whose cosine and sine are ca, sa; allatom.rs:397-455.
template <class L>
__device__ __noinline__ void rotate_downstream(int n, int r, bool phi, float ca, float sa) {
    L& S = an_smem<L>();
    const float4* rs = S.pos + (size_t)r * SLOT_STRIDE;
    const F3 a0 = f3(rs[phi ? 0 : 1]), a1 = f3(rs[phi ? 1 : 2]);
    const F3 axis = norm3(sub3(a1, a0));
    const F3 origin = a1;
    const int n_at_r = S.topo_n[S.aa[r]];
#pragma unroll 1
    for (int idx = threadIdx.x; idx < (n - r) * SLOT_STRIDE; idx += blockDim.x) {
        const int q = r + idx / SLOT_STRIDE, k = idx % SLOT_STRIDE;
        const bool mv = q == r ? (phi ? (k >= 2 && k < n_at_r) : k == 3) : k < S.topo_n[S.aa[q]];
        if (mv) {
            float4* p = S.pos + (size_t)q * SLOT_STRIDE + k;
            *p = rodrigues(*p, origin, axis, ca, sa);
        }
    }
}

// Sum, in order, of the coarse-grained pair terms (compute_forces, energy.rs:353-391)
// of the lane group's cnt candidates (list entries, or 0 .. cnt-1 without a list) inside
// the cutoff (with cells, beyond near_sq also in a cell next to the body's, as the
// reference probes), by the GL lanes of the group; the groups of a warp run in
// lockstep (every loop is warp-uniform, every ballot full: group masks would split the
// warp).  The group compacts the passing candidates, its lanes evaluate one pair each
// into the residue's x / y / z rows, and lanes 0..2 add one component each in order,
// four terms a load -- the pads are +0, which leaves a sum that starts at +0 unchanged.
// Scratch: rows xy (x at 0, y at AN_IN) and zi (z, then the compacted entries), 64
// floats each; entry k of a row lies at (k + 4 group) mod AN_IN, apart in banks from the
// warp's other groups.  Lanes 0..2 of the group return x, y, z.
template <int GL>
__device__ __noinline__ float group_force(int cnt, const uint16_t* list, const int4* cells, int cx, int cy, int cz,
                                          float near_sq, const CgB body, const float4* q, const float4* prm, float* xy, float* zi) {
    static_assert(AN_IN % GL == 0 && GL >= 4, "a round compacts whole group steps");
    const int lane = threadIdx.x & 31, gl = lane & (GL - 1), gshift = lane & ~(GL - 1);
    const int skew = 4 * (lane / GL);
    uint16_t* in = (uint16_t*)(zi + AN_IN);
    const float* row = gl == 0 ? xy : gl == 1 ? xy + AN_IN : zi;
    const unsigned below = (1u << gl) - 1u;
    const int mx = __reduce_max_sync(0xffffffffu, cnt);
    float s = 0.0f;
    int from = 0;
    while (from < mx) {
        int n_in = 0;
#pragma unroll 1
        for (int st = 0; st < AN_IN / GL && from < mx; ++st, from += GL) {
            const int j = from + gl;
            bool ok = false;
            int i = 0;
            if (j < cnt) {
                i = list ? list[j] : j;
                const float4 a = q[i];
                const float r_sq = xdist2(xsub(body.x, a.x), xsub(body.y, a.y), xsub(body.z, a.z));
                ok = !(r_sq > CUTOFF_SQ || r_sq < MIN_R_SQ);
                if (ok && cells && r_sq > near_sq) {  // the reference's cell test
                    const int4 ce = cells[i];
                    ok = abs((long long)ce.x - cx) <= 1 && abs((long long)ce.y - cy) <= 1 &&
                         abs((long long)ce.z - cz) <= 1;
                }
            }
            const unsigned m = __ballot_sync(0xffffffffu, ok) >> gshift & ((1u << GL) - 1u);
            if (ok) in[n_in + __popc(m & below)] = (uint16_t)i;
            n_in += __popc(m);
        }
        __syncwarp();
        const int kmax = __reduce_max_sync(0xffffffffu, n_in);
#pragma unroll 1
        for (int k = gl; k < kmax + gl; k += GL) {  // kmax / GL rounds, rounded up
            float tx = 0.0f, ty = 0.0f, tz = 0.0f;
            if (k < n_in) {
                const int i = in[k];
                cg_term_parts(body, q[i], prm[i], tx, ty, tz);
            }
            if (cnt > 0) {
                const int at = (k + skew) & (AN_IN - 1);
                xy[at] = tx;
                xy[AN_IN + at] = ty;
                zi[at] = tz;
            }
        }
        __syncwarp();
        if (gl < 3 && cnt > 0)
#pragma unroll 1
            for (int k = 0; k < kmax; k += 4) {
                const float4 t = *(const float4*)(row + ((k + skew) & (AN_IN - 1)));
                s = xadd(xadd(xadd(xadd(s, t.x), t.y), t.z), t.w);
            }
        __syncwarp();  // the rows are rewritten next round
    }
    return s;
}

// The network's choice of every mutation and (known-rotamer) rotamer move drawn
// this step and the moves' log Hastings ratios (all threads of the CTA call), one
// network pass per tile of moves.  A move changes neither the residue's environment
// nor its query (mutation: no amino-acid input; rotamer: the unchanged amino acid),
// so the reverse move's proposal is the same softmax: log q(reverse) - log q(move)
// = (y[move] - y[back]) / Tp, the normalisers cancelling.  The network comes by value:
// a reference to the kernel's copy would put it in local memory.  The biases are read
// from their shared-memory copies (staged by the kernel).
template <class L>
__device__ __noinline__ void an_learned_choices(int n, MlpDev mlp, float temp) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    L& S = an_smem<L>();
    mlp.b1 = S.mbias;  // the biases' shared-memory copies
    mlp.b2 = S.mbias + MLP_H;
    mlp.b3 = S.mbias + 2 * MLP_H;
    const MlpTile T = mlp_tile_carve(S.tile);
    const double inv_tp = 1.0 / (double)fmaxf(temp, mlp.t_prop_min);
    uint4 w[MT_WREGS];
    mlp_tile_prefetch(mlp, w);  // the first weights are on their way during the features
    if (warp == 0) {  // mutations, and rotamer moves from a known library rotamer, in residue order
        int k = 0;
        for (int b = 0; b < n; b += 32) {
            const int r = b + lane;
            const int kind = r < n ? S.kind[r] : MV_NONE;
            const bool m = kind == MV_MUT || (kind == MV_ROT && S.rot[r] >= 0);
            const unsigned bal = __ballot_sync(0xffffffffu, m);
            if (m) S.mvl[k + __popc(bal & ((1u << lane) - 1u))] = r;
            k += __popc(bal);
        }
        if (lane == 0) S.iscal[IS_NMV] = k;
    }
    __syncthreads();
    const int n_mv = S.iscal[IS_NMV];
    for (int base = 0; base < n_mv; base += MT_ROWS) {
        const int rows = min(MT_ROWS, n_mv - base);
        if (base > 0) mlp_tile_prefetch(mlp, w);
        an_tile_features(S, T, S.mvl, base, rows);
        __syncthreads();
        mlp_tile_forward(mlp, T, w, rows);
        for (int i = warp; i < rows; i += AN_WARPS) {  // one warp per row
            const int r = S.mvl[base + i];
            const bool rot = S.kind[r] == MV_ROT;
            // rotamer query: outputs 20 + j over the residue's rotamers; mutation: outputs 0..19
            const float* y = T.y + i * MT_YS + (rot ? N_AA : 0);
            const int k = warp_sample(y, rot ? S.rot_n[S.aa[r]] : N_AA, inv_tp, S.dz[r]);
            if (lane == 0) {
                const int back = rot ? S.rot[r] : S.aa[r];  // the reverse move's option
                if (rot) S.new_rot[r] = k;
                else S.new_aa[r] = k;
                if (back == CYS || (!rot && k == CYS)) S.iscal[IS_CYSMV] = 1;
                S.lhr[r] = ((double)y[k] - (double)y[back]) * inv_tp;
            }
        }
        __syncthreads();
    }
}

// Calpha energies (residue_contribution_allatom, diffusion.rs:425-463, and for Fv the
// partner chain's, :551-553) of four tasks by one warp, EL = 8 lanes each, in double:
// residue r as amino acid aa (live: the lane's task exists).  A residue still inside
// its list's skin reads the list's entries (it holds every Calpha within the cutoff);
// the others are scanned by the whole warp, one after another.  Every lane of a group
// gets its task's energy.
template <class L>
__device__ __noinline__ double task_energies(int r, int aa, bool live) {
    L& S = an_smem<L>();
    const int lane = threadIdx.x & 31, gl = lane & (EL - 1);
    const F3 ca = f3(S.pos[r * SLOT_STRIDE + 1]);
    const float4 b = S.ca_atom[aa];
    const int bhb = S.ca_hb[aa];
    const float4 cc = S.cgcentre[r];
    const float mx = ca.x - cc.x, my = ca.y - cc.y, mz = ca.z - cc.z;
    const int nl = S.cgnl[r];
    const bool ok = live && nl <= CG_LIST_MAX && mx * mx + my * my + mz * mz <= (cc.w - 0.01f) * (cc.w - 0.01f);
    constexpr int CAP = HIT_CAP * EL / 32;
    float2* hits = S.hits + (threadIdx.x >> 5) * HIT_CAP;
    double e = 0.0;  // the lane's partial sum
    int first = 0;   // number of the group's next in-cutoff Calpha
#pragma unroll 1
    for (unsigned m = __ballot_sync(0xffffffffu, live && !ok && gl == 0); m; m &= m - 1) {
        const int src = __ffs(m) - 1;
        const F3 c = {__shfl_sync(0xffffffffu, ca.x, src), __shfl_sync(0xffffffffu, ca.y, src),
                      __shfl_sync(0xffffffffu, ca.z, src)};
        const ScanSum v = warp_scan_energy<L>(c, __shfl_sync(0xffffffffu, aa, src), hits);
        if ((lane & ~(EL - 1)) == src) {
            e = v.e;
            first = v.n;
        }
    }
    __syncwarp();
    // the group's in-cutoff candidates queued (r^2, amino acid), EL at a time evaluated one
    // per lane
    const unsigned below = (1u << gl) - 1u;
    float2* q = hits + (lane / EL) * CAP;
    int n_in = 0;
    const uint16_t* list = S.cglist + r * CG_LIST_MAX;
    const float4* pos = S.env.pos;
    const uint8_t* ag_aa = S.env.aa;
    const int n_list = ok ? nl : 0, n_all = n_list + (L::FV && live ? S.env.np : 0);
    const int n_max = __reduce_max_sync(0xffffffffu, n_all);
#pragma unroll 1
    for (int j0 = 0; j0 < n_max; j0 += EL) {
        const int j = j0 + gl;
        bool in = false;
        int t = 0;
        float r_sq = 0.0f;
        if (j < n_all) {
            int i;
            float4 a;
            if (L::FV && j >= n_list) {
                i = j - n_list;
                a = S.ptq[i];
            } else {
                i = list[j];
                a = pos[i];
            }
            r_sq = xdist2(xsub(ca.x, a.x), xsub(ca.y, a.y), xsub(ca.z, a.z));
            in = !(r_sq > CUTOFF_SQ || r_sq < MIN_R_SQ);
            if (in) t = L::FV && j >= n_list ? S.ptaa[i] : ag_aa[i];
        }
        const unsigned m = __ballot_sync(0xffffffffu, in) >> (lane & ~(EL - 1)) & ((1u << EL) - 1u);
        if (in) q[n_in + __popc(m & below)] = make_float2(r_sq, __int_as_float(t));
        n_in += __popc(m);
        const int k_max = __reduce_max_sync(0xffffffffu, n_in);
        if (k_max + EL > CAP || j0 + EL >= n_max) {
            __syncwarp();
            const int k1 = (gl - first) & (EL - 1);  // entry k has the number first + k
#pragma unroll 1
            for (int k0 = 0; k0 < k_max; k0 += EL) {
                if (k0 + k1 >= n_in) continue;
                const float2 h = q[k0 + k1];
                const int a = __float_as_int(h.y);
                e += ca_pair_sum(b, bhb, S.ca_atom[a], S.ca_hb[a], h.x);
            }
            __syncwarp();
            first += n_in;
            n_in = 0;
        }
    }
#pragma unroll
    for (int o = EL / 2; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
    return e;
}

// EXT: the learned proposal and the proposal log are compiled in (a separate
// instance, so the plain kernel carries none of their registers).
// FV: one chain of each Fv candidate (fv_chain_step, diffusion.rs:560-698): the
// resident state interleaves heavy (2i) and light (2i + 1) chains, this launch steps
// chains 2 * blockIdx.x + fv_chain against the antigen and the other chain of the pair
// as it is in the state; Calpha energies gain the partner chain's contribution, the
// force its compute_forces term, and the mutation / rotamer moves follow the CDR
// flags fv_cdr (per residue) instead of the interface mask.  Draw streams + 4 * chain.
// L: the shared memory's fixed part; GL lanes per residue of the Langevin step; G, C
// staged antigen Calphas and cells (0: none).
template <class L, bool EXT, int GL>
__global__ void __launch_bounds__(L::W * 32, (L::W == 8 && L::RT == 32 && !L::LRN ? 3 : 16 / L::W))
    k_anneal(StateView st, const AgView* __restrict__ ags, StepParams p, int n_steps, uint32_t step0, int with_noise,
             const float* __restrict__ temps, int G, int C, uint32_t* __restrict__ err, long long* __restrict__ stats,
             MlpDev mlp, int learned, MlpTuple* __restrict__ tlog, unsigned long long* __restrict__ log_n,
             long long log_cap, int fv_chain, const uint8_t* __restrict__ fv_cdr) {
    constexpr int W = L::W;
    constexpr bool F32 = L::F32, FV = L::FV;
    using ACC = typename std::conditional<F32, float, double>::type;
    static_assert(!EXT || W == AN_WARPS, "the network tile takes 8 warps");
    static_assert(!L::LRN || EXT, "the learned proposal is an EXT instance");
    constexpr int NT = W * 32;               // threads of the CTA
    constexpr int RPP = NT / GL;             // residues per Langevin pass
    constexpr int BW = 2;                    // warps that build moves
    constexpr int EW = W - BW;               // warps that compute energies beside them
    L& S = an_smem<L>();
    // the staged antigen
    unsigned char* tail = reinterpret_cast<unsigned char*>(&S) + sizeof(L);
    float4* const s_cgq = (float4*)tail;
    float4* const s_cgp = s_cgq + G;
    float4* const s_agq = s_cgp + G;                   // F32 from here ..
    float4* const s_agp = s_agq + (F32 ? G : 0);
    float* const s_agx = (float*)(s_agp + (F32 ? G : 0));
    float* const s_agy = s_agx + (F32 ? anneal_xyz_len(G) : 0);
    float* const s_agz = s_agy + (F32 ? anneal_xyz_len(G) : 0);
    int* const s_cell = (int*)(s_agz + (F32 ? anneal_xyz_len(G) : 0));  // .. to here
    uint8_t* const s_aa = (uint8_t*)(s_cell + C);
    const int c = FV ? 2 * (int)blockIdx.x + fv_chain : (int)blockIdx.x;
    const uint32_t sh = FV ? 4u * (uint32_t)fv_chain : 0u;  // draw stream offset of the chain
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int r0 = st.cand_res_off[c];
    const int n = st.cand_res_off[c + 1] - r0;
    if (n <= 0 || n > L::RT) return;
    const int words = (n + 31) >> 5;  // of a residue bit mask
    const uint32_t cid = st.cand_id[c];
    const int c_ag = st.cand_ag[c];
    const int epoch = st.ag_epoch && st.cg_meta && st.cg_list && st.cg_centre ? *st.ag_epoch : -2;
    if (tid == 0) S.ag = ags[c_ag];
    __syncthreads();
    const AgView& A = S.ag;
    const int nag = A.n_res;
    const bool staged = nag <= G;
    const int ncell = A.ca_grid.nx * A.ca_grid.ny * A.ca_grid.nz + 1;
    const bool cells_staged = staged && ncell <= C;
#pragma unroll 2
    for (int i = tid; staged && i < nag; i += NT) {
        s_cgq[i] = A.ca_pq[i];
        s_cgp[i] = A.ca_prm[i];
        s_aa[i] = A.ca_aa[i];
        if (F32) {
            const float4 q = A.ca_atom[i];
            s_agq[i] = q;
            s_agp[i] = A.ca_atom_prm[i];
            s_agx[i] = q.x;
            s_agy[i] = q.y;
            s_agz[i] = q.z;
        }
    }
    if (F32 && tid == 0 && staged && (nag & 1)) s_agx[nag] = s_agy[nag] = s_agz[nag] = 1e30f;
#pragma unroll 2
    for (int i = tid; cells_staged && i < ncell; i += NT) s_cell[i] = A.ca_grid.cell_start[i];
    stage_side_chains(S.sct, S.scf, tid, NT);
#pragma unroll 1
    for (int i = tid; i < N_AA * 20 + 4; i += NT)
        S.rott[i] = i < N_AA * 20 ? (&s_rot_trig[0][0][0])[i] : make_float2(0.f, 1.f);
    for (int i = tid; i < N_AA; i += NT) {
        S.ca_atom[i] = s_ca_atom[i];
        S.res[i] = s_res[i];
        S.ca_hb[i] = s_hb_role[s_ca_type[i]];
        S.topo_n[i] = s_topo_n[i];
        S.sc_n[i] = s_sc_n[i];
        S.rot_n[i] = s_rot_n[i];
    }
    if (L::LRN && learned) {  // the network's features and epilogues read these every step
        for (int i = tid; i <= MLP_COUNT_CAP; i += NT) S.lg1p[i] = g_an_log1p[i];
        for (int i = tid; i < MLP_BIASES; i += NT)
            S.mbias[i] = i < MLP_H ? mlp.b1[i] : i < 2 * MLP_H ? mlp.b2[i - MLP_H] : mlp.b3[i - 2 * MLP_H];
    }
    // Fv: the partner chain's Calphas (it does not move during this launch)
    int np = 0;
    if (FV) {
        const int pc = c ^ 1, p0 = st.cand_res_off[pc];
        np = min(st.cand_res_off[pc + 1] - p0, L::RT);
        for (int i = tid; i < np; i += NT) {
            const float4 v = st.res_pos[(size_t)(p0 + i) * SLOT_STRIDE + 1];
            const int a = st.res_aa[p0 + i];
            const float4 q = s_ca_atom[a], rl = s_res[a];
            S.ptq[i] = make_float4(v.x, v.y, v.z, q.x);
            if (F32) S.ptp[i] = make_float4(q.y, q.z, q.w, (float)s_ca_type[a]);
            S.ptaa[i] = (uint8_t)a;
            S.pcq[i] = make_float4(v.x, v.y, v.z, rl.x);
            S.pcp[i] = make_float4(rl.y, rl.z, rl.w, 0.f);
        }
    }
    if (tid == 0) {
        S.env.pos = staged ? s_cgq : A.ca_pq;
        S.env.aa = staged ? s_aa : A.ca_aa;
        S.env.n = nag;
        S.env.np = np;
        S.iscal[IS_NTASK] = S.iscal[IS_CYSMV] = 0;
    }
#pragma unroll 2
    for (int i = tid; i < n * SLOT_STRIDE; i += NT) S.pos[i] = st.res_pos[(size_t)r0 * SLOT_STRIDE + i];
    for (int r = tid; r < n; r += NT) {
        const int a = st.res_aa[r0 + r];
        const float4 chi = st.res_chi[r0 + r];
        S.aa[r] = a;
        S.chi[r] = chi;
        S.trig[2 * r] = st.res_trig[2 * (r0 + r)];
        S.trig[2 * r + 1] = st.res_trig[2 * (r0 + r) + 1];
        // the residue's list of an earlier launch, if it was built for this antigen set and antigen
        const int4 meta = epoch >= 0 ? st.cg_meta[r0 + r] : make_int4(-1, -1, -1, -1);
        const bool kept = epoch >= 0 && meta.z == epoch && meta.y == c_ag && meta.x >= 0 && meta.x <= CG_LIST_MAX &&
                          nag <= 65536;
        S.cgnl[r] = kept ? meta.x : -1;
        S.cgcentre[r] = kept ? st.cg_centre[r0 + r] : make_float4(0.f, 0.f, 0.f, 0.f);
        S.dirty[r] = 0;
        if (EXT) {
            // rotamer index of the state: the library entry whose chi it holds, else -1
            int k = -1;
            for (int q = 0; q < s_rot_n[a] && k < 0; ++q) {
                const float4 t = s_rot_chi[a][q];
                if (t.x == chi.x && t.y == chi.y && t.z == chi.z && t.w == chi.w) k = q;
            }
            S.rot[r] = k;
        }
    }
    __syncthreads();
    for (int r = warp; r < n; r += W) {
        const int nl = S.cgnl[r];
        for (int j = lane; j < nl; j += 32) S.cglist[r * CG_LIST_MAX + j] = (uint16_t)st.cg_list[(size_t)(r0 + r) * CG_LIST_MAX + j];
    }
    if (tid == 0 && cells_staged) {  // the list builds read the staged copies through the view
        S.ag.ca_pq = s_cgq;
        S.ag.ca_prm = s_cgp;
        S.ag.ca_grid.cell_start = s_cell;
    }
    const float4* agq = staged ? s_agq : A.ca_atom;      // F32: residue order
    const float4* agp = staged ? s_agp : A.ca_atom_prm;
    const float4* cgq = staged ? s_cgq : A.ca_pq;        // grid (list) order
    const float4* cgp = staged ? s_cgp : A.ca_prm;
    // Calpha energies of the tasks 0 .. count-1, dealt over the warps w0 .. w0+nw-1 of the
    // CTA (one per warp in turn): get(k, r, aa) names task k's residue and amino acid
    // (false: none), put(k, e) takes its energy (one lane)
    auto run_tasks = [&](int w0, int nw, int count, auto get, auto put) {
        if constexpr (F32) {
            float4* stage = S.stage + warp * STAGE_CAP;
#pragma unroll 1
            for (int k = warp - w0; k < count; k += nw) {
                int r, a;
                if (!get(k, r, a)) continue;
                const F3 q = f3(S.pos[r * SLOT_STRIDE + 1]);
                ACC e = staged ? warp_contribution_pairs<ACC>(s_agx, s_agy, s_agz, agq, agp, nag, q, a, stage)
                               : warp_contribution<ACC>(agq, agp, nag, q, a, stage);
                if (FV) e = e + warp_contribution<ACC>(S.ptq, S.ptp, np, q, a, stage);
                if (lane == 0) put(k, (double)e);
            }
        } else {
#pragma unroll 1
            for (int k0 = warp - w0; k0 < count; k0 += nw * (32 / EL)) {
                const int k = k0 + nw * (lane / EL);
                int r = 0, a = 0;
                const bool live = k < count && get(k, r, a);
                const double e = task_energies<L>(live ? r : 0, live ? a : 0, live);
                if (live && (lane & (EL - 1)) == 0) put(k, e);
            }
        }
    };
    long long n_mc = 0, n_mc_acc = 0, n_bb = 0, n_bb_acc = 0;
    __syncthreads();

    float next_temp = temps ? temps[0] : p.t_hot;
#pragma unroll 1
    for (int s = 0; s < n_steps; ++s) {
        const uint32_t step = step0 + (uint32_t)s;
        const float temp = next_temp;
        if (temps && s + 1 < n_steps) next_temp = temps[s + 1];
        unsigned* const attw = S.attw + (s & 1) * MASK_WORDS;
        // ---- backbone move draws (diffusion.rs:403-405): 32 residues per warp, the last
        // warps first (with up to NT / GL - 32 / GL residues the Langevin step leaves them idle)
#pragma unroll 1
        for (int w = W - 1 - warp; w < words; w += W) {
            const int r = w * 32 + lane;
            bool att = false;
            if (r < n) {
                const U4 d = step_draw(p.seed, cid, step, STREAM_BACKBONE + sh, (uint32_t)r);
                att = u01(d.x) < p.backbone_move_p;
                if (att) {
                    const float delta = xmul(frange(d.y, -p.max_torsion_deg, p.max_torsion_deg), RADS_PER_DEG);
                    S.bb_trig[r] = torsion_trig(delta);
                }
                S.bb_phi[r] = (int)((d.z >> 31) & 1u);
                S.bb_u[r] = u01(d.w);
            }
            const unsigned m = __ballot_sync(0xffffffffu, att);
            if (lane == 0) attw[w] = m;
        }
        // ---- 1. Langevin (diffusion.rs:306-339), interface test, move draws ----
#pragma unroll 1
        for (int base = warp * (32 / GL); base < n; base += RPP) {  // whole warps
            const int gl = lane & (GL - 1);
            const int r = base + lane / GL;
            const bool live = r < n;
            const int rr = live ? r : 0;
            float4* row = S.pos + (size_t)rr * SLOT_STRIDE;
            const F3 ca = f3(row[1]);
            const int aa = S.aa[rr];
            float4 cc = S.cgcentre[rr];
            int nl = S.cgnl[rr];
            {   // lists the residues' Calphas outran (a backbone move, the drift): rebuilt by the
                // whole warp, one residue after another, with twice the skin
                const float mx = ca.x - cc.x, my = ca.y - cc.y, mz = ca.z - cc.z;
                const bool need = live && gl == 0 &&
                                  (nl < 0 || !(mx * mx + my * my + mz * mz <= (cc.w - 0.01f) * (cc.w - 0.01f)));
                const unsigned todo = __ballot_sync(0xffffffffu, need);
                if (todo) {
#pragma unroll 1
                    for (unsigned m = todo; m; m &= m - 1) {
                        const int q = __ffs(m) - 1;
                        const int rq = __shfl_sync(0xffffffffu, rr, q);
                        const F3 cq = f3(S.pos[(size_t)rq * SLOT_STRIDE + 1]);
                        const int nq = S.cgnl[rq];
                        float sq = nq < 0 ? AN_SKIN<FV> : fminf(2.0f * S.cgcentre[rq].w, AN_SKIN_MAX<FV>);
                        __syncwarp();
                        int len = CG_LIST_MAX + 1;
                        for (;;) {  // one that overflows the list (deep in the antigen) is built again with 1 A
                            if (nag <= 65536)
                                len = build_cg_list_warp<uint16_t>(A.ca_grid, A.ca_pq, cq, lane,
                                                                   S.cglist + (size_t)rq * CG_LIST_MAX, sq);
                            if (len <= CG_LIST_MAX || sq <= 1.0f) break;
                            sq = 1.0f;
                        }
                        if (lane == q) {
                            S.cgcentre[rq] = make_float4(cq.x, cq.y, cq.z, sq);
                            S.cgnl[rq] = len;
                            S.dirty[rq] = 1;
                        }
                    }
                    __syncwarp();
                    cc = S.cgcentre[rr];
                    nl = S.cgnl[rr];
                }
            }
            if (live && gl == 0 && err && (!isfinite(ca.x) || !isfinite(ca.y) || !isfinite(ca.z)))
                atomicOr(err, ERRF_NAN);
            const float4 rl = S.res[aa];
            const CgB body{ca.x, ca.y, ca.z, rl.x, rl.y, rl.z, rl.w};
            float* xy = (float*)(S.prop + (size_t)rr * SLOT_STRIDE);  // the residue's proposal rows are free here
            float* zi = (float*)(S.rej + (size_t)rr * SLOT_STRIDE);
            float fx, fy, fz;
            {
                const GridView& g = A.ca_grid;
                const int cx = cell_coord(ca.x, g.inv), cy = cell_coord(ca.y, g.inv), cz = cell_coord(ca.z, g.inv);
                const bool walk = nl > CG_LIST_MAX || cell_far(cx, cy, cz);  // no usable list: the one-lane walk
                // cells at least as wide as the cutoff: closer pairs are in adjacent cells (see k_langevin)
                const float near_sq = g.cell >= 10.0f && fabsf(ca.x) < 1e4f && fabsf(ca.y) < 1e4f && fabsf(ca.z) < 1e4f
                                          ? CG_NEAR_SQ : -1.0f;
                const uint16_t* list = S.cglist + (size_t)rr * CG_LIST_MAX;
                const float f = group_force<GL>(live && !walk ? nl : 0, list, A.ca_cell, cx, cy, cz, near_sq, body, cgq, cgp,
                                                xy, zi);
                fx = __shfl_sync(0xffffffffu, f, 0, GL);
                fy = __shfl_sync(0xffffffffu, f, 1, GL);
                fz = __shfl_sync(0xffffffffu, f, 2, GL);
                if (__any_sync(0xffffffffu, live && walk)) {
                    float wx = 0.0f, wy = 0.0f, wz = 0.0f;
                    if (live && walk && gl == 0) cg_force(A, body, wx, wy, wz);
                    __syncwarp();
                    wx = __shfl_sync(0xffffffffu, wx, 0, GL);
                    wy = __shfl_sync(0xffffffffu, wy, 0, GL);
                    wz = __shfl_sync(0xffffffffu, wz, 0, GL);
                    if (walk) {
                        fx = wx;
                        fy = wy;
                        fz = wz;
                    }
                }
            }
            if (FV) {  // VH-VL packing force: compute_forces over the partner's Calphas
                const float f = group_force<GL>(live ? np : 0, nullptr, nullptr, 0, 0, 0, 0.0f, body, S.pcq,
                                                S.pcp, xy, zi);
                fx = xadd(fx, __shfl_sync(0xffffffffu, f, 0, GL));
                fy = xadd(fy, __shfl_sync(0xffffffffu, f, 1, GL));
                fz = xadd(fz, __shfl_sync(0xffffffffu, f, 2, GL));
            }
            const float dx_c = xsub(ca.x, A.cx), dy_c = xsub(ca.y, A.cy), dz_c = xsub(ca.z, A.cz);
            const float d = fmaxf(xsqrt(xdist2(dx_c, dy_c, dz_c)), 0.001f);
            const float f_r = xdiv(xmul(-p.restraint_k, xsub(d, p.shell_radius)), d);
            fx = xadd(fx, xmul(f_r, dx_c));
            fy = xadd(fy, xmul(f_r, dy_c));
            fz = xadd(fz, xmul(f_r, dz_c));
            // one generator call per lane: lane 1 of the group draws the residue's move, the
            // others its noise
            const U4 u = step_draw(p.seed, cid, step, (gl == 1 ? STREAM_MC : STREAM_NOISE) + sh, (uint32_t)r);
            const U4 dm = {__shfl_sync(0xffffffffu, u.x, 1, GL), __shfl_sync(0xffffffffu, u.y, 1, GL),
                           __shfl_sync(0xffffffffu, u.z, 1, GL), __shfl_sync(0xffffffffu, u.w, 1, GL)};
            float nx = 0.f, ny = 0.f, nz = 0.f;
            if (with_noise) {
                const float sigma = xmul(p.noise_base, xsqrt(temp));
                nx = frange(__shfl_sync(0xffffffffu, u.x, 0, GL), -sigma, sigma);
                ny = frange(__shfl_sync(0xffffffffu, u.y, 0, GL), -sigma, sigma);
                nz = frange(__shfl_sync(0xffffffffu, u.z, 0, GL), -sigma, sigma);
            }
            const float md = p.max_disp;
            const F3 nca = {xadd(xadd(ca.x, fminf(fmaxf(xmul(p.step, fx), -md), md)), nx),
                            xadd(xadd(ca.y, fminf(fmaxf(xmul(p.step, fy), -md), md)), ny),
                            xadd(xadd(ca.z, fminf(fmaxf(xmul(p.step, fz), -md), md)), nz)};
            // set_ca_pos: delta = new - old; every atom (the Calpha included) += delta
            const F3 dl = sub3(nca, ca);
            const F3 cn = {xadd(ca.x, dl.x), xadd(ca.y, dl.y), xadd(ca.z, dl.z)};
            if (live) {
                const int n_at = S.topo_n[aa];
#pragma unroll
                for (int k = gl; k < SLOT_STRIDE; k += GL)
                    if (k < n_at) {
                        float4 v = row[k];
                        v.x = xadd(v.x, dl.x);
                        v.y = xadd(v.y, dl.y);
                        v.z = xadd(v.z, dl.z);
                        row[k] = v;
                    }
            }
            // interface residue (diffusion.rs:343-351), where the move's draw depends on it: from
            // the list while it reaches far enough around the moved Calpha, else from all
            // antigen Calphas
            bool itf = false;
            if (!FV) {
                const float mx = cn.x - cc.x, my = cn.y - cc.y, mz = cn.z - cc.z;
                const float reach = 10.0f + cc.w - 0.01f - sqrtf(mx * mx + my * my + mz * mz);
                const bool listed = nl <= CG_LIST_MAX && reach > 0.0f && p.iface_cutoff_sq <= reach * reach;
                const uint16_t* list = S.cglist + (size_t)rr * CG_LIST_MAX;
                const bool asked = live && u01(dm.x) < fmaxf(xmul(p.mutation_p, 3.0f), xmul(p.mutation_p, 0.4f));
                const int cnt = asked ? (listed ? nl : nag) : 0;
                const int mxc = __reduce_max_sync(0xffffffffu, cnt);
#pragma unroll 1
                for (int j = gl; j < mxc; j += GL) {
                    if (j >= cnt) continue;
                    const float4 a = cgq[listed ? (int)list[j] : j];
                    itf |= xdist2(xsub(cn.x, a.x), xsub(cn.y, a.y), xsub(cn.z, a.z)) < p.iface_cutoff_sq;
                }
                __syncwarp();
                const unsigned m = __ballot_sync(0xffffffffu, itf) >> (lane & ~(GL - 1));
                itf = (m & ((1u << GL) - 1u)) != 0u;
            }
            // mutation / rotamer proposal (diffusion.rs:354-399)
            if (live && gl == 0) {
                int kind = MV_NONE, new_aa = aa, new_rot = 0;
                if (FV) {
                    // CDR positions: mutation / rotamer moves (MUTATION_P * 3, ROTAMER_MOVE_P * 2);
                    // every residue without one: rotamer relaxation (ROTAMER_MOVE_P * 0.3)
                    if (fv_cdr[r0 + r] && u01(dm.x) < xmul(p.mutation_p, 3.0f)) {
                        if (u01(dm.y) < xmul(p.rotamer_move_p, 2.0f)) {
                            if (S.rot_n[aa] > 0) kind = MV_ROT;
                        } else {
                            kind = MV_MUT;
                        }
                    } else if (u01(dm.y) < xmul(p.rotamer_move_p, 0.3f) && S.rot_n[aa] > 0) {
                        kind = MV_ROT;
                    }
                } else {
                    const float eff_mut_p = itf ? xmul(p.mutation_p, 3.0f) : xmul(p.mutation_p, 0.4f);
                    const float eff_rot_p = itf ? xmul(p.rotamer_move_p, 2.0f) : p.rotamer_move_p;
                    if (u01(dm.x) < eff_mut_p) {
                        if (u01(dm.y) < eff_rot_p) {
                            if (S.rot_n[aa] > 0) kind = MV_ROT;
                        } else {
                            kind = MV_MUT;
                        }
                    }
                }
                if (kind == MV_ROT) new_rot = (int)urange(dm.z, (uint32_t)S.rot_n[aa]);
                else if (kind == MV_MUT) new_aa = (int)urange(dm.z, (uint32_t)N_AA);
                S.kind[r] = kind;
                S.new_aa[r] = new_aa;
                S.new_rot[r] = new_rot;
                S.sel[r] = SEL_KEEP;
                S.u_acc[r] = u01(dm.w);
                if (EXT) {
                    S.dz[r] = dm.z;
                    S.lhr[r] = 0.0;
                }
                if (kind != MV_NONE) {  // its two tasks (in any order: each writes its own results)
                    if (aa == CYS || new_aa == CYS) S.iscal[IS_CYSMV] = 1;
                    const int k = atomicAdd(&S.iscal[IS_NTASK], 2);
                    S.task[k] = 2 * r;
                    S.task[k + 1] = 2 * r + 1;
                }
            }
        }
        __syncthreads();
        // learned proposal: the choice of each drawn move comes from the network
        // (same draw d.z, inverse CDF) and the move carries its Hastings ratio
        if constexpr (L::LRN) {
            if (learned && temp <= mlp.t_max) an_learned_choices<L>(n, mlp, temp);
        }
        // ---- 2. proposals and rejection rebuilds on the last two warps (four lanes each), on
        // the others the Calpha energies before / after each move and those of the residues
        // the first backbone move starts from; without a Cys among the moves the decisions
        // need no built atom and follow the energies while the builds still run ----
        const bool cysmv = S.iscal[IS_CYSMV] != 0;
        int first_att = n;
#pragma unroll 1
        for (int w = words - 1; w >= 0; --w)
            if (const unsigned m = attw[w]) first_att = w * 32 + __ffs(m) - 1;
        {
            const int ntask = S.iscal[IS_NTASK];
            if (warp >= EW) {  // proposals on one, rejections on the other
#pragma unroll 1
                for (int k0 = warp - EW; k0 < ntask; k0 += 8 * BW) {
                    const int k = k0 + BW * (lane >> 2);
                    const int t = S.task[k < ntask ? k : 0];
                    build_move(S, t >> 1, (t & 1) ? SEL_REJ : SEL_PROP, k < ntask);
                }
            } else {
                run_tasks(
                    0, EW, ntask + (n - first_att),
                    [&](int k, int& r, int& a) {
                        if (k >= ntask) {
                            r = first_att + (k - ntask);
                            a = S.aa[r];
                            return S.kind[r] == MV_NONE;
                        }
                        const int t = S.task[k];
                        r = t >> 1;
                        const int oa = S.aa[r];
                        a = t & 1 ? S.new_aa[r] : oa;
                        return !((t & 1) && a == oa);  // same Calpha, same amino acid: same energy
                    },
                    [&](int k, double e) {
                        if (k >= ntask) {
                            S.c_cur[first_att + (k - ntask)] = e;
                            return;
                        }
                        const int t = S.task[k], r = t >> 1;
                        if (t & 1) {
                            S.c_new[r] = e;
                        } else {
                            S.c_old[r] = e;
                            if (S.new_aa[r] == S.aa[r]) S.c_new[r] = e;
                        }
                    });
            }
        }
        if (cysmv) __syncthreads();
        else if (warp < EW) asm volatile("bar.sync 1, %0;" ::"n"(EW * 32) : "memory");
        // the sweep's decisions, by warp 0 (applied after the barrier: the builds still read
        // the state)
        if (warp == 0) {
            int ncys = 0;
            bool any = first_att < n;  // a backbone move needs the disulfide energy too
#pragma unroll 1
            for (int w = 0; w < words; ++w) {
                const int r = w * 32 + lane;
                const int kd = r < n ? S.kind[r] : MV_NONE;
                const bool cys = r < n && S.aa[r] == CYS;
                const bool mc = kd != MV_NONE && (cys || S.new_aa[r] == CYS);
                const unsigned bc = __ballot_sync(0xffffffffu, cys), bx = __ballot_sync(0xffffffffu, mc);
                any |= __any_sync(0xffffffffu, kd != MV_NONE);
                if (lane == 0) {
                    S.cysw[w] = bc;
                    S.mxw[w] = bx;
                }
                ncys += __popc(bc);
            }
            __syncwarp();
            ACC D = 0;
            if (any && ncys >= 2)
                D = warp_disulfide<L, ACC>(true, words, -1);
            auto settle = [&](int r, bool side, bool acc, ACC de) {  // one lane
                ++n_mc;
                n_mc_acc += acc;
                if (EXT && tlog) S.d_turn[r] = (double)de;
                S.sel[r] = (acc ? SEL_PROP : SEL_REJ) | (side ? SEL_SIDE : 0);
                S.c_cur[r] = acc ? S.c_new[r] : S.c_old[r];
            };
#pragma unroll 1
            for (int w = 0; w < words; ++w) {  // moves without a Cys: the disulfide energy of their turn
                const int r = w * 32 + lane;
                if (r < n) S.d_turn[r] = (double)D;
            }
#pragma unroll 1
            for (int wx = 0; wx < words; ++wx)
#pragma unroll 1
                for (unsigned x = S.mxw[wx]; x; x &= x - 1) {  // the moves that involve a Cys, in residue order
                    const int r = wx * 32 + __ffs(x) - 1;
                    const unsigned bit = 1u << (r & 31);
                    const int kind = S.kind[r], oa = S.aa[r], na = S.new_aa[r];
                    const int ncys_new = ncys + (na == CYS) - (oa == CYS);
                    ACC Dn = 0;
                    __syncwarp();
                    if (lane == 0) S.cysw[wx] = na == CYS ? S.cysw[wx] | bit : S.cysw[wx] & ~bit;
                    __syncwarp();
                    if (ncys_new >= 2)
                        Dn = warp_disulfide<L, ACC>(true, words, r);
                    const ACC old_e = (ACC)S.c_old[r] + D;
                    const ACC new_e = (ACC)S.c_new[r] + Dn;
                    const double lhr = EXT ? S.lhr[r] : 0.0;
                    const bool acc = mh_accept(new_e - old_e, temp, S.u_acc[r], lhr);
                    __syncwarp();
                    if (lane == 0) {
                        if (!acc) S.cysw[wx] = oa == CYS ? S.cysw[wx] | bit : S.cysw[wx] & ~bit;
                        settle(r, kind == MV_ROT || na == oa, acc, new_e - old_e);
                    }
                    __syncwarp();
                    if (acc) {
                        D = Dn;
                        ncys = ncys_new;
                    } else if (oa == CYS && ncys >= 2) {  // SG rebuilt
                        D = warp_disulfide<L, ACC>(true, words, -1);
                    }
#pragma unroll 1
                    for (int w = wx; w < words; ++w) {
                        const int q = w * 32 + lane;
                        if (q > r && q < n) S.d_turn[q] = (double)D;
                    }
                }
#pragma unroll 1
            for (int w = 0; w < words; ++w) {  // the others, each by its lane
                const int r = w * 32 + lane;
                const int kind = r < n ? S.kind[r] : MV_NONE;
                if (kind == MV_NONE || (S.mxw[w] >> lane & 1u)) continue;
                const int na = S.new_aa[r];
                const ACC Dr = (ACC)S.d_turn[r];
                const ACC old_e = (ACC)S.c_old[r] + Dr;
                const ACC new_e = (ACC)S.c_new[r] + Dr;
                const double lhr = EXT ? S.lhr[r] : 0.0;
                const bool acc = mh_accept(new_e - old_e, temp, S.u_acc[r], lhr);
                settle(r, kind == MV_ROT || na == S.aa[r], acc, new_e - old_e);
            }
            __syncwarp();
            if (EXT && tlog) {  // the log: this step's decisions in residue order
                int total = 0;
#pragma unroll 1
                for (int w = 0; w < words; ++w) {
                    const int r = w * 32 + lane;
                    total += __popc(__ballot_sync(0xffffffffu, r < n && S.kind[r] != MV_NONE));
                }
                unsigned long long slot = 0;
                if (lane == 0 && total) slot = atomicAdd(log_n, (unsigned long long)total);
                slot = __shfl_sync(0xffffffffu, slot, 0);
#pragma unroll 1
                for (int w = 0; w < words; ++w) {
                    const int r = w * 32 + lane;
                    const int kind = r < n ? S.kind[r] : MV_NONE;
                    const unsigned m = __ballot_sync(0xffffffffu, kind != MV_NONE);
                    const long long at = (long long)slot + __popc(m & ((1u << lane) - 1u));
                    slot += __popc(m);
                    if (kind == MV_NONE || at >= log_cap) continue;
                    const float4 ca = S.pos[r * SLOT_STRIDE + 1];
                    MlpTuple t;
                    t.x = ca.x; t.y = ca.y; t.z = ca.z;
                    t.delta_e = (float)(ACC)S.d_turn[r];
                    t.cand = c;
                    t.log_ratio = (float)S.lhr[r];
                    t.residue = (int16_t)r;
                    t.aa = (uint8_t)S.aa[r];
                    t.action = (uint8_t)(kind == MV_MUT ? S.new_aa[r] : N_AA + S.new_rot[r]);
                    t.antigen = (uint8_t)st.cand_ag[c];
                    t.accepted = (S.sel[r] & 3) == SEL_PROP ? 1 : 0;
                    t.pad[0] = t.pad[1] = 0;
                    tlog[at] = t;
                }
            }
            if (lane == 0) {
                S.dscal = (double)D;
                S.iscal[IS_DVALID] = any;
            }
        }
        __syncthreads();
#pragma unroll 1
        for (int i = tid; i < n * SLOT_STRIDE; i += NT) {
            const int r = i / SLOT_STRIDE, k = i % SLOT_STRIDE;
            const int sl = S.sel[r];
            if (sl == SEL_KEEP) continue;
            if (sl & SEL_SIDE) {
                const int a = S.aa[r];
                if (k < 4 + (a != GLY ? 1 : 0) || k >= S.topo_n[a]) continue;
            }
            S.pos[i] = (sl & SEL_PROP ? S.prop : S.rej)[i];
        }
#pragma unroll 1
        for (int r = tid; r < n; r += NT) {  // accepted moves (side-chain-only ones keep the amino acid)
            if ((S.sel[r] & 3) != SEL_PROP) continue;
            const int na = S.new_aa[r], rot = S.new_rot[r];
            const bool has = S.rot_n[na] > 0;
            if (EXT) S.rot[r] = S.kind[r] == MV_ROT ? rot : (has ? 0 : -1);
            S.aa[r] = na;
            S.chi[r] = has ? s_rot_chi[na][rot] : make_float4(0.f, 0.f, 0.f, 0.f);
            const float2* t = S.rott + (has ? (na * 5 + rot) * 4 : N_AA * 20);
            S.trig[2 * r] = make_float4(t[0].x, t[0].y, t[1].x, t[1].y);
            S.trig[2 * r + 1] = make_float4(t[2].x, t[2].y, t[3].x, t[3].y);
        }
        if (tid == 0) S.iscal[IS_NTASK] = S.iscal[IS_CYSMV] = 0;
        __syncthreads();

        // ---- 3. backbone phi/psi moves (diffusion.rs:403-418) ----
        int last_cys = -1, stale = n;  // stale: residues from here on have no current Calpha energy
        if (first_att < n)
#pragma unroll 1
            for (int w = 0; w < words; ++w)
                if (const unsigned m = S.cysw[w]) last_cys = w * 32 + 31 - __clz(m);
#pragma unroll 1
        for (int wa = first_att < n ? first_att >> 5 : words; wa < words; ++wa)
#pragma unroll 1
            for (unsigned at = attw[wa]; at; at &= at - 1) {
                const int r = wa * 32 + __ffs(at) - 1;
                const bool phi = S.bb_phi[r] != 0;
                const bool cys_down = r <= last_cys;  // a Cys at or after r: the disulfide term can change
                if (stale < n) {  // after a rejected move: energies of residues r..n, and the disulfide energy
                    if (warp == W - 1 && !S.iscal[IS_DVALID]) {
                        const ACC D = warp_disulfide<L, ACC>(false, words, -1);
                        if (lane == 0) {
                            S.dscal = (double)D;
                            S.iscal[IS_DVALID] = 1;
                        }
                    }
                    run_tasks(
                        0, W, n - r,
                        [&](int k, int& i, int& a) {
                            i = r + k;
                            a = S.aa[i];
                            return true;
                        },
                        [&](int k, double e) { S.c_cur[r + k] = e; });
                    stale = n;
                    __syncthreads();
                }
                const float4 bt = S.bb_trig[r];
                rotate_downstream<L>(n, r, phi, bt.x, bt.y);
                __syncthreads();
                run_tasks(
                    0, W, n - r - 1,
                    [&](int k, int& i, int& a) {
                        i = r + 1 + k;
                        a = S.aa[i];
                        return true;
                    },
                    [&](int k, double e) { S.c_new[r + 1 + k] = e; });
                __syncthreads();
                if (warp == 0) {
                    ACC Dn = (ACC)S.dscal;
                    if (cys_down)
                        Dn = warp_disulfide<L, ACC>(false, words, -1);
                    bool acc;
                    if constexpr (F32) {  // the reference's sequential f32 sums, on every lane
                        ACC old_e = 0, new_e = 0;
#pragma unroll 1
                        for (int i = r; i < n; ++i) old_e += (ACC)S.c_cur[i];
                        old_e += (ACC)S.dscal;
                        new_e += (ACC)S.c_cur[r];
#pragma unroll 1
                        for (int i = r + 1; i < n; ++i) new_e += (ACC)S.c_new[i];
                        new_e += Dn;
                        acc = mh_accept(new_e - old_e, temp, S.bb_u[r], 0.0);
                    } else {
                        double old_e = 0.0, new_e = 0.0;
#pragma unroll 1
                        for (int i = r + lane; i < n; i += 32) {
                            old_e += S.c_cur[i];
                            new_e += i == r ? S.c_cur[i] : S.c_new[i];
                        }
#pragma unroll
                        for (int o = 16; o > 0; o >>= 1) {
                            old_e += __shfl_xor_sync(0xffffffffu, old_e, o);
                            new_e += __shfl_xor_sync(0xffffffffu, new_e, o);
                        }
                        acc = mh_accept((new_e + (double)Dn) - (old_e + S.dscal), temp, S.bb_u[r], 0.0);
                    }
                    __syncwarp();
                    if (lane == 0) {
                        ++n_bb;
                        n_bb_acc += acc;
                        if (acc) S.dscal = (double)Dn;
                        else if (cys_down) S.iscal[IS_DVALID] = 0;
                        S.iscal[IS_DECISION] = acc;
                    }
                }
                __syncthreads();
                if (S.iscal[IS_DECISION]) {
#pragma unroll 1
                    for (int i = r + 1 + tid; i < n; i += NT) S.c_cur[i] = S.c_new[i];
                } else {
                    rotate_downstream<L>(n, r, phi, bt.z, bt.w);
                    stale = r + 1;
                }
                __syncthreads();
            }
    }

#pragma unroll 1
    for (int i = tid; i < n * SLOT_STRIDE; i += NT) st.res_pos[(size_t)r0 * SLOT_STRIDE + i] = S.pos[i];
#pragma unroll 1
    for (int r = tid; r < n; r += NT) {
        st.res_aa[r0 + r] = (uint8_t)S.aa[r];
        st.res_chi[r0 + r] = S.chi[r];
        st.res_trig[2 * (r0 + r)] = S.trig[2 * r];
        st.res_trig[2 * (r0 + r) + 1] = S.trig[2 * r + 1];
    }
    for (int r = warp; epoch >= 0 && r < n; r += W) {  // lists built here, for the next launch
        if (!S.dirty[r]) continue;
        const int nl = S.cgnl[r];
        for (int j = lane; j < min(nl, CG_LIST_MAX); j += 32)
            st.cg_list[(size_t)(r0 + r) * CG_LIST_MAX + j] = S.cglist[r * CG_LIST_MAX + j];
        if (lane == 0) {
            st.cg_centre[r0 + r] = S.cgcentre[r];
            // the gradient steps take a kept list's skin for at least CG_SKIN: a narrower one stays here
            st.cg_meta[r0 + r] = make_int4(S.cgcentre[r].w >= CG_SKIN ? nl : -1, c_ag, epoch, 0);
        }
    }
    if (stats && (n_mc || n_bb)) {  // the decisions are spread over the lanes of warp 0
        atomicAdd((unsigned long long*)&stats[4 * c], (unsigned long long)n_mc);
        atomicAdd((unsigned long long*)&stats[4 * c + 1], (unsigned long long)n_mc_acc);
        atomicAdd((unsigned long long*)&stats[4 * c + 2], (unsigned long long)n_bb);
        atomicAdd((unsigned long long*)&stats[4 * c + 3], (unsigned long long)n_bb_acc);
    }
}

// The Metropolis energy of every resident candidate, the energy whose changes
// decide the mutation / rotamer / backbone moves: the sum over its residues of
// residue_contribution_allatom (diffusion.rs:425-463) plus disulfide_energy
// (allatom.rs:155-180), f32 terms summed in double in residue order (the default
// accumulation of k_anneal).  One CTA per candidate, one warp per residue.
__global__ void __launch_bounds__(AN_THREADS) k_mc_energy(StateView st, const AgView* __restrict__ ags,
                                                          double* __restrict__ out) {
    __shared__ float4 s_stage[AN_WARPS * STAGE_CAP];
    __shared__ double s_e[AN_THREADS];
    __shared__ double s_total;
    const int c = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int r0 = st.cand_res_off[c], n = st.cand_res_off[c + 1] - r0;
    const AgView& A = ags[st.cand_ag[c]];
    if (tid == 0) s_total = 0.0;
    for (int base = 0; base < n; base += AN_THREADS) {
        const int m = min(AN_THREADS, n - base);
        for (int i = warp; i < m; i += AN_WARPS) {
            const int r = r0 + base + i;
            const double e = warp_contribution<double>(A.ca_atom, A.ca_atom_prm, A.n_res,
                                                       f3(st.res_pos[(size_t)r * SLOT_STRIDE + 1]), st.res_aa[r],
                                                       s_stage + warp * STAGE_CAP);
            if (lane == 0) s_e[i] = e;
        }
        __syncthreads();
        if (tid == 0)
            for (int i = 0; i < m; ++i) s_total += s_e[i];
        __syncthreads();
    }
    if (tid == 0) {
        double d = 0.0;
        for (int i = 0; i < n; ++i) {
            if (st.res_aa[r0 + i] != CYS) continue;
            const float4 pi = st.res_pos[(size_t)(r0 + i) * SLOT_STRIDE + 5];
            for (int j = i + 1; j < n; ++j) {
                if (st.res_aa[r0 + j] != CYS) continue;
                const float4 pj = st.res_pos[(size_t)(r0 + j) * SLOT_STRIDE + 5];
                const float dd = xsqrt(xdist2(xsub(pi.x, pj.x), xsub(pi.y, pj.y), xsub(pi.z, pj.z)));
                if (dd > 4.0f) continue;
                const float z = xdiv(xsub(dd, 2.05f), 0.4f);
                d -= (double)xmul(4.0f, mc_exp(xmul(xmul(-0.5f, z), z)));
            }
        }
        out[c] = s_total + d;
    }
}

void launch_mc_energy(cudaStream_t s, const StateView& st, const AgView* ags, double* out) {
    if (st.n_cand > 0) k_mc_energy<<<st.n_cand, AN_THREADS, 0, s>>>(st, ags, out);
}

cudaError_t launch_anneal(cudaStream_t s, const StateView& st, const AgView* ags, const StepParams& p, int n_steps,
                          uint32_t step0, int with_noise, const float* temps, int accumulate, int max_res,
                          int max_ag_res, int max_cells, uint32_t* err, long long* stats, const AnnealExtras& x,
                          int fv_chain, const uint8_t* fv_cdr) {
    if (st.n_cand <= 0 || n_steps <= 0 || max_res <= 0) return cudaSuccess;
    if (max_res > ANNEAL_MAX_RES) return cudaErrorInvalidValue;
    const bool fv = fv_chain >= 0, f32 = accumulate == 1;
    const bool learned = x.learned && !fv;
    const bool ext = !fv && (x.learned || x.log);
    const int grid = fv ? st.n_cand / 2 : st.n_cand;
    if (grid <= 0) return cudaSuccess;
    int dev = 0, sms = 148, smem_max = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    // 16 warps per candidate while every candidate has an SM of its own (64 candidates: 600
    // steps in 9.5 ms, with 8 warps 11.1), else 8 and several candidates per SM (1024
    // candidates, 60 steps: 4.2 ms, with 16 warps 6.7; three CTAs of 80 registers per SM
    // for up to 32 residues 4.2, two of 128 registers 4.35): a step is a chain of latencies
    // that more warps shorten only a little.  The network path takes 8 warps.
    const int warps = ext || grid > sms ? 8 : 16;
    auto run = [&](auto kern, size_t fixed) -> cudaError_t {
        // the antigen and its cells are staged when they fit
        int G = max_ag_res <= AG_STAGE_MAX ? max_ag_res : 0;
        if (fixed + an_tail_bytes(G, 0, f32) > (size_t)smem_max) G = 0;
        int C = G && max_cells <= CELL_STAGE_MAX ? max_cells : 0;
        if (fixed + an_tail_bytes(G, C, f32) > (size_t)smem_max) C = 0;
        const size_t sm = fixed + an_tail_bytes(G, C, f32);
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
        if (e) return e;
        kern<<<grid, warps * 32, sm, s>>>(st, ags, p, n_steps, step0, with_noise, temps, G, C, err, stats, x.mlp,
                                 learned ? 1 : 0, x.log, x.log_n, x.log_cap, fv ? fv_chain : 0, fv_cdr);
        return cudaSuccess;
    };
    cudaError_t e;
#define BINDER_AN1(RT, W, F, LRN, FV, EXT, GL) run(k_anneal<AnSmem<RT, W, F, LRN, FV>, EXT, GL>, sizeof(AnSmem<RT, W, F, LRN, FV>))
#define BINDER_AN(F)                                                                       \
    (fv ? (warps == 16 ? BINDER_AN1(128, 16, F, false, true, false, 4)                     \
                       : BINDER_AN1(128, 8, F, false, true, false, 4))                     \
     : ext ? (max_res <= 32   ? BINDER_AN1(32, 8, F, true, false, true, 8)                 \
              : max_res <= 64 ? BINDER_AN1(64, 8, F, true, false, true, 4)                 \
                              : BINDER_AN1(128, 8, F, true, false, true, 4))               \
     : warps == 16 ? (max_res <= 32   ? BINDER_AN1(32, 16, F, false, false, false, 16)     \
                      : max_res <= 64 ? BINDER_AN1(64, 16, F, false, false, false, 8)      \
                                      : BINDER_AN1(128, 16, F, false, false, false, 4))    \
                   : (max_res <= 32   ? BINDER_AN1(32, 8, F, false, false, false, 8)       \
                      : max_res <= 64 ? BINDER_AN1(64, 8, F, false, false, false, 4)       \
                                      : BINDER_AN1(128, 8, F, false, false, false, 4)))
    e = f32 ? BINDER_AN(true) : BINDER_AN(false);
#undef BINDER_AN
#undef BINDER_AN1
    if (e) return e;
    return cudaGetLastError();
}

}  // namespace binder
