// score.cuh — the all-atom pair energy of one group of candidate atoms (a residue,
// or a few consecutive GpuAtoms) against a resident antigen, warp-wide: the device
// code shared by the scoring kernels (k_score.cu) and the post-search kernels
// (k_post.cu).  Pair math: the LJ/Coulomb/hydrophobic part of
// interaction_energy_atoms_breakdown (energy.rs:261-301), with H-bond
// (energy.rs:303-307, 32-39) and EEF1 solvation (solvation.rs:34-84) when FULL.
// f32 pair terms with rsqrt, per-lane compensated (Kahan) sums.
//
// Each translation unit that includes this header owns a copy of the constant
// tables and fills it with score_tables_init() (no relocatable device code).
#pragma once

#include "kernels.h"

namespace binder {

static __device__ float4 g_slot_prm[N_AA][SLOT_STRIDE];  // q*sqrt(332), r_min_half, sqrt(eps), hydrophobic
static __device__ int g_slot_type[N_AA][SLOT_STRIDE];
static __constant__ int c_topo_n[N_AA];
static __constant__ float4 c_eef1[16];  // dg_ref, vol, lambda, 1/(PI32*lambda^3)
static __constant__ int c_hb[16];       // bit0 donor, bit1 acceptor

static const float SQRT_COULOMB_K = 18.220867f;  // sqrt(332) in f32

// Fills this translation unit's copy of the tables.
static cudaError_t score_tables_init() {
    float4 slot[N_AA][SLOT_STRIDE];
    int stype[N_AA][SLOT_STRIDE];
    for (int a = 0; a < N_AA; ++a)
        for (int k = 0; k < SLOT_STRIDE; ++k) {
            if (k < BT_TOPO_N[a]) {
                int t = BT_SLOT_TYPE[a][k];
                slot[a][k] = make_float4(BT_SLOT_Q[a][k] * SQRT_COULOMB_K, BT_NB[t][0], sqrtf(BT_NB[t][1]),
                                         BT_SLOT_HYD[a][k] == 1 ? 1.0f : 0.0f);
                stype[a][k] = t;
            } else {
                slot[a][k] = make_float4(0.f, 0.f, 0.f, 0.f);
                stype[a][k] = 0;
            }
        }
    float4 eef[16];
    int hb[16];
    for (int t = 0; t < 16; ++t) {
        float lam = BT_EEF1[t][2];
        eef[t] = make_float4(BT_EEF1[t][0], BT_EEF1[t][1], lam, 1.0f / (PI32 * (lam * lam * lam)));
        hb[t] = BT_HB[t];
    }
    cudaError_t e;
    if ((e = cudaMemcpyToSymbol(g_slot_prm, slot, sizeof(slot))) != cudaSuccess) return e;
    if ((e = cudaMemcpyToSymbol(g_slot_type, stype, sizeof(stype))) != cudaSuccess) return e;
    if ((e = cudaMemcpyToSymbol(c_topo_n, BT_TOPO_N, sizeof(BT_TOPO_N))) != cudaSuccess) return e;
    if ((e = cudaMemcpyToSymbol(c_eef1, eef, sizeof(eef))) != cudaSuccess) return e;
    return cudaMemcpyToSymbol(c_hb, hb, sizeof(hb));
}

struct AtomIn {
    float x, y, z, qs, rmh, se, h;
};

struct Acc {
    float s, c;      // Kahan sum and compensation
    float abs_s;     // sum of |pair terms| (condition number), plain f32
    float fx, fy, fz;
    int pairs;
};

template <bool KAHAN>
__device__ __forceinline__ void acc_add(Acc& a, float v) {
    if (KAHAN) {
        float y = v - a.c;
        float t = a.s + y;
        a.c = (t - a.s) - y;
        a.s = t;
    } else {
        a.s += v;
    }
}

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_sum_f(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ bool finite3(float x, float y, float z) { return isfinite(x) && isfinite(y) && isfinite(z); }

// Fixed-order CTA reduction of one double per warp; thread 0 gets the total.
template <int NW>
__device__ __forceinline__ double cta_sum(double v, double* sm, int lane, int warp) {
    v = warp_sum_d(v);
    if (lane == 0) sm[warp] = v;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < NW; ++w) t += sm[w];
    __syncthreads();
    return t;
}

__device__ __forceinline__ float warp_max_f(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// ---- grouped scoring: one warp per group of <= 16 nearby candidate atoms ----------
// A group (a residue of the resident state, or a few consecutive GpuAtoms) sits in
// shared memory.  The warp takes the antigen's blocks of 32 atoms whose boxes come within
// 10 A + group radius of the group centre (warp-uniform loop, one atom per lane), keeps the
// atoms that pass a sphere test in a per-warp queue, and evaluates full batches of 32 queued
// atoms against every group atom — so the pair math never runs on idle lanes.  Every lane
// visits its antigen atoms in increasing grid order, which keeps the sums deterministic.
constexpr int GMAX = 16;

// Two group atoms side by side, as group_pairs reads them (16-byte loads, both atoms'
// values of a field one 8-byte word): coordinates, r_min_half, sqrt(epsilon),
// charge * sqrt(332), hydrophobic.  Entries past the group hold GROUP_PAD coordinates
// and zero parameters (finite terms, never added).  nz holds -0 (f2_dist2).
constexpr float GROUP_PAD = 1e30f;  // its squared distance to any atom overflows to +inf
struct __align__(16) GroupTwo {
    float x[2], y[2], z[2], rm[2], se[2], qs[2], hy[2], nz[2];
};

struct GroupSmem {
    float4 pos[GMAX];  // x, y, z, q*sqrt(332)
    float4 prm[GMAX];  // r_min_half, sqrt(epsilon), hydrophobic, AMBER type
    GroupTwo two[GMAX / 2];
    int q[64];         // queued antigen atom indices
};
// FULL scoring: the group atoms' EEF1 parameters (c_eef1), reciprocal lambdas and H-bond
// roles, looked up once per group.
struct GroupFull {
    float4 eef[GMAX];
    float rl[GMAX];
    int hb[GMAX];
};

// r / d, correctly rounded, from y = RN(1 / d): q = RN(r y), then one correction by the
// exact remainder (P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", 1990).  For the five divisors this is used with (the EEF1
// lambdas 3.15, 3.5, 3.7, 3.9 and the H-bond sigma 0.35) it equals the IEEE quotient for
// every float |r| in [2^-60, 16) and 0 (k_div_selftest compares all of them); three
// operations instead of a division's dozen.
__device__ __forceinline__ float div_by(float r, float d, float y) {
    const float q = __fmul_rn(r, y);
    return __fmaf_rn(__fmaf_rn(-d, q, r), y, q);
}

__device__ __forceinline__ void group_xyz(GroupSmem& s, int lane, int n, float x, float y, float z) {
    if (lane >= GMAX) return;
    GroupTwo& g = s.two[lane >> 1];
    const int i = lane & 1;
    g.x[i] = lane < n ? x : GROUP_PAD;
    g.y[i] = lane < n ? y : GROUP_PAD;
    g.z[i] = lane < n ? z : GROUP_PAD;
    g.nz[i] = -0.0f;
}
__device__ __forceinline__ void group_prm(GroupSmem& s, int lane, int n, float qs, float rmh, float se, float hy) {
    if (lane >= GMAX) return;
    GroupTwo& g = s.two[lane >> 1];
    const int i = lane & 1;
    g.qs[i] = lane < n ? qs : 0.0f;
    g.rm[i] = lane < n ? rmh : 0.0f;
    g.se[i] = lane < n ? se : 0.0f;
    g.hy[i] = lane < n ? hy : 0.0f;
}

// The H-bond (energy.rs:303-307) and EEF1 solvation (solvation.rs:34-50) terms of a pair
// within the cutoff, added to e: ei, yi the antigen atom's EEF1 parameters and reciprocal
// lambda, ej, yj the candidate atom's; hb = they can form an H-bond.
__device__ __forceinline__ float full_terms(float e, bool hb, const float4& ei, float yi, const float4& ej, float yj,
                                            float r2, float ir) {
    if (hb && r2 <= HB_CUTOFF_SQ) {
        const float z = div_by(r2 * ir - HB_R0, HB_SIGMA, 1.0f / HB_SIGMA);
        e += -HB_DEPTH * expf(-0.5f * z * z);
    }
    if (r2 < SOLV_CUTOFF_SQ && !(ej.y == 0.0f && ej.x == 0.0f)) {
        const float r = r2 * ir;
        const float xi = div_by(r, ei.z, yi), xj = div_by(r, ej.z, yj);
        const float pi = ei.x * ej.y * expf(-(xi * xi)), pj = ej.x * ei.y * expf(-(xj * xj));
        e -= __fmaf_rn(pj, ej.w, __fmul_rn(pi, ei.w));
    }
    return e;
}
// donor / acceptor roles of two atoms that make an H-bond (bit 0 donor, bit 1 acceptor)
__device__ __forceinline__ bool hb_pair(int a, int b) { return (a & ((b & 1) << 1 | (b >> 1 & 1))) != 0; }

// Energy of one pair within the cutoff (r2: the reference's rounding of r^2):
// candidate atom b / bp, antigen atom a / ap, each (x, y, z, q sqrt(332)) and
// (r_min_half, sqrt(epsilon), hydrophobic, AMBER type).  LJ + Coulomb + hydrophobic
// (energy.rs:269-301); ir = 1 / r for the further terms.
__device__ __forceinline__ float pair_base(const float4& b, const float4& bp, const float4& a, const float4& ap,
                                           float r2, float& ir) {
    ir = rsqrt_normal(r2);
    const float ir2 = ir * ir;
    const float R = bp.x + ap.x;
    const float s2 = R * R * ir2;
    const float s6 = s2 * s2 * s2;
    const float hyd = (r2 < HYDRO_CUTOFF_SQ) ? HYDRO_BONUS * (bp.z * ap.z) : 0.0f;
    const float le = __fmul_rn(bp.y, ap.y), ls = __fmul_rn(s6, s6 - 2.0f), qq = __fmul_rn(b.w, a.w);
    return __fmaf_rn(qq, ir, __fmul_rn(le, ls)) + hyd;
}

// One antigen atom (this lane's) against the n group atoms in shared memory, two
// group atoms per step: dx = b - a in packed f32x2 arithmetic, r^2 = (dx*dx + dy*dy)
// + dz*dz with the reference's roundings (never fused), hence its pair set;
// the terms of the pairs within the cutoff (packed) are added in group-atom order.
// Returns the atom's sum over the group (f32, group-atom order).
template <bool FULL, bool ABS, bool COUNT>
__device__ __forceinline__ float group_pairs(const float4* __restrict__ pq, const float4* __restrict__ prm,
                                            const GroupSmem& s, const GroupFull* gf, int n, int idx, Acc& acc) {
    static_assert(!FULL || !ABS, "the full energy has no absolute sum");
    const float4 a = __ldg(&pq[idx]);
    const float4 ap = __ldg(&prm[idx]);
    float part = 0.0f, pabs = 0.0f;
    int np = 0;
    // FULL: this antigen atom's parameters, once for all group atoms (the type is the
    // lane's: looked up per pair, its constant-table rows were fetched one distinct type
    // after another)
    float4 ei = make_float4(0.f, 0.f, 0.f, 0.f);
    float yi = 0.0f;
    int ahb = 0;
    if (FULL) {
        const int at = (int)ap.w;
        ei = c_eef1[at];
        yi = __frcp_rn(ei.z);
        ahb = c_hb[at];
    }
    auto term = [&](int j, float r2) {
        float ir;
        const float e = pair_base(s.pos[j], s.prm[j], a, ap, r2, ir);
        part += full_terms(e, hb_pair(gf->hb[j], ahb), ei, yi, gf->eef[j], gf->rl[j], r2, ir);
        if (COUNT) ++np;
    };
    const uint64_t ax = f2_pack(a.x, a.x), ay = f2_pack(a.y, a.y), az = f2_pack(a.z, a.z);
    const uint64_t aq = f2_pack(a.w, a.w), arm = f2_pack(ap.x, ap.x), ase = f2_pack(ap.y, ap.y);
    const uint64_t ahy = f2_pack(HYDRO_BONUS * ap.z, HYDRO_BONUS * ap.z), two = f2_pack(2.0f, 2.0f);
    const uint64_t neg0 = *(const uint64_t*)s.two[0].nz;
#pragma unroll 1
    for (int j = 0; j < n; j += 2) {
        const ulonglong2* g = (const ulonglong2*)&s.two[j >> 1];
        const ulonglong2 xy = g[0], zr = g[1];
        const uint64_t dx = f2_sub(xy.x, ax);
        const uint64_t dy = f2_sub(xy.y, ay);
        const uint64_t dz = f2_sub(zr.x, az);
        float r2a, r2b;
        f2_dist2(dx, dy, dz, neg0, r2a, r2b);
        const bool ina = r2a <= CUTOFF_SQ && r2a >= MIN_R_SQ;
        const bool inb = r2b <= CUTOFF_SQ && r2b >= MIN_R_SQ;  // j + 1 = n: a pad, +inf
        if (FULL) {
            if (ina) term(j, r2a);
            if (inb) term(j + 1, r2b);
        } else {
            // both pairs' terms in packed f32x2 arithmetic; an out-of-range element is
            // computed but never added
            const ulonglong2 sq = g[2];
            const uint64_t ir = f2_pack(rsqrt_normal(r2a), rsqrt_normal(r2b));
            const uint64_t ir2 = f2_mul(ir, ir);
            const uint64_t R = f2_add(zr.y, arm);
            const uint64_t s2 = f2_mul(f2_mul(R, R), ir2);
            const uint64_t s6 = f2_mul(f2_mul(s2, s2), s2);
            const uint64_t lj = f2_mul(f2_mul(sq.x, ase), f2_mul(s6, f2_sub(s6, two)));
            const uint64_t coul = f2_mul(f2_mul(sq.y, aq), ir);
            const uint64_t hy = f2_mul(((const uint64_t*)g)[6], ahy);
            const float hya = r2a < HYDRO_CUTOFF_SQ ? f2_lo(hy) : 0.0f;
            const float hyb = r2b < HYDRO_CUTOFF_SQ ? f2_hi(hy) : 0.0f;
            const uint64_t e = f2_add(f2_add(lj, coul), f2_pack(hya, hyb));
            if (ina) part += f2_lo(e);
            if (inb) part += f2_hi(e);
            if (ABS) {
                if (ina) pabs += fabsf(f2_lo(lj)) + fabsf(f2_lo(coul)) + fabsf(hya);
                if (inb) pabs += fabsf(f2_hi(lj)) + fabsf(f2_hi(coul)) + fabsf(hyb);
            }
            if (COUNT) np += (int)ina + (int)inb;
        }
    }
    if (ABS) acc.abs_s += pabs;
    if (COUNT) acc.pairs += np;
    return part;
}

// The antigen atoms near a group: those within 10 A + group radius of its centre, among the
// blocks b0 .. b1-1 of 32 atoms each (AgView::box; a block is taken or left by its box).
struct GroupReach {
    float cx, cy, cz, reach2;  // centre, squared reach
    int b0, b1;
    __device__ __forceinline__ bool within(float ex, float ey, float ez) const {
        return __fmaf_rn(ez, ez, __fmaf_rn(ey, ey, __fmul_rn(ex, ex))) <= reach2;
    }
    __device__ __forceinline__ bool atom(const float4& a) const { return within(a.x - cx, a.y - cy, a.z - cz); }
    // false only if no atom of the block is within reach (each operation is monotonic in the
    // atom's distance along an axis, rounding included)
    __device__ __forceinline__ bool block(const AgView* __restrict__ Ap, int b) const {
        if (b >= b1) return false;
        const float4 lo = __ldg(&Ap->box[2 * b]), hi = __ldg(&Ap->box[2 * b + 1]);
        return within(fmaxf(fmaxf(lo.x - cx, cx - hi.x), 0.0f), fmaxf(fmaxf(lo.y - cy, cy - hi.y), 0.0f),
                      fmaxf(fmaxf(lo.z - cz, cz - hi.z), 0.0f));
    }
};
// Blocks from which a group looks at those of its x-slab of the grid only (two dependent
// loads that a smaller antigen's few boxes do not repay).
constexpr int SLAB_BLOCKS = 128;
// (group atoms in shared memory, all lanes call)
__device__ __forceinline__ GroupReach group_reach(const AgView* __restrict__ Ap, const GroupSmem& s, int n, int lane) {
    GroupReach c;
    float px = 0.f, py = 0.f, pz = 0.f;
    if (lane < n) {
        const float4 p = s.pos[lane];
        px = p.x; py = p.y; pz = p.z;
    }
    const float inv_n = 1.0f / (float)n;
    c.cx = warp_sum_f(px) * inv_n;
    c.cy = warp_sum_f(py) * inv_n;
    c.cz = warp_sum_f(pz) * inv_n;
    const float dgx = px - c.cx, dgy = py - c.cy, dgz = pz - c.cz;
    const float rad2 = warp_max_f(lane < n ? dgx * dgx + dgy * dgy + dgz * dgz : 0.0f);
    const float reach = 10.01f + sqrtf(rad2) * 1.0001f + 1e-3f;
    c.reach2 = reach * reach;
    c.b0 = 0;
    c.b1 = (Ap->n_atoms + 31) >> 5;
    if (c.b1 > SLAB_BLOCKS) {
        const GridView& g = Ap->grid;
        const float ux = c.cx * g.inv - (float)g.ox, rc = reach * g.inv;
        const int i0 = max(0, (int)floorf(ux - rc)), i1 = min(g.nx - 1, (int)floorf(ux + rc));
        if (i0 <= i1) {
            c.b0 = __ldg(&g.cell_start[i0 * g.ny * g.nz]) >> 5;
            c.b1 = (__ldg(&g.cell_start[(i1 + 1) * g.ny * g.nz]) + 31) >> 5;
        } else {
            c.b1 = 0;
        }
    }
    return c;
}
// FULL scoring: the group atoms' further parameters (prm visible to the warp)
__device__ __forceinline__ void group_full(const GroupSmem& s, GroupFull* gf, int n, int lane) {
    if (lane < n) {
        const int t = (int)s.prm[lane].w;
        const float4 e = c_eef1[t];
        gf->eef[lane] = e;
        gf->rl[lane] = __frcp_rn(e.z);
        gf->hb[lane] = c_hb[t];
    }
    __syncwarp();
}

// Everything one warp does for one group already in shared memory (n atoms): centre
// and radius, the antigen's blocks that come near it (32 boxes at a time), their atoms
// within reach into the queue, batched pair evaluation.  Accumulates into the lane's acc.
// The blocks are in the atoms' grid order and hold 32 atoms each, aligned: one test per
// block, where walking the grid's columns took divisions, a square root and two dependent
// loads per 32 columns and partly filled steps at their ends (one peptide of 60 atoms
// against 2500, whole call: 60 us, 52 us now; long launches change little).
template <bool KAHAN, bool FULL, bool ABS, bool COUNT>
__device__ __forceinline__ void score_group(const AgView* __restrict__ Ap, GroupSmem& s, GroupFull* gf, int n,
                                            int lane, unsigned lt, Acc& acc) {
    const float4* __restrict__ pq = Ap->pq;
    const float4* __restrict__ prm = Ap->prm;
    const int n_atoms = Ap->n_atoms;
    const GroupReach near = group_reach(Ap, s, n, lane);
    if (FULL) group_full(s, gf, n, lane);
    int qn = 0;
    for (int w0 = near.b0; w0 < near.b1; w0 += 32) {
        for (unsigned live = __ballot_sync(0xffffffffu, near.block(Ap, w0 + lane)); live; live &= live - 1) {
            const int t = (w0 + __ffs(live) - 1) * 32 + lane;
            const bool pass = t < n_atoms && near.atom(__ldg(&pq[t]));
            const unsigned m = __ballot_sync(0xffffffffu, pass);
            if (pass) s.q[qn + __popc(m & lt)] = t;
            qn += __popc(m);
            __syncwarp();
            if (qn >= 32) {
                acc_add<KAHAN>(acc, group_pairs<FULL, ABS, COUNT>(pq, prm, s, gf, n, s.q[lane], acc));
                __syncwarp();
                if (lane < qn - 32) s.q[lane] = s.q[32 + lane];
                qn -= 32;
                __syncwarp();
            }
        }
    }
    if (lane < qn) acc_add<KAHAN>(acc, group_pairs<FULL, ABS, COUNT>(pq, prm, s, gf, n, s.q[lane], acc));
    __syncwarp();
}

// The full energy of one group by a team of TEAM warps (warp `rank`; sync(): the team's
// barrier): what score_group's lanes sum, in the same order, with the work shared.  Of the
// blocks of 32 boxes that come near the group, the warps take one each in turn, place the
// atoms within reach in the team's list -- the single warp's queue -- and evaluate its
// batches of 32 in turn into the team's slots; warp 0 adds the slots to its acc, batch after
// batch, so every lane of it sums exactly the terms it would sum alone.  Result in warp 0's acc.
constexpr int TEAM_SEG = 32;
struct TeamSmem {
    float part[TEAM_SEG + 1][32];
    int list[TEAM_SEG * 32 + 32];  // queued atoms: the last segment's rest, then this one's
    int found[TEAM_SEG][32];       // passing atoms of each block
    int count[TEAM_SEG];
};
template <bool KAHAN, int TEAM, class Sync>
__device__ __forceinline__ void score_group_team(const AgView* __restrict__ Ap, GroupSmem& s, GroupFull* gf, int n,
                                                 int lane, unsigned lt, Acc& acc, int rank, TeamSmem& T, Sync sync) {
    const float4* __restrict__ pq = Ap->pq;
    const float4* __restrict__ prm = Ap->prm;
    const int n_atoms = Ap->n_atoms;
    const GroupReach near = group_reach(Ap, s, n, lane);
    group_full(s, gf, n, lane);
    int qn = 0;
#pragma unroll 1
    for (int w0 = near.b0; w0 < near.b1; w0 += 32) {
        const unsigned live = __ballot_sync(0xffffffffu, near.block(Ap, w0 + lane));
        const int chunks = __popc(live);
        int ch = 0;
        for (unsigned m = live; m; m &= m - 1, ++ch) {
            if (ch % TEAM != rank) continue;
            const int t = (w0 + __ffs(m) - 1) * 32 + lane;
            const bool pass = t < n_atoms && near.atom(__ldg(&pq[t]));
            const unsigned pm = __ballot_sync(0xffffffffu, pass);
            if (pass) T.found[ch][__popc(pm & lt)] = t;
            if (lane == 0) T.count[ch] = __popc(pm);
        }
        sync();
        int at = lane < chunks ? T.count[lane] : 0;  // inclusive prefix over the blocks
        const int own = at;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, at, d);
            if (lane >= d) at += v;
        }
        const int found = __shfl_sync(0xffffffffu, at, 31);
#pragma unroll 1
        for (int ch = rank; ch < chunks; ch += TEAM) {
            const int cnt = __shfl_sync(0xffffffffu, own, ch), to = qn + __shfl_sync(0xffffffffu, at, ch) - cnt;
            if (lane < cnt) T.list[to + lane] = T.found[ch][lane];
        }
        qn += found;
        const bool last = w0 + 32 >= near.b1;
        sync();
        const int full = qn / 32, rest = qn - full * 32, batches = full + (last && rest ? 1 : 0);
#pragma unroll 1
        for (int b = rank; b < batches; b += TEAM) {
            if (b * 32 + lane < qn)
                T.part[b][lane] = group_pairs<true, false, false>(pq, prm, s, gf, n, T.list[b * 32 + lane], acc);
        }
        sync();
        if (rank == 0) {
#pragma unroll 1
            for (int b = 0; b < batches; ++b)
                if (b * 32 + lane < qn) acc_add<KAHAN>(acc, T.part[b][lane]);
            if (lane < rest && full) T.list[lane] = T.list[full * 32 + lane];
        }
        qn = rest;
        if (!last) sync();  // the list's rest and the slots
    }
    sync();  // the next group reuses the team's memory
}

// ---- candidate sums, by one warp ------------------------------------------------------
// v[r0] + .. + v[r1 - 1] in order (without v[skip]); the loads of 32 run in parallel; on
// every lane.
__device__ __forceinline__ double warp_ordered_sum(const double* __restrict__ v, int r0, int r1, int skip = -1) {
    const int lane = threadIdx.x & 31;
    double e = 0.0;
    for (int base = r0; base < r1; base += 32) {
        const int r = base + lane;
        const double x = r < r1 && r != skip ? v[r] : 0.0;
        const int m = min(32, r1 - base);
        for (int i = 0; i < m; ++i) e += __shfl_sync(0xffffffffu, x, i);
    }
    return e;
}

// disulfide_energy (allatom.rs:155-180) of residues r0 .. r1-1, f32 in the reference's
// pair order: Gaussian well between every pair of Cys SG atoms (topology atom 5).
// Residue sub (>= 0) is taken as amino acid sub_aa with its SG at sub_sg.  The lanes find
// the Cys residues and test one Cys's partners at a time; on every lane.
static __device__ __noinline__ float warp_disulfide(const StateView& st, int r0, int r1, int sub, int sub_aa, float4 sub_sg) {
    const int lane = threadIdx.x & 31;
    float ds = 0.0f;
    for (int bi = r0; bi < r1; bi += 32) {
        const int ri = bi + lane;
        const bool ci = ri < r1 && (ri == sub ? sub_aa : (int)st.res_aa[ri]) == CYS;
        for (unsigned mi = __ballot_sync(0xffffffffu, ci); mi; mi &= mi - 1) {
            const int i = bi + __ffs(mi) - 1;
            const float4 pi = i == sub ? sub_sg : st.res_pos[(size_t)i * SLOT_STRIDE + 5];
            for (int bj = bi; bj < r1; bj += 32) {
                const int j = bj + lane;
                float t = 0.0f;
                bool in = j > i && j < r1 && (j == sub ? sub_aa : (int)st.res_aa[j]) == CYS;
                if (in) {
                    const float4 pj = j == sub ? sub_sg : st.res_pos[(size_t)j * SLOT_STRIDE + 5];
                    const float d = xsqrt(xdist2(xsub(pi.x, pj.x), xsub(pi.y, pj.y), xsub(pi.z, pj.z)));
                    in = !(d > 4.0f);
                    if (in) {
                        const float z = xdiv(xsub(d, 2.05f), 0.4f);
                        t = xmul(4.0f, mc_exp(xmul(xmul(-0.5f, z), z)));
                    }
                }
                for (unsigned m = __ballot_sync(0xffffffffu, in); m; m &= m - 1)
                    ds = xsub(ds, __shfl_sync(0xffffffffu, t, __ffs(m) - 1));
            }
        }
    }
    return ds;
}

// the candidate's energy from its residues' (full: with its disulfide term)
__device__ __forceinline__ double warp_candidate_sum(const StateView& st, int c, const double* __restrict__ res_e,
                                                     int full) {
    const int r0 = st.cand_res_off[c], r1 = st.cand_res_off[c + 1];
    double e = warp_ordered_sum(res_e, r0, r1);
    if (full) e += (double)warp_disulfide(st, r0, r1, -1, 0, make_float4(0.f, 0.f, 0.f, 0.f));
    return e;
}

}  // namespace binder
