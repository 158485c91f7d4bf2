// k_score.cu — all-atom AMBER LJ + Coulomb + hydrophobic pair energy (and force)
// of candidates against a resident antigen, on the FP32 pipes with rsqrt.
//
// Replaces GpuContext::score_batch (gpu.rs:166-267) and its shader
// (energy.wgsl:47-118), whose pair math is the LJ/Coulomb/hydrophobic part of
// interaction_energy_atoms_breakdown (energy.rs:261-314).  The shader is brute
// force over every antigen atom.  Here the energy kernels take groups of nearby
// candidate atoms (a residue, or consecutive atoms of a flat candidate) against the
// blocks of 32 antigen atoms whose boxes come near the group (score.cuh); the force
// kernel takes one candidate atom at a time against the grid columns in reach.  The
// pair set is exactly the reference's (0.25 <= r^2 <= 100 with the reference's f32
// rounding of r^2) at a fraction of the pair tests.
//
// Precision: f32 pair terms, per-lane compensated (Kahan) sums, FP64 warp-shuffle and
// fixed-order FP64 sums above them (deterministic).
#include <algorithm>

#include "kernels.h"
#include "score.cuh"
#include "topk.cuh"

namespace binder {

cudaError_t score_init_tables() { return score_tables_init(); }

struct SrcStateG {
    StateView st;
    // residue r: its atoms into the group (the loads of its amino acid and positions are issued
    // together: the slots beyond its atoms are read and dropped)
    __device__ int load(int r, int lane, GroupSmem& s, bool& bad) const {
        const int aa = st.res_aa[r];
        const float4 p = lane < SLOTS ? st.res_pos[(size_t)r * SLOT_STRIDE + lane] : make_float4(0.f, 0.f, 0.f, 0.f);
        const int n = c_topo_n[aa];
        float4 m = make_float4(0.f, 0.f, 0.f, 0.f);
        if (lane < n) {
            m = g_slot_prm[aa][lane];
            bad = !finite3(p.x, p.y, p.z);
            s.pos[lane] = make_float4(p.x, p.y, p.z, m.x);
            s.prm[lane] = make_float4(m.y, m.z, m.w, (float)g_slot_type[aa][lane]);
        }
        group_xyz(s, lane, n, p.x, p.y, p.z);
        group_prm(s, lane, n, m.x, m.y, m.z, m.w);
        return n;
    }
};

// Resident state: persistent teams of TEAM warps take residues from a work queue (an
// atomic counter) and write one FP64 energy per residue; k_sum_residues adds a candidate's
// residues in index order.  No CTA barrier: teams never wait for each other.  The residues
// come in Calpha-cell order, so that neighbouring warps share antigen atoms in L1, or by the
// gradient steps' work bands, heaviest first, or in index order while those bands are not
// filled -- cell order or not as the autotuner timed it.  A warp evaluates only four or five
// residues of about 11 us each (20480 residues, 4736 warps), so the launch's end is decided by
// what comes last: heaviest first 61 -> 57 us, and claiming a residue ahead (to hide the
// counter's latency) cost more than it hid (60 us).
template <int NW, bool KAHAN, bool FULL, bool ABS, bool COUNT, int TEAM>
__global__ void __launch_bounds__(NW * 32) k_score_residues(StateView st, const AgView* __restrict__ ags,
                                                             const int* __restrict__ order, const int* __restrict__ bal,
                                                             int* __restrict__ queue,
                                                             double* __restrict__ res_e, double* __restrict__ res_abs,
                                                             long long* __restrict__ pair_count,
                                                             uint32_t* __restrict__ err) {
    static_assert(NW % TEAM == 0 && NW / TEAM < 16 + (TEAM == 1), "one named barrier per team");
    __shared__ GroupSmem gs[NW];
    __shared__ GroupFull gfs[FULL ? NW : 1];
    extern __shared__ __align__(16) unsigned char team_raw[];  // TEAM > 1: a TeamSmem per team
    TeamSmem* teams = reinterpret_cast<TeamSmem*>(team_raw);
    __shared__ int s_task[TEAM > 1 ? NW / TEAM : 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int team = warp / TEAM, rank = warp % TEAM;
    const unsigned lt = (1u << lane) - 1u;
    GroupSmem& s = gs[warp];
    SrcStateG src{st};
    auto sync = [team] { asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "n"(TEAM * 32) : "memory"); };
    int my_pairs = 0;
    // lane b: residues in the work bands 0 .. b; the buckets are taken when they hold every residue
    int band_end = 0, parity = 0;
    if (bal) {
        parity = __ldg(&bal[0]) & 1;
        band_end = lane < CG_BAL_BINS ? __ldg(&bal[2 + CG_BAL_BINS * parity + lane]) : 0;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, band_end, d);
            if (lane >= d) band_end += v;
        }
        if (__shfl_sync(0xffffffffu, band_end, 31) != st.total_res) bal = nullptr;
    }
    for (;;) {
        int gi = 0;
        if (lane == 0 && rank == 0) gi = atomicAdd(queue, 1);
        if (TEAM > 1) {
            if (lane == 0 && rank == 0) s_task[team] = gi;
            sync();
            gi = s_task[team];
            sync();
        } else {
            gi = __shfl_sync(0xffffffffu, gi, 0);
        }
        if (gi >= st.total_res) break;
        int r = gi;
        if (order) {
            r = order[gi];
        } else if (bal) {
            const int b = __popc(__ballot_sync(0xffffffffu, lane < CG_BAL_BINS && band_end <= gi));
            const int below = __shfl_sync(0xffffffffu, band_end, max(b - 1, 0));
            r = __ldg(bal + CG_BAL_HEADER + (size_t)(parity * CG_BAL_BINS + b) * st.total_res + gi - (b ? below : 0));
        }
        const AgView* Ap = &ags[st.cand_ag[st.res_cand[r]]];
        bool bad = false;
        const int n = src.load(r, lane, s, bad);
        Acc acc = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0};
        if (__any_sync(0xffffffffu, bad)) {
            if (lane == 0) atomicOr(err, ERRF_NAN);
        } else if (n > 0) {
            __syncwarp();
            if constexpr (TEAM > 1)
                score_group_team<KAHAN, TEAM>(Ap, s, &gfs[warp], n, lane, lt, acc, rank, teams[team], sync);
            else
                score_group<KAHAN, FULL, ABS, COUNT>(Ap, s, FULL ? &gfs[warp] : nullptr, n, lane, lt, acc);
        }
        __syncwarp();
        if (rank == 0) {
            const double e = warp_sum_d(KAHAN ? ((double)acc.s - (double)acc.c) : (double)acc.s);
            const double ea = ABS ? warp_sum_d((double)acc.abs_s) : 0.0;
            if (lane == 0) {
                if (res_e) res_e[r] = e;
                if (ABS) res_abs[r] = ea;
            }
        }
        if (COUNT) my_pairs += acc.pairs;
    }
    if (COUNT) {
        int p = my_pairs;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) p += __shfl_xor_sync(0xffffffffu, p, o);
        if (lane == 0 && p) atomicAdd((unsigned long long*)pair_count, (unsigned long long)p);
    }
    queue_retire(queue);
}

// ---- flat GpuAtom candidates (binder_gpu_atom = 2 x float4) -------------------------
// atoms of candidate c: off[c] .. off[c+1], or n_ab each (off null)
struct FlatAtoms {
    const float4* atoms;
    const long long* off;
    long long n_ab;
    __device__ long long begin(int c) const { return off ? off[c] : c * n_ab; }
};

// One CTA per candidate at a time, which it cuts into groups of up to FLAT_GROUP nearby
// consecutive atoms: a group ends where the next atom lies further than FLAT_GAP from the
// last one (the next residue of a population whose residues are placed apart, a side
// chain's tip to the next backbone), so that its sphere, and with it the antigen atoms it
// queues, stays small -- groups of eight consecutive atoms straddled residues tens of
// Angstroms apart and queued most of the antigen (1024 candidates x 170 atoms against
// 2500: 337 us, 67 us now).  Two more rules, whole calls of 1024 candidates x 160 atoms:
//  * A group with an atom further than FLAT_LONG from its first, longer than any residue
//    (Calphas in a row have no gap), is cut in two: against 6700 atoms 495 us whole, 271 in
//    two (291 in eights), 210 in fours, which short chains and small antigens pay for
//    (random walks of Calphas 308 in fours, 302 in two; against 130 atoms 171 and 160).
//  * Where gaps leave fewer than four atoms a group on average (atoms in no spatial order)
//    and the antigen is small, gaps end no group: the whole antigen is in every group's
//    reach anyway (against 130 atoms 234 us with gaps, 173 without, in eights 181; 590
//    atoms 270 and 247; 1000 atoms 283 and 270, but 295 and 356 when spread over a shell).
// Warps take groups as they come free; each group's FP64 energy has its own slot and the
// slots are added in order, so sums do not depend on the order the groups were taken in.
constexpr int FLAT_GROUP = 14;       // atoms of the largest residue
constexpr int FLAT_PART = 7;         // atoms of a long group's parts
constexpr float FLAT_GAP = 4.5f;     // A between consecutive atoms of a group
constexpr float FLAT_LONG = 12.0f;   // A from a group's first atom
constexpr int FLAT_SMALL = 640;      // antigen atoms
constexpr int FLAT_CHUNK = 256;      // atoms cut into groups at once
template <int NW, bool KAHAN, bool ABS, bool COUNT>
__global__ void __launch_bounds__(NW * 32) k_score_grouped(FlatAtoms src, int n_cand, const AgView* __restrict__ ags,
                                                            const int* __restrict__ cand_ag,
                                                            double* __restrict__ out, double* __restrict__ out_abs,
                                                            long long* __restrict__ pair_count,
                                                            uint32_t* __restrict__ err) {
    static_assert(NW * 32 >= FLAT_CHUNK, "one thread per atom of a chunk");
    __shared__ GroupSmem gs[NW];
    __shared__ double s_e[FLAT_CHUNK], s_a[ABS ? FLAT_CHUNK : 1];
    __shared__ short s_start[FLAT_CHUNK + 1];
    __shared__ bool s_long[FLAT_CHUNK];
    __shared__ int s_warp[NW], s_groups, s_next;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned lt = (1u << lane) - 1u;
    GroupSmem& s = gs[warp];
    int my_pairs = 0;
    for (int c = blockIdx.x; c < n_cand; c += gridDim.x) {
        const AgView* Ap = &ags[cand_ag ? cand_ag[c] : 0];
        const long long a0 = src.begin(c), a1 = src.begin(c + 1);
        double e = 0.0, ea = 0.0;  // thread 0
        for (long long base = a0; base < a1; base += FLAT_CHUNK) {
            const int m = (int)min((long long)FLAT_CHUNK, a1 - base);
            // group starts: atoms far from their predecessor, every FLAT_GROUP-th after one,
            // and the middles of long groups
            bool brk = false;
            float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
            auto apart = [&](int i, float d) {  // atom i of the chunk further than d from this one
                const float4 q = __ldg(&src.atoms[2 * (base + i)]);
                const float dx = p.x - q.x, dy = p.y - q.y, dz = p.z - q.z;
                return !(dx * dx + dy * dy + dz * dz <= d * d);
            };
            if (tid < m) {
                p = __ldg(&src.atoms[2 * (base + tid)]);
                brk = tid == 0 || apart(tid - 1, FLAT_GAP);
            }
            const unsigned mb = __ballot_sync(0xffffffffu, brk);
            if (lane == 0) s_warp[warp] = mb ? warp * 32 + 31 - __clz(mb) : -1;  // the warp's last break
            if (tid < FLAT_CHUNK) s_long[tid] = false;
            if (tid == 0) s_next = 0;
            const bool scattered = __syncthreads_count(brk) * 4 > m && Ap->n_atoms <= FLAT_SMALL;
            const unsigned below = mb & (lt | 1u << lane);
            int run = below ? warp * 32 + 31 - __clz(below) : -1;
            for (int w = warp - 1; run < 0 && w >= 0; --w) run = s_warp[w];
            if (scattered) run = 0;
            const int k = (tid - run) % FLAT_GROUP;
            if (tid < m && k >= FLAT_PART && !scattered && apart(tid - k, FLAT_LONG)) s_long[tid - k] = true;
            __syncthreads();
            const bool start = tid < m && (k == 0 || (k == FLAT_PART && s_long[tid - k]));
            const unsigned ms = __ballot_sync(0xffffffffu, start);
            if (lane == 0) s_warp[warp] = __popc(ms);
            __syncthreads();
            int at = __popc(ms & lt);
            for (int w = 0; w < warp; ++w) at += s_warp[w];
            if (start) s_start[at] = (short)tid;
            if (tid == m - 1) {  // the last atom: groups up to and including its own
                s_groups = at + (start ? 1 : 0);
                s_start[s_groups] = (short)m;
            }
            __syncthreads();
            const int groups = s_groups;
            for (;;) {
                int g = 0;
                if (lane == 0) g = atomicAdd(&s_next, 1);
                g = __shfl_sync(0xffffffffu, g, 0);
                if (g >= groups) break;
                const long long j0 = base + s_start[g];
                const int n = s_start[g + 1] - s_start[g];
                bool bad = false;
                if (lane < n) {
                    const float4 p0 = __ldg(&src.atoms[2 * (j0 + lane)]);
                    const float4 p1 = __ldg(&src.atoms[2 * (j0 + lane) + 1]);
                    bad = !finite3(p0.x, p0.y, p0.z);
                    s.pos[lane] = make_float4(p0.x, p0.y, p0.z, p0.w * SQRT_COULOMB_K);
                    s.prm[lane] = make_float4(p1.x, sqrtf(p1.y), p1.z > 0.5f ? 1.0f : 0.0f, 0.0f);
                    group_xyz(s, lane, n, p0.x, p0.y, p0.z);
                    group_prm(s, lane, n, s.pos[lane].w, s.prm[lane].x, s.prm[lane].y, s.prm[lane].z);
                } else {
                    group_xyz(s, lane, n, 0.f, 0.f, 0.f);
                    group_prm(s, lane, n, 0.f, 0.f, 0.f, 0.f);
                }
                Acc acc = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0};
                if (__any_sync(0xffffffffu, bad)) {
                    if (lane == 0) atomicOr(err, ERRF_NAN);
                } else {
                    __syncwarp();
                    score_group<KAHAN, false, ABS, COUNT>(Ap, s, nullptr, n, lane, lt, acc);
                }
                __syncwarp();
                const double ge = warp_sum_d(KAHAN ? ((double)acc.s - (double)acc.c) : (double)acc.s);
                const double ga = ABS ? warp_sum_d((double)acc.abs_s) : 0.0;
                if (lane == 0) {
                    s_e[g] = ge;
                    if (ABS) s_a[g] = ga;
                }
                if (COUNT) my_pairs += acc.pairs;
            }
            __syncthreads();
            if (warp == 0) {  // the groups' energies in order
                e += warp_ordered_sum(s_e, 0, groups);
                if (ABS) ea += warp_ordered_sum(s_a, 0, groups);
            }
            __syncthreads();
        }
        if (tid == 0) {
            if (out) out[c] = e;
            if (ABS) out_abs[c] = ea;
        }
    }
    if (COUNT) {
        int p = my_pairs;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) p += __shfl_xor_sync(0xffffffffu, p, o);
        if (lane == 0 && p) atomicAdd((unsigned long long*)pair_count, (unsigned long long)p);
    }
}

// All-atom force and energy: one warp per candidate atom, its 32 lanes stride over the
// antigen atoms of each culled column (the antigen is sorted by cell, so a column's z-run
// of cells is one range).  The lanes find 32 columns' ranges at once; each lane queues its
// in-cutoff atoms (FORCE_Q of its own, in order) and evaluates them when a lane's queue is
// full and at the end, so the pair terms run a few times per candidate atom instead of in
// every step that holds one in-cutoff pair: 1024 candidates x 170 atoms 249 us,
// 216 us now, the same sums per lane (the deepest lane's 4-5 pairs per atom are most of it).
constexpr int FORCE_Q = 6;
template <int NW, bool KAHAN>
__global__ void __launch_bounds__(NW * 32) k_force_flat(FlatAtoms src, int n_cand, const AgView* __restrict__ ags,
                                                         const int* __restrict__ cand_ag, double* __restrict__ out,
                                                         float* __restrict__ force, uint32_t* __restrict__ err) {
    __shared__ double sm[NW];
    __shared__ float2 s_q[NW][FORCE_Q][32];  // r^2, antigen atom
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float2(*q)[32] = s_q[warp];
    for (int c = blockIdx.x; c < n_cand; c += gridDim.x) {
        const AgView* __restrict__ Ap = &ags[cand_ag ? cand_ag[c] : 0];
        const float4* __restrict__ pq = Ap->pq;
        const float4* __restrict__ prm = Ap->prm;
        const int* __restrict__ cell_start = Ap->grid.cell_start;
        const float inv = Ap->grid.inv;
        const int gnx = Ap->grid.nx, gny = Ap->grid.ny, gnz = Ap->grid.nz;
        const float ox = (float)Ap->grid.ox, oy = (float)Ap->grid.oy, oz = (float)Ap->grid.oz;
        const long long a_begin = src.begin(c), a_end = src.begin(c + 1);
        Acc acc = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0};
        for (long long j = a_begin + warp; j < a_end; j += NW) {
            const float4 p0 = __ldg(&src.atoms[2 * j]);
            const float4 p1 = __ldg(&src.atoms[2 * j + 1]);
            if (!finite3(p0.x, p0.y, p0.z)) {
                if (lane == 0) atomicOr(err, ERRF_NAN);
                continue;
            }
            AtomIn b;
            b.x = p0.x; b.y = p0.y; b.z = p0.z;
            b.qs = p0.w * SQRT_COULOMB_K;
            b.rmh = p1.x;
            b.se = sqrtf(p1.y);
            b.h = p1.z > 0.5f ? 1.0f : 0.0f;
            acc.fx = acc.fy = acc.fz = 0.f;
            int cnt = 0;
            auto flush = [&] {
                const int k_max = __reduce_max_sync(0xffffffffu, cnt);
#pragma unroll 1
                for (int k = 0; k < k_max; ++k) {
                    if (k >= cnt) continue;
                    const float2 h = q[k][lane];
                    const int t = __float_as_int(h.y);
                    const float r2 = h.x;
                    const float4 apq = __ldg(&pq[t]);
                    const float4 aprm = __ldg(&prm[t]);
                    const float dx = b.x - apq.x, dy = b.y - apq.y, dz = b.z - apq.z;
                    const float ir = rsqrt_normal(r2);
                    const float ir2 = ir * ir;
                    const float R = b.rmh + aprm.x;
                    const float s2 = R * R * ir2;
                    const float s6 = s2 * s2 * s2;
                    const float eps = b.se * aprm.y;
                    const float lj = eps * (s6 * (s6 - 2.0f));
                    const float qq = b.qs * apq.w;
                    const float coul = qq * ir;
                    float e = lj + coul;
                    const float hyd = (r2 < HYDRO_CUTOFF_SQ) ? HYDRO_BONUS * (b.h * aprm.z) : 0.0f;
                    e += hyd;
                    acc_add<KAHAN>(acc, e);
                    // -dE/dr * r_hat / r : 12 eps (s12 - s6)/r^2 + qq/r^3
                    const float sc = 12.0f * eps * (s6 * (s6 - 1.0f)) * ir2 + coul * ir2;
                    acc.fx += sc * dx;
                    acc.fy += sc * dy;
                    acc.fz += sc * dz;
                }
                cnt = 0;
            };
            // the columns (i, j) in x-major order within the cutoff + margin, in cell units
            const float ux = b.x * inv - ox, uy = b.y * inv - oy, uz = b.z * inv - oz;
            const float reach = 10.01f * inv, reach2 = reach * reach;
            const int i0 = max(0, (int)floorf(ux - reach)), i1 = min(gnx - 1, (int)floorf(ux + reach));
            const int j0 = max(0, (int)floorf(uy - reach)), j1 = min(gny - 1, (int)floorf(uy + reach));
            const int nj = j1 - j0 + 1, ncol = (i1 >= i0 && j1 >= j0) ? (i1 - i0 + 1) * nj : 0;
            for (int c0 = 0; c0 < ncol; c0 += 32) {
                int ra0 = 0, ra1 = 0;
                if (c0 + lane < ncol) {
                    const int i = i0 + (c0 + lane) / nj, jj = j0 + (c0 + lane) % nj;
                    const float ddx = fmaxf(fmaxf((float)i - ux, ux - (float)(i + 1)), 0.0f);
                    const float ddy = fmaxf(fmaxf((float)jj - uy, uy - (float)(jj + 1)), 0.0f);
                    const float rem2 = reach2 - ddx * ddx - ddy * ddy;
                    if (rem2 >= 0.0f) {
                        const float rem = sqrtf(rem2);
                        const int k0 = max(0, (int)floorf(uz - rem)), k1 = min(gnz - 1, (int)floorf(uz + rem));
                        if (k0 <= k1) {
                            const int base = (i * gny + jj) * gnz;
                            ra0 = __ldg(&cell_start[base + k0]);
                            ra1 = __ldg(&cell_start[base + k1 + 1]);
                        }
                    }
                }
                for (unsigned live = __ballot_sync(0xffffffffu, ra1 > ra0); live; live &= live - 1) {
                    const int from = __ffs(live) - 1;
                    const int a0 = __shfl_sync(0xffffffffu, ra0, from), a1 = __shfl_sync(0xffffffffu, ra1, from);
                    for (int t0 = a0; t0 < a1; t0 += 32) {
                        const int t = t0 + lane;
                        if (t < a1) {
                            const float4 apq = __ldg(&pq[t]);
                            // reference rounding of r^2: the reference's pair set
                            const float r2 = xdist2(b.x - apq.x, b.y - apq.y, b.z - apq.z);
                            if (r2 <= CUTOFF_SQ && r2 >= MIN_R_SQ) q[cnt++][lane] = make_float2(r2, __int_as_float(t));
                        }
                        if (__any_sync(0xffffffffu, cnt == FORCE_Q)) flush();
                    }
                }
            }
            flush();
            const float fx = warp_sum_f(acc.fx), fy = warp_sum_f(acc.fy), fz = warp_sum_f(acc.fz);
            if (lane < 3) force[3 * j + lane] = lane == 0 ? fx : lane == 1 ? fy : fz;
        }
        const double e = cta_sum<NW>(KAHAN ? ((double)acc.s - (double)acc.c) : (double)acc.s, sm, lane, warp);
        if (threadIdx.x == 0 && out) out[c] = e;
    }
}

// ---- launchers ----------------------------------------------------------------------
constexpr int NW_SCORE = 8;

int launch_score_flat(cudaStream_t s, const float* atoms, const long long* offsets, long long n_ab, int n_cand,
                      const AgView* ags, const int* cand_ag, int accumulate, const ScoreOut& o, int grid_ctas) {
    if (n_cand <= 0) return 0;
    const FlatAtoms src{reinterpret_cast<const float4*>(atoms), offsets, n_ab};
    const int g = grid_ctas > 0 ? min(grid_ctas, n_cand) : n_cand;
    const bool kahan = accumulate == 0;
    if (o.force) {  // each warp owns one candidate atom's force
        if (kahan) k_force_flat<NW_SCORE, true><<<g, NW_SCORE * 32, 0, s>>>(src, n_cand, ags, cand_ag, o.energy, o.force, o.err);
        else k_force_flat<NW_SCORE, false><<<g, NW_SCORE * 32, 0, s>>>(src, n_cand, ags, cand_ag, o.energy, o.force, o.err);
        return 1;
    }
#define BINDER_G(K, A, C)                                                                                       \
    k_score_grouped<NW_SCORE, K, A, C><<<g, NW_SCORE * 32, 0, s>>>(src, n_cand, ags, cand_ag, o.energy, o.abs_sum, \
                                                                   o.pairs, o.err)
    if (o.pairs) BINDER_G(true, false, true);
    else if (o.abs_sum) { if (kahan) BINDER_G(true, true, false); else BINDER_G(false, true, false); }
    else { if (kahan) BINDER_G(true, false, false); else BINDER_G(false, false, false); }
#undef BINDER_G
    return 1;
}

// Candidate energy = its residues' energies added in index order (+ disulfide when full),
// one warp per candidate: the loads of 32 residues at a time run in parallel, the
// additions keep their order.  One thread per candidate had waited for every load and
// scanned all residues for every Cys: 64 x 20 residues 29 us, 6 us now; 64 chains of about
// 115 residues 129 us, 13 us now.
constexpr int SUM_WARPS = 4;
__global__ void __launch_bounds__(SUM_WARPS * 32) k_sum_residues(StateView st, const double* __restrict__ res_e,
                                                                 const double* __restrict__ res_abs, int full,
                                                                 double* __restrict__ out,
                                                                 double* __restrict__ out_abs) {
    const int c = blockIdx.x * SUM_WARPS + (threadIdx.x >> 5);
    if (c >= st.n_cand) return;
    double ea = 0.0;
    const double e = warp_candidate_sum(st, c, res_e, full);
    if (res_abs) ea = warp_ordered_sum(res_abs, st.cand_res_off[c], st.cand_res_off[c + 1]);
    if ((threadIdx.x & 31) == 0) {
        out[c] = e;
        if (out_abs) out_abs[c] = ea;
    }
}

// Candidate sums and survivor selection in one launch (k <= 64, segments of at most
// SS_MAX candidates): one CTA per segment.  Thread t adds the residue energies of the
// segment's entries t, t + 1024, ... in residue order (the k_sum_residues sums, loads
// issued ahead of the additions) and keeps their order-preserving keys.  A radix select, 8 bits
// of the 64-bit key per pass from the top, finds the bucket that holds the k-th
// smallest key: every key below it is a survivor, and of the keys in it (all equal
// after the last pass) the ones earliest in the segment, which is candidate-index
// order.  One warp sorts the k survivors by (key, index): the stable top-k of the
// segment, as k_topk64 computes it.  A pass costs three barriers; it ends early
// once the bucket holds exactly the survivors still missing (typically after the
// third pass, when the bucket holds a single key).
constexpr int SS_THREADS = 1024;
constexpr int SS_PER = 4;
constexpr int SS_MAX = SS_THREADS * SS_PER;

__global__ void __launch_bounds__(SS_THREADS) k_sum_select(StateView st, const double* __restrict__ res_e,
                                                           double* __restrict__ out, const int* __restrict__ idx_list,
                                                           const long long* __restrict__ seg_off, int k,
                                                           int* __restrict__ out_idx) {
    __shared__ int s_hist[256];
    __shared__ unsigned long long s_sel_k[64];
    __shared__ int s_sel_i[64];
    __shared__ unsigned long long s_prefix;
    __shared__ int s_need, s_cnt, s_nsel;
    __shared__ unsigned long long s_prefix_tot;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int seg = blockIdx.x;
    const long long b0 = seg_off[seg];
    const int n = (int)(seg_off[seg + 1] - b0);
    const int kk = min(k, n);
    // this thread's candidates: segment entries t + SS_THREADS * q
    unsigned long long key[SS_PER];
    int cid[SS_PER];
#pragma unroll
    for (int q = 0; q < SS_PER; ++q) {
        const int j = (int)threadIdx.x + SS_THREADS * q;
        key[q] = 0xFFFFFFFFFFFFFFFFull;
        cid[q] = -1;
        if (j < n) {
            const int c = idx_list ? idx_list[b0 + j] : (int)(b0 + j);
            const int r0 = st.cand_res_off[c], r1 = st.cand_res_off[c + 1];
            double e = 0.0;
            int r = r0;
            for (; r + 4 <= r1; r += 4) {
                const double v0 = res_e[r], v1 = res_e[r + 1], v2 = res_e[r + 2], v3 = res_e[r + 3];
                e += v0;
                e += v1;
                e += v2;
                e += v3;
            }
            for (; r < r1; ++r) e += res_e[r];
            out[c] = e;
            key[q] = order_key(e);
            cid[q] = c;
        }
    }
    if (threadIdx.x == 0) {
        s_prefix = 0ull;
        s_need = kk;
        s_cnt = 0;
        s_nsel = 0;
    }
    // ---- radix select of the kk-th smallest key ----
    unsigned long long mask = 0ull;
    bool all_in = false;  // the final bucket holds exactly the survivors still missing
    for (int shift = 56; shift >= 0 && kk > 0; shift -= 8) {
        for (int t = threadIdx.x; t < 256; t += SS_THREADS) s_hist[t] = 0;
        __syncthreads();
        const unsigned long long prefix = s_prefix;
#pragma unroll
        for (int q = 0; q < SS_PER; ++q) {
            if (q * SS_THREADS >= n) break;  // no thread holds entry q
            // one shared atomic per distinct digit of the warp: the lowest lane still
            // pending takes every lane with its digit
            const bool in = cid[q] >= 0 && (key[q] & mask) == prefix;
            const int dg = in ? (int)((key[q] >> shift) & 255ull) : -1;
            unsigned pend = __ballot_sync(0xffffffffu, in);
            while (pend) {
                const int leader = __ffs(pend) - 1;
                const int d = __shfl_sync(0xffffffffu, dg, leader);
                const unsigned same = __ballot_sync(0xffffffffu, in && dg == d);
                if (lane == leader) atomicAdd(&s_hist[d], __popc(same));
                pend &= ~same;
            }
        }
        __syncthreads();
        if (warp == 0) {  // the digit whose bucket holds the s_need-th key
            const int need = s_need;
            int h[8], loc = 0;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                h[i] = s_hist[lane * 8 + i];
                loc += h[i];
            }
            int inc = loc;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += v;
            }
            const int exc = inc - loc;
            if (exc < need && need <= inc) {
                int cum = exc;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    if (cum + h[i] >= need) {
                        s_prefix = prefix | ((unsigned long long)(lane * 8 + i) << shift);
                        s_need = need - cum;
                        s_cnt = h[i];
                        break;
                    }
                    cum += h[i];
                }
            }
        }
        __syncthreads();
        mask |= 0xFFull << shift;
        if (s_cnt == s_need) {
            all_in = true;
            break;
        }
    }
    __syncthreads();
    // ---- the survivors: keys below the bucket, and the bucket's first s_need ----
    const unsigned long long prefix = s_prefix;
    const int need = s_need;
    // rank of each bucket member in segment order (entry t + 1024 q: q major), from a
    // block scan of the per-q membership flags packed 16 bits per q (only needed when
    // the bucket holds more keys than survivors missing)
    int rank[SS_PER] = {0, 0, 0, 0};
    if (!all_in && kk > 0) {
        unsigned long long mine = 0ull;
#pragma unroll
        for (int q = 0; q < SS_PER; ++q)
            if (cid[q] >= 0 && (key[q] & mask) == prefix) mine |= 1ull << (16 * q);
        unsigned long long inc = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long v = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += v;
        }
        __shared__ unsigned long long s_wsum[32];
        if (lane == 31) s_wsum[warp] = inc;
        __syncthreads();
        if (warp == 0) {
            const unsigned long long w = s_wsum[lane];
            unsigned long long wi = w;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned long long v = __shfl_up_sync(0xffffffffu, wi, o);
                if (lane >= o) wi += v;
            }
            s_wsum[lane] = wi - w;
            if (lane == 31) s_prefix_tot = wi;  // per-q totals of the bucket
        }
        __syncthreads();
        const unsigned long long before = s_wsum[warp] + inc - mine;  // earlier threads, per q
        const unsigned long long tot = s_prefix_tot;
        int base = 0;
#pragma unroll
        for (int q = 0; q < SS_PER; ++q) {
            rank[q] = base + (int)((before >> (16 * q)) & 0xFFFFull);
            base += (int)((tot >> (16 * q)) & 0xFFFFull);
        }
    }
#pragma unroll
    for (int q = 0; q < SS_PER; ++q) {
        if (cid[q] < 0 || kk == 0) continue;
        const bool below = key[q] < prefix;  // prefix has zeros under the mask
        bool take = below;
        if (!below && (key[q] & mask) == prefix) take = all_in || rank[q] < need;
        if (take) {
            const int p = atomicAdd(&s_nsel, 1);
            if (p < 64) {
                s_sel_k[p] = key[q];
                s_sel_i[p] = cid[q];
            }
        }
    }
    __syncthreads();
    if (warp == 0) {  // sort the kk survivors by (key, index)
        const KI inf = {0xFFFFFFFFFFFFFFFFull, INT32_MAX};
        KI a = lane < kk ? KI{s_sel_k[lane], s_sel_i[lane]} : inf;
        KI b = lane + 32 < kk ? KI{s_sel_k[lane + 32], s_sel_i[lane + 32]} : inf;
        a = warp_sort32(a, lane);
        b = warp_sort32(b, lane);
        KI hi = inf;
        warp_merge64(a, hi, b, inf, lane);
        int* oi = out_idx + (long long)seg * k;
        if (lane < k) oi[lane] = a.i != INT32_MAX ? a.i : -1;
        if (lane + 32 < k) oi[lane + 32] = hi.i != INT32_MAX ? hi.i : -1;
    }
}

bool sum_topk_fits(int k, long long max_segment) { return k > 0 && k <= 64 && max_segment <= SS_MAX; }

void launch_sum_select(cudaStream_t s, const StateView& st, const double* res_e, double* energy, const SumTopk& tk) {
    if (st.n_cand <= 0 || tk.n_seg <= 0) return;
    k_sum_select<<<tk.n_seg, SS_THREADS, 0, s>>>(st, res_e, energy, tk.idx_list, tk.seg_off, tk.k, tk.out_idx);
}

// Four warps share a residue of the full energy while the grid's warps outnumber the
// residues twice: a warp evaluates a residue's batches one after another, and the residues
// deep in contact set the launch's length (1280 residues: 63 us with one warp each and
// per-pair table lookups, 28 us now).
static bool full_team(const StateView& st, int g, int warps) { return st.total_res * 2ll <= (long long)g * warps; }

template <int NW>
static void score_residues_nw(cudaStream_t s, int g, const StateView& st, const AgView* ags, bool kahan, bool full,
                              bool abs_, bool count, const ScoreOut& o, const StateScoreScratch& scr) {
    constexpr size_t team_bytes = NW / 4 * sizeof(TeamSmem);
#define BINDER_R(K, FU, A, C, T)                                                                                 \
    k_score_residues<NW, K, FU, A, C, T><<<g, NW * 32, T > 1 ? team_bytes : 0, s>>>(                            \
        st, ags, scr.order, scr.bal, scr.queue, count ? nullptr : scr.res_e, scr.res_abs, o.pairs, o.err)
    if (count) BINDER_R(true, false, false, true, 1);
    else if (full) {
        if constexpr (NW == NW_SCORE) {
            if (full_team(st, g, NW)) BINDER_R(true, true, false, false, 4);
            else BINDER_R(true, true, false, false, 1);
        }
    }
    else if (abs_) { if (kahan) BINDER_R(true, false, true, false, 1); else BINDER_R(false, false, true, false, 1); }
    else { if (kahan) BINDER_R(true, false, false, false, 1); else BINDER_R(false, false, false, false, 1); }
#undef BINDER_R
}

static void score_residues(cudaStream_t s, const StateView& st, const AgView* ags, bool kahan, bool full, bool abs_,
                           bool count, const ScoreOut& o, const StateScoreScratch& scr, int g, int warps) {
    switch (warps) {
        case 4: score_residues_nw<4>(s, g, st, ags, kahan, full, abs_, count, o, scr); break;
        case 16: score_residues_nw<16>(s, g, st, ags, kahan, full, abs_, count, o, scr); break;
        default: score_residues_nw<8>(s, g, st, ags, kahan, full, abs_, count, o, scr); break;
    }
}

// The full energy takes CTAs of 8 warps whatever the plain score's shape (its 79 registers
// a thread leave room for 24 warps per SM that way, for 16 in CTAs of 16).
void launch_score_full_residues(cudaStream_t s, const StateView& st, const AgView* ags, int accumulate, uint32_t* err,
                                const StateScoreScratch& scr, int grid_ctas, int warps_per_cta) {
    const ScoreOut o{nullptr, nullptr, nullptr, nullptr, err};
    score_residues_nw<NW_SCORE>(s, std::max(1, grid_ctas * warps_per_cta / NW_SCORE), st, ags, accumulate == 0, true,
                                false, false, o, scr);
}

int launch_score_state(cudaStream_t s, const StateView& st, const AgView* ags, int accumulate, int full,
                       const ScoreOut& o, const StateScoreScratch& scr, int grid_ctas, int warps_per_cta,
                       const SumTopk* tk) {
    if (st.n_cand <= 0) return 0;
    const bool kahan = accumulate == 0, abs_ = o.abs_sum != nullptr, count = o.pairs != nullptr;
    const int g = grid_ctas > 0 ? grid_ctas : 148 * 4;
    if (full && !count) launch_score_full_residues(s, st, ags, accumulate, o.err, scr, g, warps_per_cta);
    else score_residues(s, st, ags, kahan, false, abs_, count, o, scr, g, warps_per_cta);
    if (!count && tk && !abs_) {
        if (tk->defer) return 1;  // the sums and the selection come later (launch_sum_select)
        if (tk->mid) cudaEventRecord(tk->mid, s);
        launch_sum_select(s, st, scr.res_e, o.energy, *tk);
    } else if (!count) {
        k_sum_residues<<<(st.n_cand + SUM_WARPS - 1) / SUM_WARPS, SUM_WARPS * 32, 0, s>>>(
            st, scr.res_e, abs_ ? scr.res_abs : nullptr, full, o.energy, o.abs_sum);
    }
    return count ? 1 : 2;  // launches issued
}

// div_by (score.cuh) against the IEEE quotient for every float of its range, both signs and
// 0, and every divisor it is used with: the EEF1 lambdas of the table and the H-bond sigma.
__global__ void k_div_selftest(unsigned long long* __restrict__ wrong) {
    unsigned long long bad = 0;
    const unsigned lo = (127 - 60) << 23, hi = (127 + 4) << 23;  // 2^-60 .. 16
#pragma unroll 1
    for (int t = 0; t <= 16; ++t) {
        const float d = t < 16 ? c_eef1[t].z : HB_SIGMA, y = __frcp_rn(d);
        for (unsigned u = lo + blockIdx.x * blockDim.x + threadIdx.x; u < hi; u += gridDim.x * blockDim.x) {
            const float r = __uint_as_float(u);
            bad += div_by(r, d, y) != __fdiv_rn(r, d);
            bad += div_by(-r, d, y) != __fdiv_rn(-r, d);
        }
        if (blockIdx.x == 0 && threadIdx.x == 0) bad += div_by(0.0f, d, y) != 0.0f;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) bad += 1.0f / HB_SIGMA != __frcp_rn(HB_SIGMA);
    if (bad) atomicAdd(wrong, bad);
}
void launch_div_selftest(cudaStream_t s, long long* wrong, int ctas) {
    k_div_selftest<<<ctas, 256, 0, s>>>((unsigned long long*)wrong);
}

void launch_score_state_count(cudaStream_t s, const StateView& st, const AgView* ags, long long* pairs,
                              uint32_t* err, const StateScoreScratch& scr, int grid_ctas) {
    if (st.n_cand <= 0) return;
    ScoreOut o{nullptr, nullptr, nullptr, pairs, err};
    launch_score_state(s, st, ags, 0, 0, o, scr, grid_ctas, NW_SCORE);
}

}  // namespace binder
