// k_mlp.cu — the learned mutation / rotamer proposal network on sm_100a.
//
// Network: 180 environment features -> 256 (SiLU) -> 256 (SiLU) -> 25 outputs
// (predicted Metropolis energy change of a mutation to each of the 20 amino acids
// and of each of the 5 rotamers).  Weights and activations are BF16, every sum is
// FP32.  The dense layers of training and of batched inference run on the 5th-gen
// tensor cores: one kernel, k_gemm_tc, computes C = A * B^T for K-major BF16
// operands with tcgen05.mma (one elected thread issues, the FP32 accumulator
// lives in tensor memory), operands staged in shared memory in the canonical
// no-swizzle core-matrix layout by 16-byte cp.async copies through a four-stage
// ring, and the epilogue (bias, SiLU, SiLU', BF16 packing, transposed copies for
// the weight-gradient GEMMs, split-K partials) fused on the tcgen05.ld path.
//
// Features of a residue (one warp per residue): a 20-way one-hot of its amino
// acid (none for a mutation query, amino acid MLP_NO_AA), then for each of 8
// radial shells of 1.25 A around its Calpha (0..10 A) the number of antigen
// Calphas of each of the 20 amino acids, log1p-scaled.
// Shell membership compares r^2 (the reference's f32 rounding) with the exact
// f32 squares of the shell radii, and log1p comes from a table filled on the
// host, so the features are bit-identical wherever they are computed.
#include <algorithm>

#include <cuda_bf16.h>

#include "kernels.h"
#include "mlp.cuh"

namespace binder {

__constant__ float c_log1p[MLP_COUNT_CAP + 1];

cudaError_t mlp_init_tables(const float* log1p_table) {
    return cudaMemcpyToSymbol(c_log1p, log1p_table, sizeof(float) * (MLP_COUNT_CAP + 1));
}

__device__ float mlp_log1p_count(int n) { return c_log1p[n < MLP_COUNT_CAP ? n : MLP_COUNT_CAP]; }

// ---- features ---------------------------------------------------------------------
// One warp per row: rows r = warp index; Calpha ca[r], amino acid aa[r], antigen
// ag[r] (index into ags).  X is BF16 [n_pad][MLP_K1] (columns >= MLP_IN zero);
// rows n..n_pad-1 are written as zeros.
__global__ void k_features(int n, int n_pad, const float* __restrict__ ca, const uint8_t* __restrict__ aa,
                           const int* __restrict__ ag, const AgView* __restrict__ ags, __nv_bfloat16* __restrict__ X) {
    __shared__ int s_cnt[8][MLP_SHELLS * N_AA];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r = blockIdx.x * 8 + warp;
    if (r >= n_pad) return;
    int* cnt = s_cnt[warp];
    __nv_bfloat16* row = X + (size_t)r * MLP_K1;
    if (r >= n) {
        for (int j = lane; j < MLP_K1; j += 32) row[j] = __float2bfloat16_rn(0.0f);
        return;
    }
    for (int j = lane; j < MLP_SHELLS * N_AA; j += 32) cnt[j] = 0;
    __syncwarp();
    const AgView& A = ags[ag ? ag[r] : 0];
    mlp_count_env(A.ca_atom, A.res_aa, A.n_res, ca[3 * r], ca[3 * r + 1], ca[3 * r + 2], cnt);
    __syncwarp();
    const int a = aa[r];
    for (int j = lane; j < MLP_K1; j += 32) {
        float v = 0.0f;
        if (j < N_AA) v = j == a ? 1.0f : 0.0f;
        else if (j < MLP_IN) v = mlp_log1p_count(cnt[j - N_AA]);
        row[j] = __float2bfloat16_rn(v);
    }
}

// host f32 features [n][MLP_IN] -> BF16 [n_pad][MLP_K1]
__global__ void k_pack_features(int n, int n_pad, const float* __restrict__ f, __nv_bfloat16* __restrict__ X) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)n_pad * MLP_K1) return;
    const int r = (int)(t / MLP_K1), j = (int)(t % MLP_K1);
    X[t] = __float2bfloat16_rn(r < n && j < MLP_IN ? f[(size_t)r * MLP_IN + j] : 0.0f);
}

// out[c][r] = in[r][c], 32 x 32 tiles through shared memory
__global__ void k_transpose_bf16(int rows, int cols, const __nv_bfloat16* __restrict__ in,
                                 __nv_bfloat16* __restrict__ out) {
    __shared__ __nv_bfloat16 t[32][33];
    const int c = blockIdx.x * 32 + threadIdx.x, r0 = blockIdx.y * 32;
    for (int i = threadIdx.y; i < 32; i += blockDim.y)
        if (r0 + i < rows && c < cols) t[i][threadIdx.x] = in[(size_t)(r0 + i) * cols + c];
    __syncthreads();
    const int r = r0 + threadIdx.x, c0 = blockIdx.x * 32;
    for (int i = threadIdx.y; i < 32; i += blockDim.y)
        if (c0 + i < cols && r < rows) out[(size_t)(c0 + i) * rows + r] = t[threadIdx.x][i];
}

// ---- tcgen05 helpers (PTX ISA 8.7, sm_100a) ---------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool valid) {
    const int n = valid ? 16 : 0;  // 0 bytes read: the 16 destination bytes are zero-filled
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}
// generic-proxy writes of shared memory made visible to the tensor core (async proxy)
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }

__device__ __forceinline__ void mbar_init(uint64_t* b, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(b)), "r"(count) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* b, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(smem_u32(b)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait for phase `parity` of barrier b; false when it gave up.
__device__ __forceinline__ bool mbar_wait(uint64_t* b, uint32_t parity, uint32_t max_polls = 1u << 22) {
    for (uint32_t i = 0; i < max_polls; ++i) {
        if (mbar_try_wait(b, parity)) return true;
        if (i > 64) __nanosleep(64);
    }
    return false;
}

__device__ __forceinline__ void tmem_alloc(uint32_t* dst, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(dst)),
                 "r"(ncols)
                 : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
// D[tmem] (+)= A[smem desc] * B[smem desc]^T, kind::f16 (BF16 inputs, FP32 accumulator)
__device__ __forceinline__ void tc_mma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                       uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// arrive on b once every tcgen05.mma this thread issued so far has completed
__device__ __forceinline__ void tc_commit(uint64_t* b) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(smem_u32(b))
                 : "memory");
}
// 32 lanes x 8 consecutive FP32 columns: thread t of the warp gets lane (base lane + t);
// the registers are valid after tc_ld_wait
__device__ __forceinline__ void tc_ld8(uint32_t taddr, float* v) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}

// Shared-memory matrix descriptor, K-major, no swizzle: core matrices of 8 rows x
// 16 bytes; lbo = byte distance between the two 8-element K halves of an MMA,
// sbo = byte distance between consecutive 8-row groups.
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
    d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t)1 << 46;  // descriptor version of sm_100
    return d;                // base offset 0, absolute LBO mode, layout type 0 = no swizzle
}
// Instruction descriptor of kind::f16: FP32 D, BF16 A and B, both K-major, M x N.
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// logistic sigmoid with the fast exponential and the approximate reciprocal (the
// results are rounded to BF16); the network tile of the Metropolis kernel uses the same
__device__ __forceinline__ float sigmoid_fast(float z) { return rcp_approx(1.0f + __expf(-z)); }

// ---- C[M x N] = A[M x K] * B[N x K]^T on the tensor cores ----------------------------
// One CTA of 256 threads per 128-row tile of A, 64-column tile of the outputs and K
// slice (split-K), its accumulator in tensor memory; up to three GEMMs in one launch (the
// weight gradients), their CTAs numbered one after another.  A rows >= m and K beyond the
// slice are zero-filled in shared memory.  Warps w and w + 4 read the accumulator lanes
// 32 (w % 4) .. +31 and split its columns.
// These GEMMs are small (8192 x 256 x 192 and the like), so what bounds them is one CTA's
// chain of loads, MMAs and epilogue: 64-column tiles give 4 times the CTAs and a quarter of
// the epilogue each, four stages keep three chunks of K in flight (training step of 8192
// rows: forward and data-gradient GEMMs 27 us each, now 18; weight gradients 43 + 43 +
// 25 us, then 34 in one launch).  A thread's copies of a chunk differ by constant strides,
// the tile's biases wait in shared memory and the SiLU' factors are loaded before the first
// accumulator is read (a training step 174 -> 167 us).  Every output sums over K in the
// same order as before.
constexpr int G_M = 128, G_K = 64, G_N = 64, G_THREADS = 256, G_STAGES = 4;
constexpr int G_STAGE_A = G_M * G_K * 2;                       // 16 KB
constexpr int G_STAGE = G_STAGE_A + G_N * G_K * 2;
constexpr int G_SMEM = G_STAGES * G_STAGE + 1024;
struct GemmGroup {
    GemmArgs g[3];
    int first[4];  // first CTA of each GEMM, then the total
};

// core-matrix offset of (row r, 8-element K group kg) inside a stage operand
__device__ __forceinline__ uint32_t cm_off(int r, int kg) { return (uint32_t)((r >> 3) * 1024 + kg * 128 + (r & 7) * 16); }

__global__ void __launch_bounds__(G_THREADS) k_gemm_tc(const __grid_constant__ GemmGroup group,
                                                        uint32_t* __restrict__ err) {
    extern __shared__ __align__(1024) unsigned char g_smem[];
    __shared__ __align__(8) uint64_t s_bar[G_STAGES];
    __shared__ uint32_t s_tmem;
    __shared__ float s_bias[G_N];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int which = (int)blockIdx.x >= group.first[2] ? 2 : (int)blockIdx.x >= group.first[1] ? 1 : 0;
    const GemmArgs& g = group.g[which];
    // CTA -> (row tile, K slice, column tile), columns fastest (they share the rows of A)
    const int n_tiles = (g.n + G_N - 1) / G_N, m_tiles = (g.m + G_M - 1) / G_M;
    int cta = (int)blockIdx.x - group.first[which];
    const int n0 = cta % n_tiles * G_N;
    cta /= n_tiles;
    const int m0 = cta % m_tiles * G_M, slice = cta / m_tiles;
    const int nt = min(G_N, g.n - n0);  // columns of this tile (16, 32, 48 or 64)
    const int k_begin = slice * g.k_split;
    const int k_end = min(g.k, k_begin + g.k_split);
    const int n_chunks = (k_end - k_begin + G_K - 1) / G_K;
    const uint32_t base = (smem_u32(g_smem) + 1023u) & ~1023u;
    const uint32_t ncols = nt <= 32 ? 32u : 64u;

    if (warp == 0) {
        tmem_alloc(&s_tmem, ncols);
        tmem_relinquish();
    }
    if (tid == 0)
        for (int i = 0; i < G_STAGES; ++i) mbar_init(&s_bar[i], 1);
    if (tid < nt)
        s_bias[tid] = g.e.bias && (g.e.mode == EPI_SILU || n0 + tid < g.e.n_valid) ? g.e.bias[n0 + tid] : 0.0f;
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    const uint32_t idesc = idesc_bf16(G_M, nt);

    // this thread's 16-byte pieces of a chunk: K group kg of rows r0, r0 + 32, ..
    constexpr int G_RSTEP = G_THREADS / 8;
    const int r0 = tid >> 3, kg = tid & 7;
    const uint32_t s_off = cm_off(r0, kg);
    const __nv_bfloat16* const a_src = g.a + (size_t)(m0 + r0) * g.lda + k_begin + kg * 8;
    const __nv_bfloat16* const b_src = g.b + (size_t)(n0 + r0) * g.ldb + k_begin + kg * 8;
    const size_t a_step = (size_t)G_RSTEP * g.lda, b_step = (size_t)G_RSTEP * g.ldb;
    const int a_rows = g.m - m0 - r0, b_rows = nt - r0, k_left = k_end - k_begin - kg * 8;
    auto load_chunk = [&](int c) {  // (a group is committed for chunks past the end, too)
        if (c < n_chunks) {
            const uint32_t sa = base + (c % G_STAGES) * G_STAGE + s_off, sb = sa + G_STAGE_A;
            const bool k_ok = c * G_K < k_left;
#pragma unroll
            for (int i = 0; i < G_M / G_RSTEP; ++i) {
                const bool in = k_ok && i * G_RSTEP < a_rows;
                cp_async16(sa + i * (G_RSTEP / 8) * 1024, in ? a_src + i * a_step + c * G_K : g.a, in);
            }
#pragma unroll
            for (int i = 0; i < G_N / G_RSTEP; ++i)
                if (i * G_RSTEP < b_rows)
                    cp_async16(sb + i * (G_RSTEP / 8) * 1024, k_ok ? b_src + i * b_step + c * G_K : g.b, k_ok);
        }
        cp_async_commit();
    };

    bool ok = true;
    for (int c = 0; c < G_STAGES - 1; ++c) load_chunk(c);
    for (int c = 0; c < n_chunks && ok; ++c) {
        cp_async_wait<G_STAGES - 2>();
        fence_proxy_async();
        __syncthreads();
        if (tid == 0) {
            tc_fence_after();
            const uint32_t sa = base + (c % G_STAGES) * G_STAGE, sb = sa + G_STAGE_A;
            const int kc = min(G_K, k_end - (k_begin + c * G_K));
            for (int j = 0; j < kc / 16; ++j)
                tc_mma(tmem, smem_desc(sa + 256 * j, 128, 1024), smem_desc(sb + 256 * j, 128, 1024), idesc,
                       (c > 0 || j > 0) ? 1u : 0u);
            tc_commit(&s_bar[c % G_STAGES]);
        }
        // the next chunk's stage was read by the MMAs of chunk c-1: wait for them first
        if (c >= 1 && c + G_STAGES - 1 < n_chunks) ok = mbar_wait(&s_bar[(c - 1) % G_STAGES], ((c - 1) / G_STAGES) & 1);
        if (ok) load_chunk(c + G_STAGES - 1);
    }
    cp_async_wait<0>();
    if (ok && n_chunks > 0) ok = mbar_wait(&s_bar[(n_chunks - 1) % G_STAGES], ((n_chunks - 1) / G_STAGES) & 1);
    // every thread saw the same waits; a thread that gave up raises the flag
    if (!ok && err) atomicOr(err, ERRF_TIMEOUT);
    tc_fence_after();

    // ---- epilogue: warp w owns accumulator lanes (rows) 32 (w % 4) .. +31, columns
    //      [n/2 * (w / 4), n/2 * (w / 4 + 1)) (multiples of 8) ----
    const int wl = warp & 3, half = warp >> 2;
    const int row = m0 + wl * 32 + lane;
    const bool row_ok = row < g.e.m_valid;
    const GemmEpi& e = g.e;
    const int n8 = nt / 8;                         // column groups of 8
    const int cg0 = (n8 * half) / 2, cg1 = (n8 * (half + 1)) / 2;
    uint4 spv[G_N / 16];  // EPI_DSILU: the row's factors, all groups' loads in flight together
#pragma unroll
    for (int q = 0; q < G_N / 16; ++q)
        if (e.mode == EPI_DSILU && row_ok && cg0 + q < cg1)
            spv[q] = *(const uint4*)(e.sp + (size_t)row * e.ldsp + n0 + (cg0 + q) * 8);
#pragma unroll
    for (int q = 0; q < G_N / 16; ++q) {
        const int cgi = cg0 + q;
        if (cgi >= cg1 || !ok) continue;
        const int c0 = n0 + cgi * 8;
        float v[8];
        if (n_chunks > 0) tc_ld8(tmem + ((uint32_t)(wl * 32) << 16) + (uint32_t)(cgi * 8), v);
        else {
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = 0.0f;
        }
        if (e.mode == EPI_F32 || e.mode == EPI_PARTIAL) {
            if (row_ok) {
                float* out = e.c + (e.mode == EPI_PARTIAL ? (size_t)slice * e.part_stride : 0) +
                             (size_t)row * e.ldc;
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (c0 + i < e.n_valid) out[c0 + i] = v[i] + s_bias[cgi * 8 + i];
            }
        } else {
            __align__(16) __nv_bfloat16 h[8];
            __align__(16) __nv_bfloat16 dz[8];
            if (e.mode == EPI_DSILU && row_ok) *(uint4*)dz = spv[q];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                float o = 0.0f, d = 0.0f;
                if (row_ok) {
                    if (e.mode == EPI_SILU) {
                        const float z = v[i] + s_bias[cgi * 8 + i];
                        const float sg = sigmoid_fast(z);
                        o = z * sg;
                        d = sg * (1.0f + z * (1.0f - sg));
                    } else {  // EPI_DSILU
                        o = v[i] * __bfloat162float(dz[i]);
                    }
                }
                h[i] = __float2bfloat16_rn(o);
                dz[i] = __float2bfloat16_rn(d);
                if (e.ht && row < e.ht_rows) e.ht[(size_t)(c0 + i) * e.ldht + row] = h[i];
            }
            if (e.h && row < e.h_rows) *(uint4*)(e.h + (size_t)row * e.ldh + c0) = *(const uint4*)h;
            if (e.mode == EPI_SILU && e.sp && row < e.h_rows)
                *(uint4*)(e.sp + (size_t)row * e.ldsp + c0) = *(const uint4*)dz;
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, ncols);
    }
}

// The bounded wait on a barrier nothing arrives on: raises ERRF_TIMEOUT after
// max_polls polls and returns (the error path of every tcgen05 wait, exercised
// without a fault).
__global__ void k_wait_selftest(uint32_t max_polls, uint32_t* __restrict__ err) {
    __shared__ __align__(8) uint64_t bar;
    mbar_init(&bar, 1);
    __syncwarp();
    if (!mbar_wait(&bar, 0, max_polls) && err) atomicOr(err, ERRF_TIMEOUT);
}

cudaError_t launch_wait_selftest(cudaStream_t s, uint32_t max_polls, uint32_t* err) {
    k_wait_selftest<<<1, 1, 0, s>>>(max_polls, err);
    return cudaGetLastError();
}

cudaError_t launch_gemm_tc(cudaStream_t s, const GemmArgs* g, int count, uint32_t* err) {
    if (count < 1 || count > 3) return cudaErrorInvalidValue;
    GemmGroup group;
    int ctas = 0;
    for (int i = 0; i < 3; ++i) {
        group.first[i] = ctas;
        if (i >= count) {
            group.first[i] = INT32_MAX;  // no CTA
            continue;
        }
        if (g[i].n < 16 || g[i].n > 256 || g[i].n % 16 || g[i].k % 16 || g[i].lda % 8 || g[i].ldb % 8 ||
            g[i].k_split % G_K)
            return cudaErrorInvalidValue;
        group.g[i] = g[i];
        const int m_tiles = (g[i].m + G_M - 1) / G_M, k_slices = (g[i].k + g[i].k_split - 1) / g[i].k_split;
        ctas += std::max(0, m_tiles * k_slices) * ((g[i].n + G_N - 1) / G_N);
    }
    group.first[3] = ctas;
    if (ctas == 0) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(k_gemm_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, G_SMEM);
    if (e) return e;
    k_gemm_tc<<<ctas, G_THREADS, G_SMEM, s>>>(group, err);
    return cudaGetLastError();
}

// ---- training kernels -------------------------------------------------------------
// Huber loss of the predicted energy change against the logged one; writes the
// output gradient dY (BF16 [m_pad][32] and its transpose [32][m_pad]) and adds the
// batch loss.  Prediction: y[action] - y[ref] with a reference output (ref >= 0:
// a mutation query, ref = the amino acid before the move; a row with ref == action
// carries nothing), else y[action].  Rows >= m get zero gradients.
__global__ void k_mlp_loss(int m, int m_pad, const float* __restrict__ Y, const int* __restrict__ action,
                           const int* __restrict__ ref, const float* __restrict__ target, float delta,
                           __nv_bfloat16* __restrict__ dY, __nv_bfloat16* __restrict__ dYt, double* __restrict__ loss) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= m_pad) return;
    int a = -1, b = -1;
    float g = 0.0f, l = 0.0f;
    if (r < m) {
        a = action[r];
        b = ref ? ref[r] : -1;
        if (b == a) {
            a = b = -1;
        } else {
            const float* y = Y + (size_t)r * MLP_OUT_PAD;
            const float d = (b >= 0 ? y[a] - y[b] : y[a]) - target[r];
            const float ad = fabsf(d);
            l = ad <= delta ? 0.5f * d * d : delta * (ad - 0.5f * delta);
            g = fminf(fmaxf(d, -delta), delta) / (float)m;
        }
    }
    __align__(16) __nv_bfloat16 row[MLP_OUT_PAD];
#pragma unroll
    for (int j = 0; j < MLP_OUT_PAD; ++j) {
        row[j] = __float2bfloat16_rn(j == a ? g : (j == b ? -g : 0.0f));
        dYt[(size_t)j * m_pad + r] = row[j];
    }
#pragma unroll
    for (int j = 0; j < MLP_OUT_PAD; j += 8) *(uint4*)(dY + (size_t)r * MLP_OUT_PAD + j) = *(const uint4*)(row + j);
    // warp sum in fixed order, one atomic per warp
    for (int o = 16; o; o >>= 1) l += __shfl_down_sync(0xffffffffu, l, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(loss, (double)l / (double)m);
}

// out[j] = sum over k < m of G[j][k] (BF16 rows) for the rows of up to three matrices (the
// bias gradients), one CTA per row: 256 threads stage 4096 columns at a time, then the
// first warp's lane l adds k = l, l + 32, .. and the lanes are folded, a fixed order.  (A
// warp reading its 2-byte entries from global memory: 11 us for 256 rows of 8192.)
constexpr int RS_COLS = 4096;
__global__ void __launch_bounds__(256) k_rowsum_bf16(RowSums rs) {
    __shared__ __align__(16) __nv_bfloat16 s_row[RS_COLS];
    int j = blockIdx.x, w = 0;
    while (j >= rs.rows[w]) j -= rs.rows[w++];
    const __nv_bfloat16* G = rs.g[w] + (size_t)j * rs.m;
    const int tid = threadIdx.x;
    float s = 0.0f;
    for (int k0 = 0; k0 < rs.m; k0 += RS_COLS) {
        const int n = min(RS_COLS, rs.m - k0);  // a multiple of 128: rows are padded to the GEMM tile
        for (int i = tid * 8; i < n; i += 256 * 8) *(uint4*)(s_row + i) = *(const uint4*)(G + k0 + i);
        __syncthreads();
        if (tid < 32) {
#pragma unroll 8
            for (int k = tid; k < n; k += 32) s += __bfloat162float(s_row[k]);
        }
        __syncthreads();
    }
    if (tid >= 32) return;
    for (int o = 16; o; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (tid == 0) rs.out[w][j] = s;
}

// The weight gradients from their split-K partials (summed slice after slice) into g
// (whose bias entries are there already), and with ADAM the update (Kingma & Ba 2015) of
// the FP32 master parameters and of their BF16 copies: row-major, transposed and in
// fragment order.  One thread per parameter (three reductions, the update and the packing
// took five launches).
__device__ __forceinline__ void store_frag(uint4* f, int K, int n, int k, __nv_bfloat16 v) {
    const int g = n & 7, hi = n >> 3 & 1, c = k & 7, half = k >> 3 & 1;
    ((__nv_bfloat16*)&f[frag_index(n >> 4, k >> 4, g * 4 + (c >> 1), K)])[(half * 2 + hi) * 2 + (c & 1)] = v;
}
template <bool ADAM>
__global__ void __launch_bounds__(256) k_update(MlpPartials part, float* __restrict__ w, float* __restrict__ g,
                                                float* __restrict__ m1, float* __restrict__ m2, float lr, float b1,
                                                float b2, float eps, float bc1, float bc2, MlpBf16 o) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= MLP_N_PARAMS) return;
    const int l = i < MLP_OFF_B1 ? 0 : i >= MLP_OFF_W2 && i < MLP_OFF_B2 ? 1 : i >= MLP_OFF_W3 && i < MLP_OFF_B3 ? 2 : -1;
    const int t = l == 0 ? i - MLP_OFF_W1 : l == 1 ? i - MLP_OFF_W2 : i - MLP_OFF_W3;
    float gi;
    if (l >= 0) {
        const float* p = part.p[l] + t;
        const size_t stride = l == 0 ? MLP_H * MLP_K1 : l == 1 ? MLP_H * MLP_H : MLP_OUT_PAD * MLP_H;
        gi = 0.0f;
#pragma unroll 8
        for (int q = 0; q < part.slices; ++q) gi += p[q * stride];
        g[i] = gi;
    } else {
        gi = g[i];
    }
    if (!ADAM) return;
    const float a = b1 * m1[i] + (1.0f - b1) * gi;
    const float b = b2 * m2[i] + (1.0f - b2) * gi * gi;
    m1[i] = a;
    m2[i] = b;
    float x = w[i];
    x -= lr * (a / bc1) / (sqrtf(b / bc2) + eps);
    w[i] = x;
    const __nv_bfloat16 v = __float2bfloat16_rn(x);
    if (l == 0) {
        o.w1[t] = v;
        store_frag(o.f1, MLP_K1, t / MLP_K1, t % MLP_K1, v);
    } else if (l == 1) {
        const int n = t / MLP_H, k = t % MLP_H;
        o.w2[t] = v;
        o.w2t[(size_t)k * MLP_H + n] = v;
        store_frag(o.f2, MLP_H, n, k, v);
    } else if (l == 2) {
        const int n = t / MLP_H, k = t % MLP_H;
        o.w3[t] = v;
        o.w3t[(size_t)k * MLP_OUT_PAD + n] = v;
        store_frag(o.f3, MLP_H, n, k, v);
    }
}

// 16-byte fragment-order element (mt, s, lane) of W [N][K] at w (FP32 master copy)
__device__ __forceinline__ uint4 pack_frag(const float* __restrict__ w, int K, int mt, int s, int lane) {
    const int g = lane / 4, c = 2 * (lane % 4), k0 = 16 * s;
    const float* r0 = w + (size_t)(16 * mt + g) * K + k0;
    const float* r1 = w + (size_t)(16 * mt + g + 8) * K + k0;
    const __nv_bfloat162 a0 = __floats2bfloat162_rn(r0[c], r0[c + 1]);
    const __nv_bfloat162 a1 = __floats2bfloat162_rn(r1[c], r1[c + 1]);
    const __nv_bfloat162 a2 = __floats2bfloat162_rn(r0[8 + c], r0[9 + c]);
    const __nv_bfloat162 a3 = __floats2bfloat162_rn(r1[8 + c], r1[9 + c]);
    return make_uint4(*(const uint32_t*)&a0, *(const uint32_t*)&a1, *(const uint32_t*)&a2, *(const uint32_t*)&a3);
}

// BF16 copies of the weights: W1 [H][192], W2 [H][H] and W2^T, W3 [32][H] and W3^T,
// and the fragment-order copies of W1, W2, W3 (one thread per element of the
// largest of them)
__global__ void k_pack_weights(const float* __restrict__ p, MlpBf16 o) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < (MLP_H / 16) * (MLP_K1 / 16) * 32) {
        const int lane = t % 32, ks = (t / 32) % (MLP_K1 / 16), mt = t / (32 * (MLP_K1 / 16));
        o.f1[t] = pack_frag(p + MLP_OFF_W1, MLP_K1, mt, ks, lane);
    }
    if (t < (MLP_H / 16) * (MLP_H / 16) * 32) {
        const int lane = t % 32, ks = (t / 32) % (MLP_H / 16), mt = t / (32 * (MLP_H / 16));
        o.f2[t] = pack_frag(p + MLP_OFF_W2, MLP_H, mt, ks, lane);
    }
    if (t < (MLP_OUT_PAD / 16) * (MLP_H / 16) * 32) {
        const int lane = t % 32, ks = (t / 32) % (MLP_H / 16), mt = t / (32 * (MLP_H / 16));
        o.f3[t] = pack_frag(p + MLP_OFF_W3, MLP_H, mt, ks, lane);
    }
    if (t < MLP_H * MLP_K1) o.w1[t] = __float2bfloat16_rn(p[MLP_OFF_W1 + t]);
    if (t < MLP_H * MLP_H) {
        const int n = t / MLP_H, k = t % MLP_H;
        const __nv_bfloat16 v = __float2bfloat16_rn(p[MLP_OFF_W2 + t]);
        o.w2[t] = v;
        o.w2t[(size_t)k * MLP_H + n] = v;
    }
    if (t < MLP_OUT_PAD * MLP_H) {
        const int n = t / MLP_H, k = t % MLP_H;
        const __nv_bfloat16 v = __float2bfloat16_rn(p[MLP_OFF_W3 + t]);
        o.w3[t] = v;
        o.w3t[(size_t)k * MLP_OUT_PAD + n] = v;
    }
}

// Gather a minibatch of logged tuples: features input rows, action, reference
// output, target.  A mutation is a query without amino acid (MLP_NO_AA) whose
// energy change is predicted as y[new] - y[old]; a rotamer move queries with its
// amino acid and is predicted by y[20 + rotamer].
// The rows are drawn with the Philox generator: row r takes tuple
// (u n_tuples) >> 32.
__global__ void k_gather_tuples(int m, int n_tuples, uint64_t seed, uint32_t step, const MlpTuple* __restrict__ tup,
                                float* __restrict__ ca, uint8_t* __restrict__ aa, int* __restrict__ ag,
                                int* __restrict__ action, int* __restrict__ ref, float* __restrict__ target) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= m) return;
    const U4 u = philox((uint32_t)r, step, 0xB47Cu, 0u, (uint32_t)seed, (uint32_t)(seed >> 32));
    const MlpTuple t = tup[(int)(((uint64_t)u.x * (uint32_t)n_tuples) >> 32)];
    const bool mut = t.action < N_AA;
    ca[3 * r] = t.x;
    ca[3 * r + 1] = t.y;
    ca[3 * r + 2] = t.z;
    aa[r] = mut ? (uint8_t)MLP_NO_AA : t.aa;
    ag[r] = t.antigen;
    action[r] = t.action;
    ref[r] = mut ? (int)t.aa : -1;
    target[r] = t.delta_e;
}

// ---- launchers ----------------------------------------------------------------------
void launch_features(cudaStream_t s, int n, int n_pad, const float* ca, const uint8_t* aa, const int* ag,
                     const AgView* ags, __nv_bfloat16* X) {
    if (n_pad > 0) k_features<<<(n_pad + 7) / 8, 256, 0, s>>>(n, n_pad, ca, aa, ag, ags, X);
}
void launch_pack_features(cudaStream_t s, int n, int n_pad, const float* f, __nv_bfloat16* X) {
    const long long t = (long long)n_pad * MLP_K1;
    if (t > 0) k_pack_features<<<(unsigned)((t + 255) / 256), 256, 0, s>>>(n, n_pad, f, X);
}
void launch_transpose_bf16(cudaStream_t s, int rows, int cols, const __nv_bfloat16* in, __nv_bfloat16* out) {
    if (rows > 0 && cols > 0) k_transpose_bf16<<<dim3((cols + 31) / 32, (rows + 31) / 32), dim3(32, 8), 0, s>>>(rows, cols, in, out);
}
void launch_mlp_loss(cudaStream_t s, int m, int m_pad, const float* Y, const int* action, const int* ref,
                     const float* target, float delta, __nv_bfloat16* dY, __nv_bfloat16* dYt, double* loss) {
    if (m_pad > 0)
        k_mlp_loss<<<(m_pad + 255) / 256, 256, 0, s>>>(m, m_pad, Y, action, ref, target, delta, dY, dYt, loss);
}
void launch_rowsum_bf16(cudaStream_t s, const RowSums& rs) {
    const int rows = rs.rows[0] + rs.rows[1] + rs.rows[2];
    if (rows > 0) k_rowsum_bf16<<<rows, 256, 0, s>>>(rs);
}
void launch_update(cudaStream_t s, const MlpPartials& part, float* w, float* g, float* m1, float* m2, float lr,
                   float b1, float b2, float eps, float bc1, float bc2, const MlpBf16& o, bool adam) {
    const int n = (MLP_N_PARAMS + 255) / 256;
    if (adam) k_update<true><<<n, 256, 0, s>>>(part, w, g, m1, m2, lr, b1, b2, eps, bc1, bc2, o);
    else k_update<false><<<n, 256, 0, s>>>(part, w, g, m1, m2, lr, b1, b2, eps, bc1, bc2, o);
}
void launch_pack_weights(cudaStream_t s, const float* p, const MlpBf16& o) {
    const int n = std::max(MLP_H * MLP_K1, std::max(MLP_H * MLP_H, MLP_OUT_PAD * MLP_H));
    k_pack_weights<<<(n + 255) / 256, 256, 0, s>>>(p, o);
}
void launch_gather_tuples(cudaStream_t s, int m, int n_tuples, uint64_t seed, uint32_t step, const MlpTuple* tup,
                          float* ca, uint8_t* aa, int* ag, int* action, int* ref, float* target) {
    if (m > 0)
        k_gather_tuples<<<(m + 255) / 256, 256, 0, s>>>(m, n_tuples, seed, step, tup, ca, aa, ag, action, ref, target);
}

}  // namespace binder
