// True 32-bit matrix product for the float path:  C[M,N] = A[M,K] * W[N,K]^T.
//
// Plain FMA on float operands with float accumulation: no TF32, no split
// operands, no tensor cores.  The reference has no such path; its products always
// round the operands to half precision (src/layers/linear.cpp:67-77).
// W is stored as the checkpoint stores it, [out_features, in_features] row-major.
//
// One order of summation for every M: K is cut into S slices (by N and K alone), a slice is one chain of FMAs in rising k, and the
// slices are added in their order.  A row's result therefore does not depend on which other rows are in the call,
// and each of the kernels below may be picked by speed alone.  The S slices of a tile are the S CTAs of a cluster;
// they hand their partial tiles over through distributed shared memory.
//
// Two kernels, by what bounds the product:
//   rows  (few M)    the weights are read once and each is used M times: bound by memory.  A thread owns one or two columns
//                    of C (rows of W) and up to 16 rows; W passes through a ring of asynchronous copies, 128-byte pieces of a row.
//   tiles (many M)   bound by the FMA pipe.  128 columns and 32, 64 or 128 rows a CTA; a thread holds TM x 16 sums as packed
//                    pairs (fma.rn.f32x2), because at 8 x 16 the shared-memory reads take three quarters of the FMAs' time
//                    (at 8 x 8 as long as the FMAs).
// Every edge is guarded, so any M, N, K >= 1 and any strides work; 16-byte copies are used where addresses, strides and K allow
// them, single floats elsewhere.
#include "common.cuh"
#include <cooperative_groups.h>

namespace {

namespace cg = cooperative_groups;

// Slices of a product with N columns.  A product with few columns has too few tiles to fill the device (3,584 columns are 28
// tiles of the tiles kernel, 56 of the rows kernel), so its K is cut eight ways: [3,584 x 18,944] by 3 rows takes 67 us in 8
// slices and 103 in 4, by 500 rows 1,439 and 1,668.  One with many columns fills it anyway, and smaller clusters are placed better
// and pass less through distributed shared memory: [37,888 x 3,584] by 500 rows 2,779 us in 8 slices, 2,590 in 4, 2,432 in 2
// (by 3 rows 104 and 108 in 8 and 4).  Short sums stay whole.
__host__ __device__ inline int f32_slices(int N, int K) { return K < 512 ? 1 : N >= 16384 ? 2 : K < 2048 ? 4 : 8; }
// first k of a slice: slices are multiples of 32 long, so that a copy of 32 k's never crosses into the next one
__host__ __device__ inline int f32_slice_len(int K, int slices) { return ((K + slices - 1) / slices + 31) & ~31; }

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool valid) {
    const int bytes = valid ? 16 : 0;                      // 0: nothing is read, the 16 bytes become zero
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

typedef unsigned long long pair_t;
__device__ __forceinline__ pair_t pair_of(float a, float b) {
    pair_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void pair_split(pair_t p, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(p)); }
__device__ __forceinline__ void pair_fma(pair_t& acc, pair_t a, pair_t b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b)); }

struct F32Args {
    const float *A, *W;
    float* C;
    int M, N, K, lda, ldw, ldc;
    int slices;                  // CTAs of a cluster: block b is slice b % slices of tile b / slices
};

// The slices' sums of `count` outputs stand in each CTA's shared memory at `part`; CTA r of the cluster adds and stores its share.
// at(e, m, n): the row and column of output e.
template <int THREADS, typename At>
__device__ __forceinline__ void add_slices(const F32Args& a, float* part, int count, At at) {
    cg::cluster_group cluster = cg::this_cluster();
    const int slices = a.slices, rank = (int)cluster.block_rank();
    if (slices == 1) {
        __syncthreads();
        for (int e = threadIdx.x; e < count; e += THREADS) {
            int m, n;
            at(e, m, n);
            if (m < a.M && n < a.N) a.C[(size_t)m * a.ldc + n] = part[e];
        }
        return;
    }
    cluster.sync();
    const int share = count / slices;                      // count is a multiple of 128, slices at most 8
    for (int e = rank * share + threadIdx.x; e < (rank + 1) * share; e += THREADS) {
        int m, n;
        at(e, m, n);
        if (m >= a.M || n >= a.N) continue;
        float v[8];
#pragma unroll
        for (int s = 0; s < 8; ++s) v[s] = s < slices ? *cluster.map_shared_rank(part + e, s) : 0.0f;
        float sum = v[0];
#pragma unroll
        for (int s = 1; s < 8; ++s)
            if (s < slices) sum += v[s];
        a.C[(size_t)m * a.ldc + n] = sum;
    }
    cluster.sync();                                        // nobody leaves while its sums are being read
}

// ---- few rows: groups of at most MT rows, NT threads with TN columns each
template <int MT, int TN, int NT, int BK_> struct RowsCfg {
    static constexpr int BN = NT * TN, BK = BK_, LD = BK + 4;              // eight lanes' 16-byte reads meet all 32 banks
    static constexpr int STAGE_FLOATS = BN * LD + MT * BK;
    static constexpr int STAGES = STAGE_FLOATS * 4 * 4 <= 76 * 1024 ? 4 : 3;
    static constexpr int SMEM = STAGES * STAGE_FLOATS * 4;
};

template <int MT, int TN, int NT, int BK_, bool VEC>
__global__ void __launch_bounds__(NT)
gemm_f32_rows_kernel(F32Args a) {
    using Cfg = RowsCfg<MT, TN, NT, BK_>;
    extern __shared__ __align__(16) float smem[];
    pdl_start();
    const int tile = blockIdx.x / a.slices, slice = blockIdx.x % a.slices, len = f32_slice_len(a.K, a.slices);
    const int groups = (a.M + MT - 1) / MT, m0 = tile % groups * MT;       // groups that share weights run together
    const int k_lo = min(a.K, slice * len), k_hi = min(a.K, k_lo + len), n0 = tile / groups * Cfg::BN;
    const int steps = (k_hi - k_lo + Cfg::BK - 1) / Cfg::BK;
    constexpr int LANES = Cfg::BK / 4, PASS = NT / LANES;                  // LANES threads copy a row's piece, PASS rows at a time
    const int chunk = threadIdx.x % LANES, row0 = threadIdx.x / LANES;

    auto load = [&](int step) {
        float* ws = smem + (step % Cfg::STAGES) * Cfg::STAGE_FLOATS;
        float* as = ws + Cfg::BN * Cfg::LD;
        const int k = k_lo + step * Cfg::BK + chunk * 4;
        if (VEC) {
#pragma unroll
            for (int i = 0; i < Cfg::BN / PASS; ++i) {
                const int r = row0 + PASS * i, n = n0 + r;
                const bool ok = n < a.N && k < k_hi;
                cp_async16(cx_smem(ws + r * Cfg::LD + chunk * 4), ok ? a.W + (size_t)n * a.ldw + k : a.W, ok);
            }
            for (int r = row0; r < MT; r += PASS) {
                const bool ok = m0 + r < a.M && k < k_hi;
                cp_async16(cx_smem(as + r * Cfg::BK + chunk * 4), ok ? a.A + (size_t)(m0 + r) * a.lda + k : a.A, ok);
            }
        } else {
            for (int i = 0; i < Cfg::BN / PASS; ++i) {
                const int r = row0 + PASS * i, n = n0 + r;
                for (int j = 0; j < 4; ++j)
                    ws[r * Cfg::LD + chunk * 4 + j] = n < a.N && k + j < k_hi ? a.W[(size_t)n * a.ldw + k + j] : 0.0f;
            }
            for (int r = row0; r < MT; r += PASS)
                for (int j = 0; j < 4; ++j)
                    as[r * Cfg::BK + chunk * 4 + j] = m0 + r < a.M && k + j < k_hi ? a.A[(size_t)(m0 + r) * a.lda + k + j] : 0.0f;
        }
    };

    float acc[MT][TN];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int t = 0; t < TN; ++t) acc[m][t] = 0.0f;

    for (int s = 0; s < Cfg::STAGES - 1; ++s) {
        if (s < steps) load(s);
        cp_commit();
    }
    for (int step = 0; step < steps; ++step) {
        cp_wait<Cfg::STAGES - 2>();
        __syncthreads();                                   // this stage has arrived; the one before it has been read by all
        if (step + Cfg::STAGES - 1 < steps) load(step + Cfg::STAGES - 1);
        cp_commit();
        const float* ws = smem + (step % Cfg::STAGES) * Cfg::STAGE_FLOATS;
        const float* as = ws + Cfg::BN * Cfg::LD;
#pragma unroll 8
        for (int kk = 0; kk < Cfg::BK; kk += 4) {
            float4 w[TN];
#pragma unroll
            for (int t = 0; t < TN; ++t) w[t] = *reinterpret_cast<const float4*>(ws + (threadIdx.x + t * NT) * Cfg::LD + kk);
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                const float4 x = *reinterpret_cast<const float4*>(as + m * Cfg::BK + kk);
#pragma unroll
                for (int t = 0; t < TN; ++t) {
                    acc[m][t] = fmaf(x.x, w[t].x, acc[m][t]);
                    acc[m][t] = fmaf(x.y, w[t].y, acc[m][t]);
                    acc[m][t] = fmaf(x.z, w[t].z, acc[m][t]);
                    acc[m][t] = fmaf(x.w, w[t].w, acc[m][t]);
                }
            }
        }
    }
    cp_wait<0>();
    __syncthreads();
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int t = 0; t < TN; ++t) smem[m * Cfg::BN + t * NT + threadIdx.x] = acc[m][t];
    add_slices<NT>(a, smem, MT * Cfg::BN, [&](int e, int& m, int& n) { m = m0 + e / Cfg::BN; n = n0 + e % Cfg::BN; });
}

// ---- many rows
template <int TM> struct TileCfg {
    static constexpr int BM = 16 * TM, BN = 128, BK = 16, LDA = BM + 4, LDW = BN + 4;
    static constexpr int STAGE_FLOATS = BK * (LDA + LDW);
    static constexpr int FLOATS = 2 * STAGE_FLOATS > BM * BN ? 2 * STAGE_FLOATS : BM * BN;
    static constexpr int SMEM = FLOATS * 4;
    static constexpr int THREADS = 128, A_VECS = BM * BK / 4 / THREADS, W_VECS = BN * BK / 4 / THREADS;      // 16-byte pieces a thread stages
};

template <int TM, bool VEC>
__global__ void __launch_bounds__(128, 2)
gemm_f32_tiles_kernel(F32Args a) {
    using Cfg = TileCfg<TM>;
    constexpr int TN = 16;
    extern __shared__ __align__(16) float smem[];
    pdl_start();
    const int tile = blockIdx.x / a.slices, slice = blockIdx.x % a.slices, len = f32_slice_len(a.K, a.slices);
    const int k_lo = min(a.K, slice * len), k_hi = min(a.K, k_lo + len);
    const int row_tiles = (a.M + Cfg::BM - 1) / Cfg::BM;
    const int m0 = tile % row_tiles * Cfg::BM, n0 = tile / row_tiles * Cfg::BN;               // tiles that share weights run together
    const int steps = (k_hi - k_lo + Cfg::BK - 1) / Cfg::BK;
    const int quad = threadIdx.x & 3, row0 = threadIdx.x >> 2;             // four threads read the 64 bytes of a row's k's

    float4 sa[Cfg::A_VECS], sw[Cfg::W_VECS];
    auto read = [&](const float* base, int ld, int row, int rows, int k) -> float4 {
        if (row >= rows) return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        const float* p = base + (size_t)row * ld + k;
        if (VEC) return k < k_hi ? *reinterpret_cast<const float4*>(p) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        return make_float4(k < k_hi ? p[0] : 0.0f, k + 1 < k_hi ? p[1] : 0.0f, k + 2 < k_hi ? p[2] : 0.0f, k + 3 < k_hi ? p[3] : 0.0f);
    };
    auto fetch = [&](int step) {
        const int k = k_lo + step * Cfg::BK + quad * 4;
#pragma unroll
        for (int i = 0; i < Cfg::A_VECS; ++i) sa[i] = read(a.A, a.lda, m0 + row0 + 32 * i, a.M, k);
#pragma unroll
        for (int i = 0; i < Cfg::W_VECS; ++i) sw[i] = read(a.W, a.ldw, n0 + row0 + 32 * i, a.N, k);
    };
    auto put = [&](int step) {                                             // k-major: a thread's sums read runs of rows and columns
        float* as = smem + (step & 1) * Cfg::STAGE_FLOATS;
        float* ws = as + Cfg::BK * Cfg::LDA;
#pragma unroll
        for (int i = 0; i < Cfg::A_VECS; ++i) {
            float* p = as + quad * 4 * Cfg::LDA + row0 + 32 * i;
            p[0] = sa[i].x; p[Cfg::LDA] = sa[i].y; p[2 * Cfg::LDA] = sa[i].z; p[3 * Cfg::LDA] = sa[i].w;
        }
#pragma unroll
        for (int i = 0; i < Cfg::W_VECS; ++i) {
            float* p = ws + quad * 4 * Cfg::LDW + row0 + 32 * i;
            p[0] = sw[i].x; p[Cfg::LDW] = sw[i].y; p[2 * Cfg::LDW] = sw[i].z; p[3 * Cfg::LDW] = sw[i].w;
        }
    };

    // thread (tm, tn): rows tm * TM .., columns tn * 4 + 32 j ..; a warp is 4 x 8 threads
    const int tm = threadIdx.x >> 3, tn = threadIdx.x & 7;
    pair_t acc[TM][TN / 2];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0ull;                 // (0.0f, 0.0f)

    if (steps > 0) {
        fetch(0);
        put(0);
    }
    __syncthreads();
    for (int step = 0; step < steps; ++step) {
        if (step + 1 < steps) fetch(step + 1);
        const float* as = smem + (step & 1) * Cfg::STAGE_FLOATS + tm * TM;
        const float* ws = smem + (step & 1) * Cfg::STAGE_FLOATS + Cfg::BK * Cfg::LDA + tn * 4;
#pragma unroll
        for (int k = 0; k < Cfg::BK; ++k) {
            float x[TM];
            pair_t w[TN / 2];
            if (TM == 2) *reinterpret_cast<float2*>(x) = *reinterpret_cast<const float2*>(as + k * Cfg::LDA);
            else
#pragma unroll
                for (int i = 0; i < TM; i += 4) *reinterpret_cast<float4*>(x + i) = *reinterpret_cast<const float4*>(as + k * Cfg::LDA + i);
#pragma unroll
            for (int j = 0; j < TN / 4; ++j) {
                const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(ws + k * Cfg::LDW + 32 * j);
                w[2 * j] = v.x;
                w[2 * j + 1] = v.y;
            }
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const pair_t xx = pair_of(x[i], x[i]);
#pragma unroll
                for (int j = 0; j < TN / 2; ++j) pair_fma(acc[i][j], xx, w[j]);
            }
        }
        if (step + 1 < steps) put(step + 1);               // the other half: read last before the barrier at the end of the step before
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN / 4; ++j) {
            float4 v;
            pair_split(acc[i][2 * j], v.x, v.y);
            pair_split(acc[i][2 * j + 1], v.z, v.w);
            *reinterpret_cast<float4*>(smem + (tm * TM + i) * Cfg::BN + tn * 4 + 32 * j) = v;
        }
    add_slices<Cfg::THREADS>(a, smem, Cfg::BM * Cfg::BN, [&](int e, int& m, int& n) { m = m0 + e / Cfg::BN; n = n0 + e % Cfg::BN; });
}

// ---- launches
static int launch_clustered(void (*kernel)(F32Args), long long tiles, int threads, int smem, cudaStream_t stream, const F32Args& a, unsigned long long* done) {
    if (tiles * a.slices > 0x7fffffffLL) return VCB_ERR_UNSUPPORTED;
    if (int e = vcb_allow_dynamic_smem(kernel, smem, done)) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(tiles * a.slices));
    cfg.blockDim = threads;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = a.slices;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = vcb_pdl_enabled ? 2 : 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, a);
    return e != cudaSuccess ? (int)e : vcb_last_error();
}

template <int MT, int TN, int NT, int BK>
static int launch_rows(const F32Args& a, bool vec, cudaStream_t stream) {
    static unsigned long long done[2];
    using Cfg = RowsCfg<MT, TN, NT, BK>;
    const long long tiles = (((long long)a.N + Cfg::BN - 1) / Cfg::BN) * ((a.M + MT - 1) / MT);
    return vec ? launch_clustered(gemm_f32_rows_kernel<MT, TN, NT, BK, true>, tiles, NT, Cfg::SMEM, stream, a, &done[0])
               : launch_clustered(gemm_f32_rows_kernel<MT, TN, NT, BK, false>, tiles, NT, Cfg::SMEM, stream, a, &done[1]);
}

template <int TM>
static int launch_tiles(const F32Args& a, bool vec, cudaStream_t stream) {
    static unsigned long long done[2];
    using Cfg = TileCfg<TM>;
    const long long tiles = (((long long)a.N + Cfg::BN - 1) / Cfg::BN) * (((long long)a.M + Cfg::BM - 1) / Cfg::BM);
    return vec ? launch_clustered(gemm_f32_tiles_kernel<TM, true>, tiles, Cfg::THREADS, Cfg::SMEM, stream, a, &done[0])
               : launch_clustered(gemm_f32_tiles_kernel<TM, false>, tiles, Cfg::THREADS, Cfg::SMEM, stream, a, &done[1]);
}

}  // namespace

VCB_EXPORT int vcb_gemm_f32(const float* A, const float* W, float* C, int M, int N, int K,
                            int lda, int ldw, int ldc, void* stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0 || lda < K || ldw < K || ldc < N) return VCB_ERR_BAD_ARG;
    const cudaStream_t s = (cudaStream_t)stream;
    const bool vec = ((((uintptr_t)A) | ((uintptr_t)W)) & 15) == 0 && ((lda | ldw | K) & 3) == 0;
    const F32Args a{A, W, C, M, N, K, lda, ldw, ldc, f32_slices(N, K)};
    // Measured at [37,888 x 3,584] and [3,584 x 18,944], us: 3 rows 104 / 67 in groups of 4 on 64 threads (118 / 84 on 128); 8 rows
    // 124 / 86 in groups of 8 on 64 threads (125 / 112 with two columns a thread on 128); 16 rows 208 / 161 in one group, 230 / 123 in two
    // of 8 with two columns a thread.  Small products of any M go there too: they wait for a few round trips to memory, and the ring of
    // copies has them all in flight.
    if (M <= 2) return launch_rows<2, 1, 64, 32>(a, vec, s);
    if (M <= 4) return launch_rows<4, 1, 64, 32>(a, vec, s);
    if (M <= 8 || (long long)M * N * K < (1 << 24)) return launch_rows<8, 1, 64, 32>(a, vec, s);
    if (M <= 16) return N >= 16384 ? launch_rows<16, 1, 128, 32>(a, vec, s) : launch_rows<8, 2, 128, 32>(a, vec, s);
    // Relative time of the product in tiles of 128, 64 and 32 rows: where they fill the device, tiles times what one takes of it (the smaller
    // ones are bound by their shared-memory reads), and at least what one takes alone on its SM: 1,000 rows of [256 x 96] are 16
    // tiles of 128 rows and 15.7 us, 64 of 32 rows and 8.6; 100 rows of [2,048 x 255] 32.2 and 20.3.  (A tile an SM is where the two meet, taken a
    // little earlier: 700 rows of [4,096 x 129], 192 tiles of 128 rows 34.9 us, 704 of 32 rows 43.3.)
    const double wide = (double)((N + 127LL) / 128) * a.slices * 1.4 / vcb_sm_count();
    const auto time = [&](int rows, double full, double alone) { const double t = full * wide * ((M + rows - 1LL) / rows); return t > alone ? t : alone; };
    const double t128 = time(128, 1.0, 1.0), t64 = time(64, 0.625, 0.69), t32 = time(32, 0.5625, 0.63);
    if (t128 <= t64 && t128 <= t32) return launch_tiles<8>(a, vec, s);
    return t64 <= t32 ? launch_tiles<4>(a, vec, s) : launch_tiles<2>(a, vec, s);
}
