// Sampling on the device, one CTA or a cluster of eight per logits row, so that only token ids cross
// to the host.  The reference samples on the CPU after copying the whole row
// (src/core/engine.cpp:209-214, src/sampler/sampler.cpp:23-79).
//
// Per row, in the reference's order:
//   1. repetition penalty on the ids generated so far, each once:
//      l > 0 ? l / penalty : l * penalty            (sampler.cpp:81-92)
//   2. temperature <= 0: the largest logit, the lowest id on ties (sampler.cpp:11-21)
//   3. else l *= 1/temperature (sampler.cpp:94-99), softmax (topk_topp.cpp:37-47),
//      optional top-k and top-p in order of falling probability with ties by
//      lower id (topk_topp.cpp:8-35), and an inverse-CDF draw with the given
//      uniform number u: the first kept entry whose running sum exceeds u
//      (topk_topp.cpp:49-56).
// The uniform numbers come from the host (a counter-based generator keyed by the
// request's seed and the index of the token), which the reference does not do: its
// generator is seeded from random_device (sampler.cpp:68).
#include "common.cuh"
#include <cooperative_groups.h>

namespace cg = cooperative_groups;

// A row is read by the CTAs of a cluster, each a contiguous run of ids (a multiple of 128 long).  One SM takes 32 us for the 608 KB of
// 152,064 logits (64 rows at once, greedy); eight SMs take an eighth each, 13 us.  How many is decided by
// the vocabulary alone, so that a row's sums (whose order follows the cut) do not depend on the batch it is in.  Below 16,384
// ids a row is a few round trips to memory for one CTA too, and the cluster's barriers would cost more than they save.
#define SAMPLE_THREADS 512
static inline int sample_ctas(int vocab) { return vocab >= 65536 ? 8 : vocab >= 16384 ? 4 : 1; }
__device__ __forceinline__ int sample_run(int vocab, int ctas) { return ((vocab + ctas - 1) / ctas + 127) & ~127; }

template <typename... KArgs, typename... Args>
static int sample_launch(void (*kernel)(KArgs...), int n_rows, int ctas, cudaStream_t stream, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)n_rows * ctas);
    cfg.blockDim = SAMPLE_THREADS;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ctas;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
    return e != cudaSuccess ? (int)e : vcb_last_error();
}

// ------------------------------------------------------------ penalty
// ids: unique generated ids of all rows, CSR by row_start[n_rows + 1].
__global__ void repetition_penalty_kernel(float* logits, int ld, const int* ids, const int* row_start,
                                          const float* penalty, int vocab) {
    const int row = blockIdx.x;
    const float p = penalty[row];
    if (p == 1.0f) return;
    float* l = logits + (size_t)row * ld;
    for (int i = row_start[row] + threadIdx.x; i < row_start[row + 1]; i += blockDim.x) {
        const int id = ids[i];
        if (id < 0 || id >= vocab) continue;
        const float v = l[id];
        l[id] = v > 0.0f ? v / p : v * p;
    }
}

VCB_EXPORT int vcb_repetition_penalty(float* logits, int ld, const int* ids, const int* row_start,
                                      const float* penalty, int n_rows, int vocab, void* stream) {
    if (n_rows <= 0) return 0;
    repetition_penalty_kernel<<<n_rows, 256, 0, (cudaStream_t)stream>>>(logits, ld, ids, row_start, penalty, vocab);
    return vcb_last_error();
}

// ------------------------------------------------- greedy / temperature
__device__ __forceinline__ void argmax_combine(float& bv, int& bi, float ov, int oi) {
    if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
}

__device__ __forceinline__ void
sample_row(const float* __restrict__ logits, int ld, int vocab, const float* __restrict__ temperature,
           const float* __restrict__ uniform, int* __restrict__ out, int ctas) {
    __shared__ float scratch[33];
    __shared__ float sval[32];
    __shared__ int sidx[32];
    __shared__ int winner;
    __shared__ float cta_max, cta_sum;                     // read by the row's other CTAs
    __shared__ int cta_idx;
    cg::cluster_group cluster = cg::this_cluster();
    const int row = blockIdx.x / ctas, rank = blockIdx.x % ctas;
    const float* l = logits + (size_t)row * ld;
    const float temp = temperature[row];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int run = sample_run(vocab, ctas), first = min(vocab, rank * run), last = min(vocab, first + run);
    const bool aligned = (((uintptr_t)l) & 15) == 0;       // runs and slabs start at multiples of 128

    // The largest logit and its lowest id; the maximum is also softmax's shift.
    float bv = -INFINITY;
    int bi = vocab;
    if (aligned) {
        const int nvec = (last - first) >> 2;
        const float4* l4 = reinterpret_cast<const float4*>(l + first);
        // four loads in flight per thread: one at a time is a round trip to the L2 cache per 16 bytes
        constexpr int U = 4;
        int i = threadIdx.x;
        for (; i + (U - 1) * (int)blockDim.x < nvec; i += U * blockDim.x) {
            float4 v[U];
#pragma unroll
            for (int u = 0; u < U; ++u) v[u] = l4[i + u * blockDim.x];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int id = first + 4 * (i + u * (int)blockDim.x);
                argmax_combine(bv, bi, v[u].x, id); argmax_combine(bv, bi, v[u].y, id + 1);
                argmax_combine(bv, bi, v[u].z, id + 2); argmax_combine(bv, bi, v[u].w, id + 3);
            }
        }
        for (; i < nvec; i += blockDim.x) {
            const float4 v = l4[i];
            const int id = first + 4 * i;
            argmax_combine(bv, bi, v.x, id); argmax_combine(bv, bi, v.y, id + 1);
            argmax_combine(bv, bi, v.z, id + 2); argmax_combine(bv, bi, v.w, id + 3);
        }
        for (int j = first + (nvec << 2) + threadIdx.x; j < last; j += blockDim.x) argmax_combine(bv, bi, l[j], j);
    } else {
        for (int i = first + threadIdx.x; i < last; i += blockDim.x) argmax_combine(bv, bi, l[i], i);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        argmax_combine(bv, bi, ov, oi);
    }
    if (lane == 0) { sval[warp] = bv; sidx[warp] = bi; }
    __syncthreads();
    if (warp == 0) {
        bv = lane < nwarps ? sval[lane] : -INFINITY;
        bi = lane < nwarps ? sidx[lane] : vocab;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            argmax_combine(bv, bi, ov, oi);
        }
        if (lane == 0) { cta_max = bv; cta_idx = bi; }
    }
    cluster.sync();
    float lmax = -INFINITY;
    int imax = vocab;
    for (int c = 0; c < ctas; ++c) argmax_combine(lmax, imax, *cluster.map_shared_rank(&cta_max, c), *cluster.map_shared_rank(&cta_idx, c));
    if (imax >= vocab) imax = 0;
    if (temp <= 0.0f) {                                    // the whole cluster: a row has one temperature
        if (rank == 0 && threadIdx.x == 0) out[row] = imax;
        cluster.sync();                                    // nobody leaves while its maximum is being read
        return;
    }

    // e_i = exp((l_i - max) / T).  Every warp owns a contiguous slab of ids, so the warps' sums, taken in the
    // order of the warps, follow the order of the ids; inside its slab a warp reads rows of 128 ids (a float4
    // a lane, four rows in flight), each lane adding up what it reads.  The slab that holds the draw is then
    // walked once more by its warp, row by row in the order of the ids.
    const float inv_t = 1.0f / temp;
    const float xmax = temp != 1.0f ? lmax * inv_t : lmax;
    const bool scaled = temp != 1.0f;
    auto weight = [&](float v) { return expf((scaled ? v * inv_t : v) - xmax); };
    const int slab = ((run + nwarps - 1) / nwarps + 127) & ~127;
    const int lo = min(last, first + warp * slab), hi = min(last, lo + slab);
    // the four weights of this lane in the row that starts at id `base` (zero beyond the slab)
    auto row_weights = [&](int base, float (&e)[4]) {
        const int i = base + lane * 4;
        if (aligned && i + 3 < hi) {
            const float4 v = *reinterpret_cast<const float4*>(l + i);
            e[0] = weight(v.x); e[1] = weight(v.y); e[2] = weight(v.z); e[3] = weight(v.w);
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) e[k] = i + k < hi ? weight(l[i + k]) : 0.0f;
        }
    };
    float local = 0.0f;
    {
        constexpr int U = 4;
        int base = lo;
        if (aligned) {
            for (; base + U * 128 <= hi; base += U * 128) {
                float4 v[U];
#pragma unroll
                for (int u = 0; u < U; ++u) v[u] = *reinterpret_cast<const float4*>(l + base + u * 128 + lane * 4);
#pragma unroll
                for (int u = 0; u < U; ++u) local += (weight(v[u].x) + weight(v[u].y)) + (weight(v[u].z) + weight(v[u].w));
            }
        }
        for (; base < hi; base += 128) {
            float e[4];
            row_weights(base, e);
            local += (e[0] + e[1]) + (e[2] + e[3]);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) local += __shfl_xor_sync(0xffffffffu, local, o);      // the slab's sum, in all lanes
    if (lane == 0) scratch[warp] = local;
    __syncthreads();
    if (warp == 0) {
        float w = lane < nwarps ? scratch[lane] : 0.0f;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        scratch[lane] = w;                 // inclusive sums of the slabs
        // The run's sum is that of its last slab with ids: an empty slab behind it adds nothing, but its sum is another tree of the same
        // numbers and may be a unit in the last place larger, and a draw between the two would lie in no slab.
        if (lane == (last > first ? (last - first - 1) / slab : 0)) cta_sum = w;
    }
    if (threadIdx.x == 0) winner = nwarps;
    cluster.sync();
    float before_cta = 0.0f, total = 0.0f;                 // the runs before this one; all
    for (int c = 0; c < ctas; ++c) {
        if (c == rank) before_cta = total;
        total += *cluster.map_shared_rank(&cta_sum, c);
    }
    cluster.sync();                                        // the other CTAs' sums are read: from here on each is alone
    const float target = uniform[row] * total;
    if (!(target < total)) {                               // u * total >= total after rounding: the last id
        if (rank == 0 && threadIdx.x == 0) out[row] = vocab - 1;
        return;
    }
    // the run that holds the draw: the first whose inclusive sum exceeds it
    if (!(target < before_cta + cta_sum) || (rank > 0 && target < before_cta)) return;
    const float incl = before_cta + scratch[warp];
    if (lane == 0 && hi > lo && target < incl) atomicMin(&winner, warp);
    __syncthreads();
    if (warp != winner) return;                            // there is one: the last slab that has ids ends at the run's sum
    float c = incl - local;                      // the sum before this slab
    int tok = hi - 1;                            // if rounding keeps the walk's sums below the draw: the slab's last id
    for (int base = lo; base < hi; base += 128) {
        float e[4];
        row_weights(base, e);
        const float p1 = e[0], p2 = p1 + e[1], p3 = p2 + e[2], p4 = p3 + e[3];
        float upto = p4;                         // inclusive sum of the lanes' four
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float y = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += y;
        }
        const float before = c + (upto - p4);
        const int i = base + lane * 4;
        int hit = -1;
        if (i < hi) {
            if (target < before + p1) hit = i;
            else if (target < before + p2 && i + 1 < hi) hit = i + 1;
            else if (target < before + p3 && i + 2 < hi) hit = i + 2;
            else if (target < before + p4 && i + 3 < hi) hit = i + 3;
        }
        const unsigned found = __ballot_sync(0xffffffffu, hit >= 0);
        if (found) {
            tok = __shfl_sync(0xffffffffu, hit, __ffs(found) - 1);
            break;
        }
        c += __shfl_sync(0xffffffffu, upto, 31);
    }
    if (lane == 0) out[row] = tok;
}

__global__ void __launch_bounds__(SAMPLE_THREADS)
sample_kernel(const float* __restrict__ logits, int ld, int vocab, const float* __restrict__ temperature,
              const float* __restrict__ uniform, int* __restrict__ out, int ctas) {
    sample_row(logits, ld, vocab, temperature, uniform, out, ctas);
}

VCB_EXPORT int vcb_sample(const float* logits, int ld, int vocab, const float* temperature,
                          const float* uniform, int* out, int n_rows, void* stream) {
    if (n_rows <= 0) return 0;
    if (vocab <= 0 || ld < vocab) return VCB_ERR_BAD_ARG;
    const int ctas = sample_ctas(vocab);
    return sample_launch(sample_kernel, n_rows, ctas, (cudaStream_t)stream, logits, ld, vocab, temperature, uniform, out, ctas);
}

// --------------------------------------------------------- top-k / top-p
// Rows with temperature > 0 and (top_p < 1 or top_k > 0) are drawn here, in order
// of falling probability with ties by lower id, as the reference does after its
// sort (src/sampler/sampler.cpp:52-71, src/sampler/topk_topp.cpp:8-35,49-56).
// Nothing is sorted.  Every id gets the 52-bit key  (bits of e_i) << 20 | (0xFFFFF - i)
// with e_i = exp((l_i - max) / T) >= 0, so a larger key means "earlier in the
// reference's order".  With count(T) and sum(T) taken over the ids whose key is >= T:
//   top-k keeps keys >= T_k, the largest T with count(T) >= k;
//   top-p keeps keys >= T_p, the largest T with sum(T) >= p * sum(T_k);
//   the draw returns the id of the largest T with sum(T) > u * sum(T_p).
// Mostly few ids are kept.  One pass counts all ids by the twelve leading bits of their weights (1,017 bins); the bin that the
// first of the two bounds falls into (for top-p with every id's weight taken at its bin's lower end, so not too high a
// bin) says which ids can be kept at all.  Up to FILT_LIST of them are gathered into the first CTA's shared memory by one more pass,
// sorted there by key, and their running sums, in double, give both bounds and the draw.
//
// Where more are left (flat rows), each threshold is found ten bits at a time, from the top (the first digit has twelve): a pass over the row bins
// the ids that agree with the bits found so far by their next ten bits and takes the largest digit for which the condition
// still holds; it ends when a bin holds a single id, mostly after two.  The first digit's bins (every id's) are made once and serve
// all three searches.  Counts and sums are exact whatever the order of the ids: a bin's weights share their leading bits, so its
// sum is its count times those plus a whole number of units in the last place, kept as two counters of ten bits each (2^20 ids
// fit 32 bits); bins are added up in double.
//
// 64 rows of 152,064 (temperature 0.8, top-k 50 and top-p 0.9): digits of four bits, one CTA a row, 39 passes bound by sixteen comparisons an
// id, 1,549 us; digits of ten bits in clusters 268 us (bound by three shared-memory counters an id and by eight passes); the list 114 us.
// (Flat rows, top-p 0.9 of logits of deviation 2: 374 us by digits.)
// e is kept in scratch memory supplied by the caller: rows * vocab floats.
enum { COND_COUNT_GE = 0, COND_SUM_GE = 1, COND_SUM_GT = 2 };
constexpr int FILT_BINS = 1024, FILT_MINE = FILT_BINS / SAMPLE_THREADS;       // bins of a digit; of a thread

__device__ __forceinline__ unsigned long long filt_key(float e, int id) {
    return ((unsigned long long)__float_as_uint(e) << 20) | (unsigned long long)(0xFFFFF - id);
}

constexpr int FILT_LIST = 4096, FILT_PER = FILT_LIST / SAMPLE_THREADS;

struct FiltShared {
    unsigned long long list[FILT_LIST];                    // the first CTA's: keys
    int listed;
    double cta_total;
    unsigned count[FILT_BINS], low[FILT_BINS], high[FILT_BINS];               // read by the row's other CTAs
    double wsum[32], above_sum, at_sum;
    unsigned wcnt[32], above_cnt, at_cnt;
    int chosen;
    float cta_max;
};

// What the CTAs of a row share; a thread's bins are 1023 - (2 t), 1023 - (2 t + 1): falling weights.
struct FiltRow {
    const float* e;
    int first, last, ctas;
    bool vec;
    FiltShared* sh;

    template <typename F> __device__ __forceinline__ void for_each(F f) const {
        if (vec) {
            const float4* e4 = reinterpret_cast<const float4*>(e + first);
            const int nvec = (last - first) >> 2;
            constexpr int U = 4;
            int i = threadIdx.x;
            for (; i + (U - 1) * SAMPLE_THREADS < nvec; i += U * SAMPLE_THREADS) {
                float4 v[U];
#pragma unroll
                for (int u = 0; u < U; ++u) v[u] = e4[i + u * SAMPLE_THREADS];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int id = first + 4 * (i + u * SAMPLE_THREADS);
                    f(v[u].x, id); f(v[u].y, id + 1); f(v[u].z, id + 2); f(v[u].w, id + 3);
                }
            }
            for (; i < nvec; i += SAMPLE_THREADS) {
                const float4 v = e4[i];
                const int id = first + 4 * i;
                f(v.x, id); f(v.y, id + 1); f(v.z, id + 2); f(v.w, id + 3);
            }
            for (int j = first + (nvec << 2) + threadIdx.x; j < last; j += SAMPLE_THREADS) f(e[j], j);
        } else {
            for (int i = first + threadIdx.x; i < last; i += SAMPLE_THREADS) f(e[i], i);
        }
    }
    __device__ __forceinline__ void clear() const {
        for (int i = threadIdx.x; i < FILT_BINS; i += SAMPLE_THREADS) { sh->count[i] = 0; sh->low[i] = 0; sh->high[i] = 0; }
        __syncthreads();
    }
    __device__ __forceinline__ void add(int bin, unsigned rest) const {       // rest: the key's weight bits below the digit, at most 20
        atomicAdd(&sh->count[bin], 1u);
        if (rest & 1023u) atomicAdd(&sh->low[bin], rest & 1023u);
        if (rest >> 10) atomicAdd(&sh->high[bin], rest >> 10);
    }
    // This thread's bins over all CTAs; ends with the counters free to be cleared.  value(bin): the weight's leading bits.
    template <typename V>
    __device__ __forceinline__ void collect(unsigned (&cnt)[FILT_MINE], double (&sum)[FILT_MINE], V value) const {
        cg::cluster_group cluster = cg::this_cluster();
        cluster.sync();
#pragma unroll
        for (int j = 0; j < FILT_MINE; ++j) {
            const int bin = FILT_BINS - 1 - (threadIdx.x * FILT_MINE + j);
            unsigned c = 0, lo = 0, hi = 0;
            for (int r = 0; r < ctas; ++r) {
                c += *cluster.map_shared_rank(&sh->count[bin], r);
                lo += *cluster.map_shared_rank(&sh->low[bin], r);
                hi += *cluster.map_shared_rank(&sh->high[bin], r);
            }
            const unsigned bits = value(bin);
            const double at = (double)__uint_as_float(bits), unit = (double)__uint_as_float(bits + 1) - at;
            cnt[j] = c;
            sum[j] = c ? (double)c * at + ((double)hi * 1024.0 + (double)lo) * unit : 0.0;
        }
        cluster.sync();
    }
};

// The first of the row's bins (largest weights first) at which the running count or sum, on top of above_*, meets the bound.
// Sets sh.chosen, sh.above_* (before that bin) and sh.at_* (with it).
template <int COND>
__device__ __forceinline__ void filt_choose(FiltShared& sh, const unsigned (&cnt)[FILT_MINE], const double (&sum)[FILT_MINE],
                                            unsigned above_cnt, double above_sum, double bound) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned c = 0;
    double s = 0.0;
#pragma unroll
    for (int j = 0; j < FILT_MINE; ++j) { c += cnt[j]; s += sum[j]; }
    unsigned ci = c;
    double si = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned cy = __shfl_up_sync(0xffffffffu, ci, o);
        const double sy = __shfl_up_sync(0xffffffffu, si, o);
        if (lane >= o) { ci += cy; si += sy; }
    }
    __syncthreads();                                       // what the last call left in sh has been read by all
    if (threadIdx.x == 0) sh.chosen = FILT_BINS;
    if (lane == 31) { sh.wcnt[warp] = ci; sh.wsum[warp] = si; }
    __syncthreads();
    unsigned cb = above_cnt;
    double sb = above_sum;
    for (int w = 0; w < warp; ++w) { cb += sh.wcnt[w]; sb += sh.wsum[w]; }
    cb += ci - c;
    sb += si - s;                                          // exact enough: doubles of at most 2^20 terms
    int hit = FILT_BINS, lowest = -1;
    unsigned hit_cb = 0, hit_c = 0, low_cb = 0, low_c = 0;
    double hit_sb = 0.0, hit_s = 0.0, low_sb = 0.0, low_s = 0.0;
#pragma unroll
    for (int j = 0; j < FILT_MINE; ++j) {
        const unsigned c1 = cb + cnt[j];
        const double s1 = sb + sum[j];
        const bool ok = COND == COND_COUNT_GE ? (double)c1 >= bound : COND == COND_SUM_GE ? s1 >= bound : s1 > bound;
        const int at = threadIdx.x * FILT_MINE + j;
        if (cnt[j]) {
            if (ok && hit == FILT_BINS) { hit = at; hit_cb = cb; hit_c = c1; hit_sb = sb; hit_s = s1; }
            lowest = at; low_cb = cb; low_c = c1; low_sb = sb; low_s = s1;
        }
        cb = c1;
        sb = s1;
    }
    if (hit < FILT_BINS) atomicMin(&sh.chosen, hit);
    __syncthreads();
    int chosen = sh.chosen;
    if (chosen == FILT_BINS) {
        // The bin before was taken because its sum met the bound; added up digit by digit the same ids fall short of it by the
        // last bit of a double.  The bound then lies at the end of this prefix's range: its lowest digit that has any id.
        __syncthreads();
        if (threadIdx.x == 0) sh.chosen = -1;
        __syncthreads();
        if (lowest >= 0) atomicMax(&sh.chosen, lowest);
        __syncthreads();
        chosen = sh.chosen;
        hit = lowest; hit_cb = low_cb; hit_c = low_c; hit_sb = low_sb; hit_s = low_s;
    }
    if (chosen >= 0 && hit == chosen) { sh.above_cnt = hit_cb; sh.at_cnt = hit_c; sh.above_sum = hit_sb; sh.at_sum = hit_s; }
    __syncthreads();
}

// The largest key T for which the condition holds, counting only ids with key >= floor_key; cnt1, sum1: this thread's bins of
// the first digit, of those ids.  On return sh.at_* are count(T) and sum(T), `shift` the bits of T that were not needed.
template <int COND>
__device__ unsigned long long filt_search(const FiltRow& row, const unsigned (&cnt1)[FILT_MINE], const double (&sum1)[FILT_MINE],
                                          unsigned long long floor_key, double bound, int& shift) {
    FiltShared& sh = *row.sh;
    filt_choose<COND>(sh, cnt1, sum1, 0u, 0.0, bound);
    unsigned long long prefix = (unsigned long long)(FILT_BINS - 1 - max(sh.chosen, 0));
    shift = 40;
    while (shift > 0 && sh.at_cnt - sh.above_cnt > 1) {
        const unsigned above_cnt = sh.above_cnt;
        const double above_sum = sh.above_sum;
        shift -= 10;
        const unsigned top = (unsigned)(prefix >> (30 - shift));              // the first digit, of every level
        row.clear();
        row.for_each([&](float e, int id) {
            const unsigned bits = __float_as_uint(e);
            if ((bits >> 20) != top) return;
            const unsigned long long key = filt_key(e, id);
            if ((key >> (shift + 10)) != prefix || key < floor_key) return;
            row.add((int)((key >> shift) & (FILT_BINS - 1)), shift > 20 ? bits & ((1u << (shift - 20)) - 1) : 0u);
        });
        unsigned cnt[FILT_MINE];
        double sum[FILT_MINE];
        const int level = shift;
        row.collect(cnt, sum, [&](int bin) { return (unsigned)((((prefix << 10) | (unsigned)bin) << level) >> 20); });
        filt_choose<COND>(sh, cnt, sum, above_cnt, above_sum, bound);
        prefix = (prefix << 10) | (unsigned long long)(FILT_BINS - 1 - max(sh.chosen, 0));
    }
    return prefix << shift;
}

// The first CTA's part of the list path: n keys in sh.list, no sum before the first; `whole` is the row's sum.
__device__ __forceinline__ int filt_draw(FiltShared& sh, int n, int vocab, int k, float p, float u, double whole) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int size = 2;
    while (size < n) size <<= 1;
    for (int i = n + threadIdx.x; i < size; i += SAMPLE_THREADS) sh.list[i] = 0ull;        // below every key: ids are below 0xFFFFF
    __syncthreads();
    // bitonic, falling
    for (int run = 2; run <= size; run <<= 1)
        for (int step = run >> 1; step > 0; step >>= 1) {
            for (int t = threadIdx.x; t < size / 2; t += SAMPLE_THREADS) {
                const int i = 2 * t - (t & (step - 1)), j = i + step;
                const unsigned long long a = sh.list[i], b = sh.list[j];
                if ((a < b) == ((i & run) == 0)) { sh.list[i] = b; sh.list[j] = a; }
            }
            __syncthreads();
        }
    // running sums of this thread's entries
    const int first = threadIdx.x * FILT_PER;
    double own[FILT_PER], s = 0.0;
#pragma unroll
    for (int j = 0; j < FILT_PER; ++j) {
        if (first + j < n) s += (double)__uint_as_float((unsigned)(sh.list[first + j] >> 20));
        own[j] = s;
    }
    double si = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double y = __shfl_up_sync(0xffffffffu, si, o);
        if (lane >= o) si += y;
    }
    if (lane == 31) sh.wsum[warp] = si;
    if (threadIdx.x == 0) sh.chosen = n;
    __syncthreads();
    double before = si - s;
    for (int w = 0; w < warp; ++w) before += sh.wsum[w];
    // the first entry whose running sum meets the bound (or the last one if rounding keeps all below), and its sum
    auto find = [&](double bound, bool strictly, int most, double& at) {
        int hit = n;
#pragma unroll
        for (int j = FILT_PER - 1; j >= 0; --j) {
            const double c = before + own[j];
            if (first + j < n && (strictly ? c > bound : c >= bound)) hit = first + j;
        }
        if (hit < n) atomicMin(&sh.chosen, hit);
        __syncthreads();
        const int found = min(sh.chosen, most - 1);
        if (found >= first && found < first + FILT_PER) sh.at_sum = before + own[found - first];
        __syncthreads();
        at = sh.at_sum;
        if (threadIdx.x == 0) sh.chosen = n;
        __syncthreads();
        return found;
    };
    int kept = n;
    double sum = whole, unused;
    if (k > 0 && k < vocab) {
        kept = min(k, n);
        if (kept - 1 >= first && kept - 1 < first + FILT_PER) sh.at_sum = before + own[kept - 1 - first];
        __syncthreads();
        sum = sh.at_sum;
        __syncthreads();
    }
    if (p < 1.0f) kept = find((double)p * sum, false, kept, sum) + 1;
    const int at = find((double)u * sum, true, kept, unused);
    return 0xFFFFF - (int)(sh.list[at] & 0xFFFFFull);
}

// ALL: rows without top-k and top-p are drawn too (as sample_kernel draws them).
template <bool ALL>
__global__ void __launch_bounds__(SAMPLE_THREADS)
sample_filtered_kernel(const float* __restrict__ logits, int ld, int vocab, const float* __restrict__ temperature,
                       const float* __restrict__ uniform, const float* __restrict__ top_p,
                       const int* __restrict__ top_k, float* __restrict__ scratch, int* __restrict__ out, int ctas) {
    __shared__ FiltShared sh;
    __shared__ float red[33];
    __shared__ double dred[SAMPLE_THREADS / 32];
    cg::cluster_group cluster = cg::this_cluster();
    const int row = blockIdx.x / ctas, rank = blockIdx.x % ctas;
    const float temp = temperature[row], p = top_p[row];
    const int k = top_k[row];
    if (!(temp > 0.0f) || !(p < 1.0f || k > 0)) {            // the whole cluster
        if (ALL) sample_row(logits, ld, vocab, temperature, uniform, out, ctas);
        return;
    }
    const float* l = logits + (size_t)row * ld;
    float* e = scratch + (size_t)row * vocab;
    const float inv_t = 1.0f / temp;
    const bool scaled = temp != 1.0f;
    const int run = sample_run(vocab, ctas), first = min(vocab, rank * run), last = min(vocab, first + run);

    const bool vec = ((((uintptr_t)l) | ((uintptr_t)e)) & 15) == 0;
    FiltRow logit_row{l, first, last, ctas, vec, &sh}, weight_row{e, first, last, ctas, vec, &sh};
    float mx = -INFINITY;
    logit_row.for_each([&](float v, int) { mx = fmaxf(mx, scaled ? __fmul_rn(v, inv_t) : v); });
    mx = block_max(mx, red);
    if (threadIdx.x == 0) sh.cta_max = mx;
    weight_row.clear();
    cluster.sync();
    for (int c = 0; c < ctas; ++c) mx = fmaxf(mx, *cluster.map_shared_rank(&sh.cta_max, c));
    // (The largest has weight 1 even where the difference of two infinities would be no number; what is no number has no weight.)
    // The product is rounded on its own wherever this is inlined: the ids counted and the ids gathered have the same weights.
    auto weight = [&](float v) {
        const float x = scaled ? __fmul_rn(v, inv_t) : v;
        const float w = x == mx ? 1.0f : expf(x - mx);
        return w <= 1.0f ? w : 0.0f;
    };
    unsigned cnt[FILT_MINE];
    double sum[FILT_MINE];
    double total = 0.0;
    logit_row.for_each([&](float v, int) {
        const float w = weight(v);
        atomicAdd(&sh.count[__float_as_uint(w) >> 20], 1u);
        total += (double)w;                                  // a thread's ids in their order, then threads, warps and CTAs in theirs
    });
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
    if ((threadIdx.x & 31) == 0) dred[threadIdx.x >> 5] = total;
    if (threadIdx.x == 0) sh.listed = 0;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < SAMPLE_THREADS / 32; ++w) t += dred[w];
        sh.cta_total = t;
    }
    weight_row.collect(cnt, sum, [](int bin) { return (unsigned)bin << 20; });      // (sums at the bins' lower ends: low and high are zero)
    // sh.cta_total stands until the clusters' next barrier but one
    total = 0.0;
    for (int c = 0; c < ctas; ++c) total += *cluster.map_shared_rank(&sh.cta_total, c);
    if (k > 0 && k < vocab) filt_choose<COND_COUNT_GE>(sh, cnt, sum, 0u, 0.0, (double)k);
    else filt_choose<COND_SUM_GE>(sh, cnt, sum, 0u, 0.0, (p < 1.0f ? (double)p : 1.0) * total);
    if (sh.at_cnt <= FILT_LIST) {
        const unsigned least = (unsigned)(FILT_BINS - 1 - max(sh.chosen, 0)) << 20;
        int* listed = cluster.map_shared_rank(&sh.listed, 0);
        unsigned long long* list = cluster.map_shared_rank(sh.list, 0);
        logit_row.for_each([&](float v, int id) {
            const float w = weight(v);
            if (__float_as_uint(w) < least) return;
            const int at = atomicAdd(listed, 1);
            if (at < FILT_LIST) list[at] = filt_key(w, id);
        });
        cluster.sync();
        if (rank != 0) return;
        const int id = filt_draw(sh, min(sh.listed, FILT_LIST), vocab, k, p, uniform[row], total);
        if (threadIdx.x == 0) out[row] = id;
        return;
    }

    // A thread writes the weights it reads later: no other thread's are needed.
    weight_row.clear();
    logit_row.for_each([&](float v, int id) {
        const float w = weight(v);
        e[id] = w;
        const unsigned bits = __float_as_uint(w);
        weight_row.add((int)(bits >> 20), bits & 0xFFFFFu);
    });
    weight_row.collect(cnt, sum, [](int bin) { return (unsigned)bin << 20; });

    unsigned long long floor_key = 0;
    int shift;
    // the first digit's bins of the ids with key >= T: those above T's digit whole, T's own what the search found, none below
    auto cut = [&](unsigned long long t) {
        const int digit = (int)(t >> 40);
        const double kept_sum = sh.at_sum;
        const unsigned kept_cnt = sh.at_cnt;
        // above T's digit: a fixed-order sum of whole bins, as filt_choose takes them
        filt_choose<COND_COUNT_GE>(sh, cnt, sum, 0u, 0.0, (double)kept_cnt);
        const unsigned above_cnt = sh.above_cnt;
        const double above_sum = sh.above_sum;
        __syncthreads();
#pragma unroll
        for (int j = 0; j < FILT_MINE; ++j) {
            const int bin = FILT_BINS - 1 - (threadIdx.x * FILT_MINE + j);
            if (bin < digit) { cnt[j] = 0; sum[j] = 0.0; }
            else if (bin == digit) { cnt[j] = kept_cnt - above_cnt; sum[j] = kept_sum - above_sum; }
        }
        if (t > floor_key) floor_key = t;                  // (t's open bits are zero: it may lie below the floor it was found above)
        return kept_sum;
    };
    double kept = 0.0;
    {
        // the row's whole weight: the condition that only the last bin meets
        filt_choose<COND_COUNT_GE>(sh, cnt, sum, 0u, 0.0, (double)vocab);
        kept = sh.at_sum;
    }
    if (k > 0 && k < vocab) kept = cut(filt_search<COND_COUNT_GE>(weight_row, cnt, sum, floor_key, (double)k, shift));
    if (p < 1.0f) kept = cut(filt_search<COND_SUM_GE>(weight_row, cnt, sum, floor_key, (double)p * kept, shift));
    const unsigned long long t = filt_search<COND_SUM_GT>(weight_row, cnt, sum, floor_key, (double)uniform[row] * kept, shift);
    if (shift == 0) {
        if (rank == 0 && threadIdx.x == 0) out[row] = 0xFFFFF - (int)(t & 0xFFFFFull);
    } else {
        // a single id has these leading bits
        weight_row.for_each([&](float w, int id) {
            const unsigned long long key = filt_key(w, id);
            if ((key >> shift) == (t >> shift) && key >= floor_key) out[row] = id;
        });
    }
}

static int sample_filtered_rows(bool all, const float* logits, int ld, int vocab, const float* temperature, const float* uniform, const float* top_p,
                                const int* top_k, float* scratch, int* out, int n_rows, void* stream) {
    if (n_rows <= 0) return 0;
    if (vocab <= 0 || ld < vocab) return VCB_ERR_BAD_ARG;
    if (vocab > (1 << 20)) return VCB_ERR_UNSUPPORTED;      // ids take 20 bits of the key
    const int ctas = sample_ctas(vocab);
    return sample_launch(all ? sample_filtered_kernel<true> : sample_filtered_kernel<false>, n_rows, ctas, (cudaStream_t)stream, logits, ld, vocab,
                         temperature, uniform, top_p, top_k, scratch, out, ctas);
}

VCB_EXPORT int vcb_sample_filtered(const float* logits, int ld, int vocab, const float* temperature,
                                   const float* uniform, const float* top_p, const int* top_k,
                                   float* scratch, int* out, int n_rows, void* stream) {
    return sample_filtered_rows(false, logits, ld, vocab, temperature, uniform, top_p, top_k, scratch, out, n_rows, stream);
}

// Every row in one launch: what vcb_sample and then vcb_sample_filtered leave.
VCB_EXPORT int vcb_sample_all(const float* logits, int ld, int vocab, const float* temperature,
                              const float* uniform, const float* top_p, const int* top_k,
                              float* scratch, int* out, int n_rows, void* stream) {
    return sample_filtered_rows(true, logits, ld, vocab, temperature, uniform, top_p, top_k, scratch, out, n_rows, stream);
}
