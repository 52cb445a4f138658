// Paged attention over the cache on the FMA pipe, for any head size up to 1024
// and both storage types.  It is the 32-bit path's attention and the reference
// that the tensor-core kernels are compared with.
//
// Two kernels: one warp per (query token, query head), for any row; and one warp per (query token, up to eight heads of a kv head), for
// rows of at most 256 elements that 4-element pieces cover (below).  The query at position p of request r
// attends keys j of the same request with  j <= p  and, when window > 0,
// j > p - window;  key j lives in page block_table[r, j / page], slot j % page, its row in the
// layout of kv_pos (common.cuh).
// Scores, softmax and the output accumulation are float; softmax is computed
// online over chunks of 32 keys (one key per lane; four keys at a time in the other).
//
// Replaces paged_attention_kernel (src/attention/paged_attention.cu:7-93), which
// handles one query token per sequence, has no mask, walks the context twice and
// lets lane 0 accumulate the output alone.  Its "+1e-10" in the denominator is
// not kept: a row always has at least its own key.
#include "common.cuh"

#define ATT_MAX_D 1024
#define ATT_WARPS 4

struct AttnArgs {
    const void* q;              // [n_tokens, nh * d]
    const void* cache;          // [pages][planes][nkv][page][d]; planes 2: keys, then values; planes 1: a row is
                                // key and value at once (attention over cached latent rows)
    void* out;                  // [n_tokens, nh * d]
    const int* positions;
    const int* req_of_token;
    const int* block_table;
    int bt_stride, n_tokens, nh, nkv, d, page, window;
    float scale;
    int num_pages;              // a table entry outside [0, num_pages) is not read through: the key is left
    int* status;                // out and VCB_STATUS_BAD_PAGE is recorded here (may be null)
    int planes;
    const float* sink;          // [nh] or null: a logit per head that joins the softmax's denominator once, unscaled, and has no value
};

template <typename T, int MAXD>
__global__ void attention_simt_kernel(AttnArgs a) {
    extern __shared__ float qs_all[];
    pdl_start();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long item = (long long)blockIdx.x * ATT_WARPS + warp;
    if (item >= (long long)a.n_tokens * a.nh) return;
    const int t = (int)(item / a.nh), h = (int)(item % a.nh);
    const int g = h / (a.nh / a.nkv);                       // src/attention/paged_attention.cu:19
    const int pos = a.positions[t];
    const int* bt = a.block_table + (size_t)a.req_of_token[t] * a.bt_stride;
    float* qs = qs_all + warp * a.d;
    const T* qrow = (const T*)a.q + ((size_t)t * a.nh + h) * a.d;
    for (int i = lane; i < a.d; i += 32) qs[i] = to_f32<T>(qrow[i]) * a.scale;
    __syncwarp();

    const size_t page_elems = (size_t)a.planes * a.nkv * a.page * a.d;
    const size_t v_off = (size_t)(a.planes - 1) * a.nkv * a.page * a.d;
    const T* cache = (const T*)a.cache;

    float o[MAXD / 32];
#pragma unroll
    for (int k = 0; k < MAXD / 32; ++k) o[k] = 0.0f;
    float m = -INFINITY, l = 0.0f;
    const int kstart = a.window > 0 ? max(0, pos - a.window + 1) : 0;

    for (int kb = kstart; kb <= pos; kb += 32) {
        const int j = kb + lane;
        bool valid = j <= pos;
        float s = -INFINITY;
        unsigned long long koff = 0;
        int pg = 0;
        if (valid) {
            const int lp = j / a.page;
            pg = lp < a.bt_stride ? bt[lp] : -1;
            if ((unsigned)pg >= (unsigned)a.num_pages) {
                if (a.status) atomicCAS(a.status, 0, VCB_STATUS_BAD_PAGE);
                valid = false;
            }
        }
        if (valid) {
            koff = (unsigned long long)pg * page_elems + (size_t)g * a.page * a.d;      // the head's block of the page
            const T* kr = cache + koff;
            const int slot = j % a.page;
            float acc = 0.0f;
            for (int i = 0; i < a.d; ++i) acc += qs[i] * to_f32<T>(kr[kv_pos(i, slot, a.d, a.page, (int)sizeof(T))]);
            s = acc;
        }
        const float m_new = fmaxf(m, warp_max(s));
        const float corr = expf(m - m_new);
        const float p = valid ? expf(s - m_new) : 0.0f;
        l = l * corr + warp_sum(p);
#pragma unroll
        for (int k = 0; k < MAXD / 32; ++k) o[k] *= corr;
        const int nvalid = min(32, pos - kb + 1);
        for (int jj = 0; jj < nvalid; ++jj) {
            const float pj = __shfl_sync(0xffffffffu, p, jj);
            const unsigned long long off = __shfl_sync(0xffffffffu, koff, jj);
            const T* vr = cache + off + v_off;
            const int slot = (kb + jj) % a.page;
#pragma unroll
            for (int k = 0; k < MAXD / 32; ++k) {
                const int dim = lane + 32 * k;
                if (dim < a.d) o[k] += pj * to_f32<T>(vr[kv_pos(dim, slot, a.d, a.page, (int)sizeof(T))]);
            }
        }
        m = m_new;
    }
    T* orow = (T*)a.out + ((size_t)t * a.nh + h) * a.d;
    float inv = 1.0f / l;
    if (a.sink) {
        // the reference of the exponents moves if the sink is the largest
        const float sk = a.sink[h], mf = fmaxf(m, sk), keep = expf(m - mf);
        inv = keep / (l * keep + expf(sk - mf));
    }
#pragma unroll
    for (int k = 0; k < MAXD / 32; ++k) {
        const int dim = lane + 32 * k;
        if (dim < a.d) orow[dim] = from_f32<T>(o[k] * inv);
    }
}

// The same for rows of at most 256 elements, a multiple of 4: a warp owns up to GH heads of one kv head's group for one token and
// walks four keys at a time, so that a key's row is read once for all of them, 16 bytes a lane.  LPR lanes hold a row (CH
// 16-byte pieces each; 32 / LPR rows are read side by side).  The products of a lane's piece with GH queries and four keys are
// summed over the row's lanes by halving: each exchange adds two lanes' values and leaves each lane half of them, 31
// exchanges for 32 sums where a butterfly per sum takes 160.  A token's keys are walked in parts, one per ATT_PART_KEYS keys up to eight, every
// part with a softmax of its own; the parts are joined in their order.  Where there are too few tokens to fill the device `split` warps
// take parts side by side, else one warp walks them one after another: the sums are the same, so a token's bits do not depend on the batch.
// The kernel above reads 32 rows 4 bytes at a time, a sector each, once per head: at 28 heads on 4 kv heads of 128, float32, it took
// 1,404 us for one token after 2,048, 125 us for three after 170, 12.2 ms for a prompt of 2,048; this one takes 88, 16 and 2.7.  Bound by
// the latency of a round (a row's loads, five exchanges, two exponentials): a CTA of 8 warps is all that 200 registers a thread allow.
#define ATT_ROW_WARPS 8
#define ATT_PART_KEYS 32            // with 64: 113, 25 and, the reads not running ahead across parts, 3.5

template <typename T> struct RowPiece;
template <> struct RowPiece<float> {
    static __device__ __forceinline__ float4 load(const float* p) { return *reinterpret_cast<const float4*>(p); }
    static __device__ __forceinline__ void store(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
};
template <> struct RowPiece<__nv_bfloat16> {
    static __device__ __forceinline__ float4 load(const __nv_bfloat16* p) {
        const uint2 v = *reinterpret_cast<const uint2*>(p);
        const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.x)), b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.y));
        return make_float4(a.x, a.y, b.x, b.y);
    }
    static __device__ __forceinline__ void store(__nv_bfloat16* p, float4 v) {
        const __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
        *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
    }
};

// s[0 .. N) summed over the lanes whose numbers differ in the bits from BIT down: while a lane holds several sums an exchange halves
// them (lanes with the bit set keep the upper ones), afterwards it adds.  Ends in s[0].
template <int N, int BIT>
__device__ __forceinline__ void sum_over_lanes(float* s, int lane) {
    if constexpr (BIT >= 1) {
        if constexpr (N > 1) {
            const bool upper = (lane & BIT) != 0;
#pragma unroll
            for (int i = 0; i < N / 2; ++i) {
                const float keep = upper ? s[i + N / 2] : s[i], give = upper ? s[i] : s[i + N / 2];
                s[i] = keep + __shfl_xor_sync(0xffffffffu, give, BIT);
            }
            sum_over_lanes<N / 2, BIT / 2>(s, lane);
        } else {
            s[0] += __shfl_xor_sync(0xffffffffu, s[0], BIT);
            sum_over_lanes<1, BIT / 2>(s, lane);
        }
    }
}

// What a part's sums and those before it are multiplied by when both are taken to the larger of their maxima (one of them is finite, or both
// sums are zeros).
__device__ __forceinline__ float part_factor(float m, float m_new) { return m > -INFINITY ? expf(m - m_new) : 0.0f; }
__device__ __forceinline__ float part_join(float before, float f, float part, float g) { return fmaf(part, g, __fmul_rn(before, f)); }

template <typename T, int LPR, int CH, int GH>
__global__ void __launch_bounds__(ATT_ROW_WARPS * 32)
attention_rows_kernel(AttnArgs a, int split) {
    constexpr int GROUPS = 32 / LPR, KPG = 4 / GROUPS;     // row groups of a warp; keys of the four that a group reads
    constexpr int NV = GH * KPG, REP = LPR / NV;           // sums per lane before the halving; lanes that end with the same sum
    static_assert(NV <= LPR && GROUPS * KPG == 4, "a lane ends with one sum");
    __shared__ float p_all[ATT_ROW_WARPS][4 * GH];
    __shared__ float join_o[ATT_ROW_WARPS][GH][CH * LPR * 4];
    __shared__ float join_ml[ATT_ROW_WARPS][2][GH];
    pdl_start();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rg = lane / LPR, rl = lane % LPR;
    const int group = a.nh / a.nkv, chunks = (group + GH - 1) / GH;
    const long long items = (long long)a.n_tokens * a.nkv * chunks;
    const int sub = warp % split;
    const long long item = (long long)blockIdx.x * (ATT_ROW_WARPS / split) + warp / split;      // neighbours: tokens of the same kv head
    const bool live = item < items;
    const int t = live ? (int)(item % a.n_tokens) : 0, gc = live ? (int)(item / a.n_tokens) : 0, g = gc / chunks, h0 = (gc % chunks) * GH;
    const int heads = min(GH, group - h0);                 // of this warp; the sums beyond them are zero and not stored
    const int pos = live ? a.positions[t] : -1;
    const int* bt = a.block_table + (live ? (size_t)a.req_of_token[t] * a.bt_stride : 0);

    const size_t page_elems = (size_t)a.planes * a.nkv * a.page * a.d, v_off = (size_t)(a.planes - 1) * a.nkv * a.page * a.d;
    const T* cache = (const T*)a.cache + (size_t)g * a.page * a.d;
    const bool swizzled = ((a.d * (int)sizeof(T)) & 127) == 0;
    constexpr int PER_PLANE = 128 / (int)sizeof(T), PER_CHUNK = 16 / (int)sizeof(T);
    bool has[CH];
    int base[CH], chunk[CH], within[CH];                   // of this lane's pieces: see kv_pos
#pragma unroll
    for (int c = 0; c < CH; ++c) {
        const int e = (c * LPR + rl) * 4, w = e % PER_PLANE;
        has[c] = e < a.d;
        base[c] = swizzled ? e / PER_PLANE * (a.page * PER_PLANE) : e;
        chunk[c] = w / PER_CHUNK;
        within[c] = w % PER_CHUNK;
    }
    auto at = [&](int c, int slot) {
        return swizzled ? base[c] + slot * PER_PLANE + ((chunk[c] ^ (slot & 7)) * PER_CHUNK) + within[c] : base[c] + slot * a.d;
    };

    float4 q[GH][CH], o[GH][CH];                           // o: of one part, at the end of the row
#pragma unroll
    for (int h = 0; h < GH; ++h)
#pragma unroll
        for (int c = 0; c < CH; ++c) {
            float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (live && h < heads && has[c]) v = RowPiece<T>::load((const T*)a.q + ((size_t)t * a.nh + g * group + h0 + h) * a.d + (c * LPR + rl) * 4);
            q[h][c] = make_float4(v.x * a.scale, v.y * a.scale, v.z * a.scale, v.w * a.scale);
        }
    // the (head, key) whose score this lane ends with
    const int mine = rl / REP, my_head = mine / KPG, my_key = rg * KPG + mine % KPG;
    float m, l;                                            // of my_head, over the part's keys of all lanes
    const int kstart = a.window > 0 ? max(0, pos - a.window + 1) : 0;
    const int parts = max(1, min(ATT_ROW_WARPS, (pos - kstart + ATT_PART_KEYS) / ATT_PART_KEYS));
    const int stride = 4 * parts, steps = (pos - kstart + stride) / stride;      // of four keys, per part; the last ones of a part may be past pos
    const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);

    // Rows are read a round ahead of their use, pages' numbers two: a round waits for neither (unpipelined it took 3,500 cycles).
    auto find = [&](int kb, int& page_of, int& slot_of) {
        const int j = kb + (lane & 3);
        page_of = -1;
        slot_of = 0;
        if (j > pos) return;
        const int lp = j / a.page;
        slot_of = j - lp * a.page;
        page_of = lp < a.bt_stride ? bt[lp] : -1;
        if ((unsigned)page_of >= (unsigned)a.num_pages) {
            if (a.status) atomicCAS(a.status, 0, VCB_STATUS_BAD_PAGE);
            page_of = -1;
        }
    };
    auto fetch = [&](int page_of, int slot_of, float4 (&k)[KPG][CH], float4 (&v)[KPG][CH]) {
#pragma unroll
        for (int kk = 0; kk < KPG; ++kk) {
            const int pg = __shfl_sync(0xffffffffu, page_of, rg * KPG + kk), slot = __shfl_sync(0xffffffffu, slot_of, rg * KPG + kk);
            const T* row = cache + (size_t)max(pg, 0) * page_elems;
#pragma unroll
            for (int c = 0; c < CH; ++c) {
                const bool ok = pg >= 0 && has[c];
                const int off = at(c, slot);
                k[kk][c] = ok ? RowPiece<T>::load(row + off) : zero;
                v[kk][c] = ok ? RowPiece<T>::load(row + v_off + off) : zero;
            }
        }
    };
    // part round + sub of every round; joined in their order by the group's first warp, whose slot of shared memory keeps the sums between rounds
    auto group_barrier = [&]() {
        if (split == 1) __syncwarp();
        else asm volatile("bar.sync %0, %1;" ::"r"(1 + warp / split), "r"(32 * split) : "memory");
    };
    auto leave = [&]() {
        if (rg == 0) {
#pragma unroll
            for (int h = 0; h < GH; ++h)
#pragma unroll
                for (int c = 0; c < CH; ++c) *reinterpret_cast<float4*>(&join_o[warp][h][(c * LPR + rl) * 4]) = o[h][c];
            if (mine % KPG == 0 && rl % REP == 0) { join_ml[warp][0][my_head] = m; join_ml[warp][1][my_head] = l; }
        }
    };
    auto join = [&](int w, bool first_is_slot) {           // the sums before and a part: slot w and the registers, or the other way round
        const float ms = join_ml[w][0][my_head], ls = join_ml[w][1][my_head], mj = fmaxf(m, ms);
        const float fs = part_factor(ms, mj), fr = part_factor(m, mj);
        l = first_is_slot ? part_join(ls, fs, l, fr) : part_join(l, fr, ls, fs);
        m = mj;
#pragma unroll
        for (int h = 0; h < GH; ++h) {
            const float hs = __shfl_sync(0xffffffffu, fs, h * KPG * REP), hr = __shfl_sync(0xffffffffu, fr, h * KPG * REP);
#pragma unroll
            for (int c = 0; c < CH; ++c) {
                const float4 x = *reinterpret_cast<const float4*>(&join_o[w][h][(c * LPR + rl) * 4]);
                if (first_is_slot)
                    o[h][c] = make_float4(part_join(x.x, hs, o[h][c].x, hr), part_join(x.y, hs, o[h][c].y, hr), part_join(x.z, hs, o[h][c].z, hr),
                                          part_join(x.w, hs, o[h][c].w, hr));
                else
                    o[h][c] = make_float4(part_join(o[h][c].x, hr, x.x, hs), part_join(o[h][c].y, hr, x.y, hs), part_join(o[h][c].z, hr, x.z, hs),
                                          part_join(o[h][c].w, hr, x.w, hs));
            }
        }
    };
    // what is found next: four keys of a part, then the next part of this warp, so that the reads run ahead across parts
    int find_part = sub, find_step = 0;
    auto find_next = [&](int& page_of, int& slot_of) {
        find(find_part < parts ? kstart + 4 * find_part + find_step * stride : pos + 1, page_of, slot_of);
        if (++find_step == steps) {
            find_step = 0;
            find_part += split;
        }
    };
    int page_now, slot_now, page_next, slot_next;
    float4 k[KPG][CH], v[KPG][CH], k_next[KPG][CH], v_next[KPG][CH];
    find_next(page_now, slot_now);
    find_next(page_next, slot_next);
    fetch(page_now, slot_now, k, v);
    for (int round = 0; round < parts; round += split) {
        m = -INFINITY;
        l = 0.0f;
#pragma unroll
        for (int h = 0; h < GH; ++h)
#pragma unroll
            for (int c = 0; c < CH; ++c) o[h][c] = zero;
        for (int step = round + sub < parts ? 0 : steps; step < steps; ++step) {
            const int page_of = page_now;
            fetch(page_next, slot_next, k_next, v_next);
            page_now = page_next;
            find_next(page_next, slot_next);
            float s[NV];
#pragma unroll
            for (int h = 0; h < GH; ++h)
#pragma unroll
                for (int kk = 0; kk < KPG; ++kk) {
                    float x = 0.0f;
#pragma unroll
                    for (int c = 0; c < CH; ++c) {
                        x = fmaf(q[h][c].x, k[kk][c].x, x);
                        x = fmaf(q[h][c].y, k[kk][c].y, x);
                        x = fmaf(q[h][c].z, k[kk][c].z, x);
                        x = fmaf(q[h][c].w, k[kk][c].w, x);
                    }
                    s[h * KPG + kk] = x;
                }
            sum_over_lanes<NV, LPR / 2>(s, rl);                // lane rl ends with sum rl / REP
            const bool valid = __shfl_sync(0xffffffffu, page_of, my_key) >= 0;
            const float score = valid ? s[0] : -INFINITY;
            // over the four keys: those of a row group differ in the lane's bits above REP, the groups in the bits above LPR
            float top = score;
#pragma unroll
            for (int bit = REP; bit < REP * KPG; bit <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, bit));
#pragma unroll
            for (int bit = LPR; bit < 32; bit <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, bit));
            const float m_new = fmaxf(m, top);
            const float p = valid ? expf(score - m_new) : 0.0f;
            float sum = p;
#pragma unroll
            for (int bit = REP; bit < REP * KPG; bit <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, bit);
#pragma unroll
            for (int bit = LPR; bit < 32; bit <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, bit);
            const bool moved = m_new > m;
            if (__any_sync(0xffffffffu, moved)) {
                const float corr = moved ? expf(m - m_new) : 1.0f;
                l *= corr;
#pragma unroll
                for (int h = 0; h < GH; ++h) {
                    const float f = __shfl_sync(0xffffffffu, corr, h * KPG * REP);
#pragma unroll
                    for (int c = 0; c < CH; ++c) { o[h][c].x *= f; o[h][c].y *= f; o[h][c].z *= f; o[h][c].w *= f; }
                }
                m = m_new;
            }
            l += sum;
            __syncwarp();
            if (rl % REP == 0) p_all[warp][rg * NV + mine] = p;
            __syncwarp();
#pragma unroll
            for (int h = 0; h < GH; ++h)
#pragma unroll
                for (int kk = 0; kk < KPG; ++kk) {
                    const float w = p_all[warp][rg * NV + h * KPG + kk];
#pragma unroll
                    for (int c = 0; c < CH; ++c) {
                        o[h][c].x = fmaf(w, v[kk][c].x, o[h][c].x);
                        o[h][c].y = fmaf(w, v[kk][c].y, o[h][c].y);
                        o[h][c].z = fmaf(w, v[kk][c].z, o[h][c].z);
                        o[h][c].w = fmaf(w, v[kk][c].w, o[h][c].w);
                    }
                }
#pragma unroll
            for (int kk = 0; kk < KPG; ++kk)
#pragma unroll
                for (int c = 0; c < CH; ++c) { k[kk][c] = k_next[kk][c]; v[kk][c] = v_next[kk][c]; }
        }
        // the row groups' sums (they share the maxima)
#pragma unroll
        for (int bit = LPR; bit < 32; bit <<= 1)
#pragma unroll
            for (int h = 0; h < GH; ++h)
#pragma unroll
                for (int c = 0; c < CH; ++c) {
                    o[h][c].x += __shfl_xor_sync(0xffffffffu, o[h][c].x, bit);
                    o[h][c].y += __shfl_xor_sync(0xffffffffu, o[h][c].y, bit);
                    o[h][c].z += __shfl_xor_sync(0xffffffffu, o[h][c].z, bit);
                    o[h][c].w += __shfl_xor_sync(0xffffffffu, o[h][c].w, bit);
                }
        if (parts == 1) break;
        if (sub > 0) leave();                              // nothing but -inf and zeros where the parts are used up
        group_barrier();
        if (sub == 0) {
            if (round > 0) join(warp, true);
            for (int w = 1; w < split && round + w < parts; ++w) join(warp + w, false);
            __syncwarp();                                  // read before it is written
            if (round + split < parts) leave();
        }
        if (round + split < parts) group_barrier();
    }
    if (sub > 0) return;
    if (!live) return;
    float inv = 1.0f / l;
    if (a.sink) {
        // the reference of the exponents moves if the sink is the largest
        const float sk = my_head < heads ? a.sink[g * group + h0 + my_head] : 0.0f, mf = fmaxf(m, sk), keep = expf(m - mf);
        inv = keep / (l * keep + expf(sk - mf));
    }
#pragma unroll
    for (int h = 0; h < GH; ++h) {
        const float f = __shfl_sync(0xffffffffu, inv, h * KPG * REP);
        if (h >= heads || rg != 0) continue;
#pragma unroll
        for (int c = 0; c < CH; ++c)
            if (has[c])
                RowPiece<T>::store((T*)a.out + ((size_t)t * a.nh + g * group + h0 + h) * a.d + (c * LPR + rl) * 4,
                                   make_float4(o[h][c].x * f, o[h][c].y * f, o[h][c].z * f, o[h][c].w * f));
    }
}

template <typename T, int LPR, int CH, int GH>
static void launch_attention_rows(const AttnArgs& a, cudaStream_t stream) {
    const int group = a.nh / a.nkv;
    const long long items = (long long)a.n_tokens * a.nkv * ((group + GH - 1) / GH);
    // one warp a token where that gives every SM two CTAs and more; fewer tokens share their keys among two to eight warps
    int split = 1;
    while (split < ATT_ROW_WARPS && items * split < 2LL * ATT_ROW_WARPS * vcb_sm_count()) split *= 2;
    const int per = ATT_ROW_WARPS / split;
    vcb_launch(attention_rows_kernel<T, LPR, CH, GH>, (unsigned)((items + per - 1) / per), ATT_ROW_WARPS * 32, 0, stream, a, split);
}

template <typename T>
static void launch_attention_rows(const AttnArgs& a, cudaStream_t stream) {
    const int group = a.nh / a.nkv;
    const bool pairs = group <= 2;                         // heads a key's row is read for
    if (a.d > 64 && a.d <= 96) {
        // Rows of 17 to 24 pieces leave a third of the 32 lanes idle: eight lanes hold three pieces each, four keys are read side by side and a
        // key's product is summed in three exchanges.  One head at a time for one of its own, and in bfloat16 up to three (16 heads of
        // 80, a prompt of 512, us: with two heads on 32 lanes 566, so 302, the kernel above 445; 24 on 8 638, 409 and 596), four for three and
        // four (32 on 8 of 96 637, 458 and 1,134); more heads fill eight on 32 lanes (28 on 4 of 80 334, four of them 455), and two in float32
        // two (407, one 445).
        if (group == 1 || (sizeof(T) == 2 && group <= 3)) return launch_attention_rows<T, 8, 3, 1>(a, stream);
        if (group == 3 || group == 4) return launch_attention_rows<T, 8, 3, 4>(a, stream);
    }
    if (a.d <= 32) pairs ? launch_attention_rows<T, 8, 1, 2>(a, stream) : launch_attention_rows<T, 8, 1, 8>(a, stream);
    else if (a.d <= 64) pairs ? launch_attention_rows<T, 16, 1, 2>(a, stream) : launch_attention_rows<T, 16, 1, 8>(a, stream);
    else if (a.d <= 128) pairs ? launch_attention_rows<T, 32, 1, 2>(a, stream) : launch_attention_rows<T, 32, 1, 8>(a, stream);
    else pairs ? launch_attention_rows<T, 32, 2, 2>(a, stream) : launch_attention_rows<T, 32, 2, 4>(a, stream);
}

VCB_EXPORT int vcb_attention_simt_sink(const void* q, const void* cache, void* out, const int* positions,
                                       const int* req_of_token, const int* block_table, int bt_stride,
                                       int n_tokens, int nh, int nkv, int d, int page, int window,
                                       float scale, int num_pages, int* status, int planes, const float* sink, int dtype, void* stream) {
    if (n_tokens <= 0) return 0;
    if (d <= 0 || d > ATT_MAX_D || nh <= 0 || nkv <= 0 || nh % nkv || page <= 0 || window < 0 || num_pages < 0 ||
        (planes != 1 && planes != 2))
        return VCB_ERR_BAD_ARG;
    AttnArgs a{q, cache, out, positions, req_of_token, block_table, bt_stride, n_tokens, nh, nkv, d,
               page, window, scale, num_pages, status, planes, sink};
    const long long items = (long long)n_tokens * nh;
    const int blocks = (int)((items + ATT_WARPS - 1) / ATT_WARPS);
    const size_t smem = (size_t)ATT_WARPS * d * sizeof(float);
    cudaStream_t s = (cudaStream_t)stream;
    // rows of up to 256 elements that 4-element pieces cover, at addresses these may be read at; a lane of the kernel for the others
    // holds 8 floats of the output row up to 256 elements, 32 up to 1024
    const uintptr_t at = (uintptr_t)q | (uintptr_t)cache | (uintptr_t)out;
    if (d <= 256 && d % 4 == 0 && (at & (dtype == VCB_F32 ? 15 : 7)) == 0 && (dtype == VCB_F32 || dtype == VCB_BF16)) {
        if (dtype == VCB_F32) launch_attention_rows<float>(a, s);
        else launch_attention_rows<__nv_bfloat16>(a, s);
        return vcb_last_error();
    }
    if (dtype == VCB_F32) {
        if (d > 256) vcb_launch(attention_simt_kernel<float, 1024>, blocks, ATT_WARPS * 32, smem, s, a);
        else vcb_launch(attention_simt_kernel<float, 256>, blocks, ATT_WARPS * 32, smem, s, a);
    } else if (dtype == VCB_BF16) {
        if (d > 256) vcb_launch(attention_simt_kernel<__nv_bfloat16, 1024>, blocks, ATT_WARPS * 32, smem, s, a);
        else vcb_launch(attention_simt_kernel<__nv_bfloat16, 256>, blocks, ATT_WARPS * 32, smem, s, a);
    } else return VCB_ERR_BAD_ARG;
    return vcb_last_error();
}

VCB_EXPORT int vcb_attention_simt_planes(const void* q, const void* cache, void* out, const int* positions,
                                  const int* req_of_token, const int* block_table, int bt_stride,
                                  int n_tokens, int nh, int nkv, int d, int page, int window,
                                  float scale, int num_pages, int* status, int planes, int dtype, void* stream) {
    return vcb_attention_simt_sink(q, cache, out, positions, req_of_token, block_table, bt_stride, n_tokens, nh, nkv, d, page, window, scale,
                                   num_pages, status, planes, nullptr, dtype, stream);
}

// Keys and values in planes of their own (planes = 2), the form every cache with separate keys and values has.
VCB_EXPORT int vcb_attention_simt(const void* q, const void* cache, void* out, const int* positions,
                                  const int* req_of_token, const int* block_table, int bt_stride,
                                  int n_tokens, int nh, int nkv, int d, int page, int window,
                                  float scale, int num_pages, int* status, int dtype, void* stream) {
    return vcb_attention_simt_planes(q, cache, out, positions, req_of_token, block_table, bt_stride, n_tokens, nh, nkv, d,
                                     page, window, scale, num_pages, status, 2, dtype, stream);
}
