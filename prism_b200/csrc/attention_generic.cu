// Paged causal grouped-query attention, shape-generic version: any head size
// up to 256, any page size, any number of heads and groups, float32 or bf16
// storage, optional sliding window.  It is the attention of the float32 path
// and the fallback of the bf16 path for shapes the tensor-core kernels refuse.
//
// For query token t of request seg at absolute position p, head h:
//     s_j = (q . k_j) * scale          for keys  max(0, p - window + 1) <= j <= p
//     o   = softmax(s) @ v             q-head h reads kv-head h / (nh / nkv)
// i.e. flash_attn_with_kvcache(causal=True) over the request's pages
// (andre-fu/prism engine/executor.py:119-120), with scores, running max and
// sum and the output accumulation in float32.  Keys are visited in blocks of
// 32 starting at the window's first key, so the order of additions for a
// position depends only on that position, not on how the request was cut
// into steps or on what else is in the batch.
//
// A CTA takes a token and HPW query heads of one kv head; block b of the position's keys belongs to warp b % W.
// A lane scores one key of the block (for every head of the CTA, from one read of the key), the block's
// probabilities are exchanged by shuffles, and a lane accumulates the output entries lane, lane + 32, ...; the W
// warps' sums meet in shared memory in their order.  W is a constant of the layer (its value and key sizes and its heads per kv
// head), never of the batch, so within a layer the order of additions stays a matter of the position alone; HPW changes no sum.
//
// Bound by latency (a step of few tokens: one chain of page lookup, key rows, softmax, value rows per block) or by the
// reads of keys and values through the caches (prompts).  Hence blocks side by side, eight rows of loads in flight
// and one read of keys and values for several heads.  14 heads over 2 of 64, float32, against one warp per head and
// token: 3 tokens behind 100 keys 38 -> 7.2 us, 16 behind 400 139 -> 16 us, a prompt of 512 304 -> 93 us; 32 heads of 128 of their
// own, bf16, the same prompt 682 -> 466 us.
#include "common.cuh"

namespace prism {

// 16 bytes of a key row as floats
template <typename T> struct Piece;
template <> struct Piece<float> {
    static constexpr int N = 4;
    static __device__ __forceinline__ void load(const float* __restrict__ p, float (&v)[N]) {
        const float4 x = *reinterpret_cast<const float4*>(p);
        v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w;
    }
};
template <> struct Piece<__nv_bfloat16> {
    static constexpr int N = 8;
    static __device__ __forceinline__ void load(const __nv_bfloat16* __restrict__ p, float (&v)[N]) {
        const uint4 raw = *reinterpret_cast<const uint4*>(p);
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 f = __bfloat1622float2(h[i]);
            v[2 * i] = f.x, v[2 * i + 1] = f.y;
        }
    }
};

// Which keys the token at position p sees.  All three are causal (keys <= p):
//   MASK_CAUSAL  every key from 0;
//   MASK_WINDOW  the last `size` keys, p - size < key;
//   MASK_CHUNK   the keys of p's own block of `size` positions, blocks counted from position 0.
__host__ __device__ __forceinline__ int mask_first_key(int kind, int size, int pos) {
    if (kind == PRISM_MASK_WINDOW && size > 0) return pos - size + 1 > 0 ? pos - size + 1 : 0;
    if (kind == PRISM_MASK_CHUNK && size > 0) return pos / size * size;
    return 0;
}

// MAXD: output dims per lane, value size <= 32 * MAXD.  Keys of `dk` and values of `dv` entries per head may
// differ in size and live in planes with strides of their own (elements between tokens' rows and between
// heads), so that the values may also be a slice of the key rows.  `sink` (per query head, or null): one more
// term exp(sink_h) in the softmax's denominator, with no value; it is not multiplied by `scale`.
// `dist_bias` (float32 [nh, dist_max + 1], or null): a bias by distance, added to the scaled score of the key
// n = pos - j positions back: dist_bias[h][min(n, dist_max)] (distances beyond the table's end share its last entry).
template <typename T, int MAXD, int HPW, int W>
__global__ void __launch_bounds__(W * 32)
attn_generic_kernel(const T* q, int q_stride, int q_head_stride, T* out,
                    int out_stride, const T* kc, long long k_row_stride, int k_head_stride,
                    const T* vc, long long v_row_stride, int v_head_stride,
                    const int* __restrict__ block_table, int bt_width, const int* __restrict__ positions,
                    const int* __restrict__ tok_seg, int nh, int nkv,
                    int dk, int dv, int page_size, int num_pages, int mask_kind, int mask_size,
                    int mask_keep, float scale, const void* __restrict__ sink, int sink_bf16, int* err,
                    const float* __restrict__ dist_bias, int dist_max) {
    pdl_trigger();
    pdl_wait();
    q = pdl_fresh(q), kc = pdl_fresh(kc), vc = pdl_fresh(vc);
    extern __shared__ __align__(16) float smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int group = nh / nkv, per_kv = (group + HPW - 1) / HPW;      // CTAs of a token: nkv * per_kv
    const int t = blockIdx.x / (nkv * per_kv), at = blockIdx.x % (nkv * per_kv);
    const int kvh = at / per_kv, h0 = kvh * group + at % per_kv * HPW;
    const int heads = min(HPW, (kvh + 1) * group - h0);
    const int pos = positions[t];
    const int* bt = block_table + (size_t)tok_seg[t] * bt_width;
    const int lo = mask_first_key(mask_kind, mask_size, pos);
    // the first `mask_keep` positions stay visible behind a window: they are visited first, in blocks of 32 from
    // key 0, then the window's keys from its first key - an order that depends on the position only
    const int keep = mask_keep < lo ? mask_keep : lo;
    const int keep_blocks = (keep + 31) / 32, blocks = keep_blocks + (pos - lo + 32) / 32;

    constexpr int N = Piece<T>::N;
    const int dkp = (dk + N - 1) / N * N;
    float* qs = smem;                                  // [HPW][dkp]
    float* sums = smem + HPW * dkp;                    // [W][HPW][dv + 2]
    for (int d = threadIdx.x; d < HPW * dkp; d += W * 32) {
        const int p = d / dkp, c = d - p * dkp;
        qs[d] = p < heads && c < dk ? to_float(q[(size_t)t * q_stride + (size_t)(h0 + p) * q_head_stride + c]) : 0.f;
    }
    __syncthreads();

    float acc[HPW][MAXD], m[HPW], l[HPW];
#pragma unroll
    for (int p = 0; p < HPW; ++p) {
        m[p] = -INFINITY, l[p] = 0.f;
#pragma unroll
        for (int i = 0; i < MAXD; ++i) acc[p][i] = 0.f;
    }
    const bool vec_ok = dk % N == 0 && k_row_stride % N == 0 && k_head_stride % N == 0 &&
                        (reinterpret_cast<uintptr_t>(kc) % (N * sizeof(T))) == 0;

    for (int b = warp; b < blocks; b += W) {
        const int kb = b < keep_blocks ? b * 32 : lo + (b - keep_blocks) * 32;
        const int j = kb + lane;
        const int last = b < keep_blocks ? keep - 1 : pos;     // the last key of the run this block lies in
        bool valid = j <= last;
        int rowidx = -1;
        if (valid) {
            const int page = bt[j / page_size];
            if (page < 0 || page >= num_pages) {
                report_error(err, PRISM_ERR_PAGE_RANGE);
                valid = false;
            } else {
                rowidx = page * page_size + j % page_size;
            }
        }
        float s[HPW];
#pragma unroll
        for (int p = 0; p < HPW; ++p) s[p] = 0.f;
        if (valid) {
            const T* kr = kc + (size_t)rowidx * k_row_stride + (size_t)kvh * k_head_stride;
            if (vec_ok) {
#pragma unroll 8
                for (int d = 0; d < dk; d += N) {
                    float kv[N];
                    Piece<T>::load(kr + d, kv);
#pragma unroll
                    for (int p = 0; p < HPW; ++p)
#pragma unroll
                        for (int e = 0; e < N; e += 4) {
                            const float4 qv = *reinterpret_cast<const float4*>(qs + p * dkp + d + e);
                            s[p] += kv[e] * qv.x + kv[e + 1] * qv.y + kv[e + 2] * qv.z + kv[e + 3] * qv.w;
                        }
                }
            } else {
                for (int d = 0; d < dk; ++d) {
                    const float kv = to_float(kr[d]);
#pragma unroll
                    for (int p = 0; p < HPW; ++p) s[p] += qs[p * dkp + d] * kv;
                }
            }
        }
        float pr[HPW];
        bool any = false;
#pragma unroll
        for (int p = 0; p < HPW; ++p) {
            float x = valid ? s[p] * scale : -INFINITY;
            if (valid && dist_bias != nullptr && p < heads) x += dist_bias[(size_t)(h0 + p) * (dist_max + 1) + min(pos - j, dist_max)];
            const float m_new = fmaxf(m[p], warp_max(x));
            pr[p] = 0.f;
            if (m_new == -INFINITY) continue;            // only after a page error
            any = true;
            pr[p] = valid ? expf(x - m_new) : 0.f;
            const float corr = expf(m[p] - m_new);
            l[p] = l[p] * corr + warp_sum(pr[p]);
            m[p] = m_new;
#pragma unroll
            for (int i = 0; i < MAXD; ++i) acc[p][i] *= corr;
        }
        if (!any) continue;
        const int cnt = min(32, last - kb + 1);
        constexpr int ROWS = MAXD <= 8 ? 8 : 32 / MAXD;  // value rows on their way together
        for (int j0 = 0; j0 < cnt; j0 += ROWS) {
            float v[ROWS][MAXD];
#pragma unroll
            for (int e = 0; e < ROWS; ++e) {             // lanes beyond cnt hold row -1
                const int rj = __shfl_sync(0xffffffffu, rowidx, j0 + e);
                const T* vr = vc + (size_t)(rj < 0 ? 0 : rj) * v_row_stride + (size_t)kvh * v_head_stride;
#pragma unroll
                for (int i = 0; i < MAXD; ++i) {
                    // always a load, of an entry that exists: a test ahead of it puts the loads one behind the other
                    const float x = to_float(vr[min(lane + 32 * i, dv - 1)]);
                    v[e][i] = rj >= 0 ? x : 0.f;
                }
            }
#pragma unroll
            for (int e = 0; e < ROWS; ++e)
#pragma unroll
                for (int p = 0; p < HPW; ++p) {
                    const float pj = __shfl_sync(0xffffffffu, pr[p], j0 + e);
#pragma unroll
                    for (int i = 0; i < MAXD; ++i) acc[p][i] += pj * v[e][i];
                }
        }
    }
#pragma unroll
    for (int p = 0; p < HPW; ++p) {
        float* mine = sums + (warp * HPW + p) * (dv + 2);
        if (lane == 0) mine[dv] = m[p], mine[dv + 1] = l[p];
#pragma unroll
        for (int i = 0; i < MAXD; ++i)
            if (lane + 32 * i < dv) mine[lane + 32 * i] = acc[p][i];
    }
    __syncthreads();
    const int used = min(W, blocks);                   // the warps that had keys
    for (int x = threadIdx.x; x < heads * dv; x += W * 32) {
        const int p = x / dv, d = x - p * dv;
        float top = sink != nullptr ? load_param(sink, sink_bf16, h0 + p) : -INFINITY;
        for (int w = 0; w < used; ++w) top = fmaxf(top, sums[(w * HPW + p) * (dv + 2) + dv]);
        float o = 0.f, sum = 0.f;
        for (int w = 0; w < used; ++w) {
            const float* part = sums + (w * HPW + p) * (dv + 2);
            const float f = part[dv] == -INFINITY ? 0.f : expf(part[dv] - top);
            o += part[d] * f;
            sum += part[dv + 1] * f;
        }
        if (sink != nullptr) sum += expf(load_param(sink, sink_bf16, h0 + p) - top);
        out[(size_t)t * out_stride + (size_t)(h0 + p) * dv + d] = from_float<T>(sum > 0.f ? o / sum : o * 0.f);      // no key: zero; not a number stays that
    }
}

template <typename T, int MAXD, int HPW, int W>
static int launch_generic(const void* q, int q_stride, int q_head_stride, void* out, int out_stride, const void* kc,
                          long long k_row_stride, int k_head_stride, const void* vc, long long v_row_stride,
                          int v_head_stride, const int* block_table, int bt_width, const int* positions,
                          const int* tok_seg, int T_, int nh, int nkv, int dk, int dv, int page_size, int num_pages,
                          int mask_kind, int mask_size, int mask_keep, float scale, const void* sink, int sink_bf16,
                          int* err, const float* dist_bias, int dist_max, cudaStream_t stream) {
    const int per_kv = (nh / nkv + HPW - 1) / HPW;
    const long long blocks = (long long)T_ * nkv * per_kv;
    if (blocks > 0x7fffffffLL) return (int)cudaErrorInvalidValue;
    const size_t smem = (size_t)HPW * ((dk + 7) / 8 * 8 + W * (dv + 2)) * sizeof(float);
    auto kern = attn_generic_kernel<T, MAXD, HPW, W>;
    open_smem(kern, smem);
    return (int)launch_kernel(kern, dim3((unsigned)blocks), dim3(W * 32), smem, stream,
        (const T*)q, q_stride, q_head_stride, (T*)out, out_stride, (const T*)kc, k_row_stride, k_head_stride,
        (const T*)vc, v_row_stride, v_head_stride, block_table, bt_width, positions, tok_seg, nh, nkv, dk, dv,
        page_size, num_pages, mask_kind, mask_size, mask_keep, scale, sink, sink_bf16, err, dist_bias, dist_max);
}

}  // namespace prism

// Keys of dk and values of dv entries, each plane with its own strides (in elements: between the rows of
// consecutive cache slots, and between kv heads); mask_kind PRISM_MASK_*; mask_keep: under PRISM_MASK_WINDOW
// the first mask_keep positions stay visible to every later query; sink: per-head float32 or bf16
// (sink_dtype) or null; dist_bias: float32 [nh, dist_max + 1] or null.  Returns cudaErrorInvalidValue for dv > 1024 or dk > 8192.
PRISM_EXPORT int prism_attention_masked_generic(const void* q, int q_stride, int q_head_stride, void* out,
                                                int out_stride, const void* kc, long long k_row_stride,
                                                int k_head_stride, const void* vc, long long v_row_stride,
                                                int v_head_stride, int dtype, const int* block_table, int bt_width,
                                                const int* positions, const int* tok_seg, int T, int nh, int nkv,
                                                int dk, int dv, int page_size, int num_pages, int mask_kind,
                                                int mask_size, int mask_keep, float scale, const void* sink,
                                                int sink_dtype, int* err, const float* dist_bias, int dist_max,
                                                cudaStream_t stream) {
    if (T <= 0) return 0;
    if (dist_bias != nullptr && dist_max < 0) return (int)cudaErrorInvalidValue;
    if (mask_keep < 0 || (mask_keep > 0 && mask_kind != PRISM_MASK_WINDOW)) return (int)cudaErrorInvalidValue;
    if (dv > 1024 || dv <= 0 || dk <= 0 || dk > 8192 || nkv <= 0 || nh % nkv != 0) return (int)cudaErrorInvalidValue;
    const int sb = sink_dtype == PRISM_DTYPE_BF16;
    // Several heads of a kv head: eight warps, since their blocks are the decode steps' chain (14 over 2 heads of 64, float32, 16 tokens
    // behind 400 keys: 16 us, four warps 27), and four heads a CTA (a prompt of 512: 94 us, a CTA a head 196), but one where all of them
    // fit the 148 SMs at once and a CTA's four would follow one another (3 tokens behind 100 keys: 7.2 us, four heads 8.7; 16 behind 400
    // have 224: 20 and 16).  A kv head for every head: four warps (8 heads of 128, bf16, prompt of 512: 139 us, 8 warps 147).
    const bool several = nh / nkv >= 2 && dk <= 512, wide = several && (long long)T * nh > 148;
#define PRISM_GENERIC(TT, MD, HP, WW)                                                                               \
    return prism::launch_generic<TT, MD, HP, WW>(q, q_stride, q_head_stride, out, out_stride, kc, k_row_stride,     \
                                                 k_head_stride, vc, v_row_stride, v_head_stride, block_table,       \
                                                 bt_width, positions, tok_seg, T, nh, nkv, dk, dv, page_size,       \
                                                 num_pages, mask_kind, mask_size, mask_keep, scale, sink, sb, err,  \
                                                 dist_bias, dist_max, stream)
#define PRISM_GENERIC_BY_SIZE(TT)                                                                                   \
    do {                                                                                                            \
        if (dv <= 64 && wide) PRISM_GENERIC(TT, 2, 4, 8);                                                           \
        if (dv <= 64 && several) PRISM_GENERIC(TT, 2, 1, 8);                                                        \
        if (dv <= 64) PRISM_GENERIC(TT, 2, 1, 4);                                                                   \
        if (dv <= 128 && wide) PRISM_GENERIC(TT, 4, 4, 8);                                                          \
        if (dv <= 128 && several) PRISM_GENERIC(TT, 4, 1, 8);                                                       \
        if (dv <= 128) PRISM_GENERIC(TT, 4, 1, 4);                                                                  \
        if (dv <= 256) PRISM_GENERIC(TT, 8, 1, 4);                                                                  \
        if (dv <= 512) PRISM_GENERIC(TT, 16, 1, 4);                                                                 \
        PRISM_GENERIC(TT, 32, 1, 4);                                                                                \
    } while (0)
    if (dtype == PRISM_DTYPE_BF16) PRISM_GENERIC_BY_SIZE(__nv_bfloat16);
    PRISM_GENERIC_BY_SIZE(float);
#undef PRISM_GENERIC_BY_SIZE
#undef PRISM_GENERIC
}

// Keys and values of one size hd in planes [slots, nkv, hd]; window <= 0: all keys.  Returns
// cudaErrorInvalidValue for head_dim > 256.
PRISM_EXPORT int prism_attention_generic(const void* q, int q_stride, void* out, int out_stride,
                                         const void* kc, const void* vc, int dtype,
                                         const int* block_table, int bt_width,
                                         const int* positions, const int* tok_seg, int T, int nh,
                                         int nkv, int hd, int page_size, int num_pages, int window,
                                         float scale, int* err, cudaStream_t stream) {
    if (hd > 256) return (int)cudaErrorInvalidValue;
    return prism_attention_masked_generic(q, q_stride, hd, out, out_stride, kc, (long long)nkv * hd, hd, vc,
                                          (long long)nkv * hd, hd, dtype, block_table, bt_width, positions, tok_seg,
                                          T, nh, nkv, hd, hd, page_size, num_pages,
                                          window > 0 ? PRISM_MASK_WINDOW : PRISM_MASK_CAUSAL, window, 0, scale, nullptr, 0,
                                          err, nullptr, 0, stream);
}
