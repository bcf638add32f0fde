// Recurrent mixers: layers whose memory of a sequence is a matrix of fixed size per head instead of a cache of
// keys.  The recurrences share one scan kernel; S is [dk, dv] per head, float32, one per request slot:
//
//   delta rule with a scalar decay (SCAN_DELTA), per token with unit-length q, k and g, beta in (0, 1):
//       S <- g S;   u = beta (v - S^T k);   S <- S + k u^T;   o = S^T q          (the read-out sees this token's write)
//   delta rule with one decay per key channel (SCAN_CHANNEL), w a vector over the key channels:
//       S <- diag(w) S;   u = beta (v - S^T k);   S <- S + k u^T;   o = S^T q
//   decayed outer-product sum with a bonus for the current token (SCAN_BONUS), w, u vectors over the key channels:
//       o = (S + diag(u) k v^T)^T r;   S <- diag(w) S + k v^T                    (the read-out sees S before the write)
//   generalized delta rule (SCAN_GENERAL), w, e, c vectors over the key channels (e the unit key, c = a * e a removal
//   rate per channel times it):
//       S <- diag(w) S - c (e^T S) + k v^T;   o = S^T r         (decay and removal both read the state before the token)
//   decayed sum with one constant decay per head (SCAN_RETAIN):
//       S <- g S + k v^T;   o = S^T q                           (the read-out sees this token's write)
//   decayed sum with a step size per head and token (SCAN_TOKEN), dt and g = exp(-rate dt) scalars, D a constant per head:
//       S <- g S + dt k v^T;   o = S^T q + D v
//   decayed sum with one decay per key channel and token (SCAN_GATED), w a vector over the key channels:
//       S <- diag(w) S + k v^T;   o = S^T q
//
// Everything that enters the recurrence is float32: the kernels here read the float32 results of the input
// projections, and the state never leaves float32.  A request's state lives in its slot between steps, so
// the result at a position does not depend on how the request was cut into steps: the scan visits the
// tokens one after another either way, and the order of additions inside a token depends on the sizes only.
//
// Around the scans:
//   * prism_conv_unit_gates  per token: the short causal convolution over time of the q | k | v channels (its
//     last taps - 1 inputs per request are state too) with silu, q and k made unit vectors per head (q also
//     times dk^-1/2), beta = sigmoid(b), g = exp(-exp(A_log) softplus(a + dt_bias));
//   * prism_state_tail       the last rows of a step's input per request into a [slots, rows, width] state (the
//     convolution's tail; with one row, the previous token's input of a token-shift mix);
//   * prism_shift_mix        x + (x_prev - x) mu_s for several mu at once (x_prev of a step's first token comes
//     from the state);
//   * prism_headnorm_gate    o / rms(o) per head, times a weight, times silu(gate), times a constant;
//   * prism_part_norm_gate   the same over equal parts of the concatenated heads, the gate before or after the norm;
//   * prism_step_sizes       softplus(z + bias) and the decay exp(-exp(a_log) times it) per head and token.
#include "f32x2.cuh"
#include "mma_helpers.cuh"

#define PRISM_SCAN_DELTA 0
#define PRISM_SCAN_BONUS 1
#define PRISM_SCAN_CHANNEL 2
#define PRISM_SCAN_GENERAL 3
#define PRISM_SCAN_RETAIN 4
#define PRISM_SCAN_TOKEN 5
#define PRISM_SCAN_GATED 6

namespace prism {

__device__ __forceinline__ float sigmoid_f(float z) { return 1.f / (1.f + expf(-z)); }
__device__ __forceinline__ float silu_f(float z) { return z / (1.f + expf(-z)); }
__device__ __forceinline__ float softplus_f(float z) { return z > 20.f ? z : log1pf(expf(z)); }

// ---------------------------------------------------------------------------------------------------------
// conv + silu, unit vectors, gates.  One CTA per token.
//   proj   [T, *] float32, row stride ps: columns [0, C) are the q | k | v channels (C = 2 G dk + H dv),
//          columns ob .. ob + H the beta projection, oa .. oa + H the decay projection
//   taps   [C, K] (last column: the current token's)
//   tail   [slots, K - 1, C] float32: the K - 1 inputs before the step's first token, oldest first
//   qkv    [T, C] float32 out;   bg [T, 2 H] float32 out: beta | g
// ---------------------------------------------------------------------------------------------------------
__global__ void conv_unit_gates_kernel(const float* __restrict__ proj_in, long long ps, int ob, int oa,
                                       const void* __restrict__ taps, int taps_bf16, int K,
                                       const float* tail, const void* __restrict__ a_log, int a_log_bf16,
                                       const void* __restrict__ dt_bias, int dt_bf16, const int* __restrict__ tok_seg,
                                       const int* __restrict__ seg_start, const int* __restrict__ slots, int G, int H,
                                       int dk, int dv, float unit_eps, float* __restrict__ qkv, float* __restrict__ bg,
                                       int move_tail) {
    pdl_trigger();
    pdl_wait();
    const float* proj = pdl_fresh(proj_in);
    extern __shared__ float y[];                       // [C]
    const int t = blockIdx.x, seg = tok_seg[t];
    const int i = t - seg_start[seg];                  // place of the token in its segment
    const int C = 2 * G * dk + H * dv;
    float* tl = const_cast<float*>(tail) + (size_t)slots[seg] * (K - 1) * C;
    for (int c = threadIdx.x; c < C; c += blockDim.x) {
        float acc = 0.f;
        for (int j = K - 1; j >= 0; --j) {             // lag j: the input j tokens back; oldest first
            const int src = i - j;
            const float x = src >= 0 ? proj[(size_t)(t - j) * ps + c] : tl[(size_t)(K - 1 + src) * C + c];
            acc += load_param(taps, taps_bf16, (size_t)c * K + (K - 1 - j)) * x;
        }
        y[c] = silu_f(acc);
        // a step of single tokens: this CTA is the only reader of its request's tail, and a thread the only one of
        // its channel, so it moves the tail up by this token itself (no second launch)
        if (move_tail && K > 1) {
            for (int r = 0; r + 2 < K; ++r) tl[(size_t)r * C + c] = tl[(size_t)(r + 1) * C + c];
            tl[(size_t)(K - 2) * C + c] = proj[(size_t)t * ps + c];
        }
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    float* out = qkv + (size_t)t * C;
    for (int hh = warp; hh < 2 * G; hh += nwarps) {    // q heads, then k heads
        const float* row = y + hh * dk;
        float ss = 0.f;
        for (int d = lane; d < dk; d += 32) ss += row[d] * row[d];
        ss = warp_sum(ss);
        const float inv = (1.f / sqrtf(ss + unit_eps)) * (hh < G ? 1.f / sqrtf((float)dk) : 1.f);
        for (int d = lane; d < dk; d += 32) out[hh * dk + d] = row[d] * inv;
    }
    for (int c = 2 * G * dk + threadIdx.x; c < C; c += blockDim.x) out[c] = y[c];
    if (a_log == nullptr) {            // the decay is formed elsewhere (one per key channel): bg [T, H] holds beta alone
        for (int h = threadIdx.x; h < H; h += blockDim.x) bg[(size_t)t * H + h] = sigmoid_f(proj[(size_t)t * ps + ob + h]);
        return;
    }
    for (int h = threadIdx.x; h < H; h += blockDim.x) {
        bg[(size_t)t * 2 * H + h] = sigmoid_f(proj[(size_t)t * ps + ob + h]);
        const float dt = softplus_f(proj[(size_t)t * ps + oa + h] + load_param(dt_bias, dt_bf16, h));
        bg[(size_t)t * 2 * H + H + h] = expf(-expf(load_param(a_log, a_log_bf16, h)) * dt);
    }
}

// The same for a step of many tokens: a warp takes one head's channels (q, k or v; d = lane + 32 m) of RUN tokens one
// after another with the inputs of the last K - 1 tokens and the taps in registers, so that every input is read once
// instead of K times and nothing passes through shared memory; sums in the order of the kernel above.  One more "head"
// forms the gates.  Bound by the bytes of proj and qkv (2,048 tokens of 6,144 channels, 101 MB, inputs from memory: 145 us by the
// kernel above, 38 us here; what the projection just wrote is in L2 in part).
constexpr int CONV_RUN = 16, CONV_TAPS = 4;
template <int M>
__global__ void __launch_bounds__(128) conv_unit_gates_run_kernel(const float* __restrict__ proj_in, long long ps, int ob, int oa,
                                                                  const void* __restrict__ taps, int taps_bf16, int K,
                                                                  const float* tail, const void* __restrict__ a_log, int a_log_bf16,
                                                                  const void* __restrict__ dt_bias, int dt_bf16,
                                                                  const int* __restrict__ tok_seg, const int* __restrict__ seg_start,
                                                                  const int* __restrict__ slots, int T, int G, int H, int dk, int dv,
                                                                  float unit_eps, float* __restrict__ qkv, float* __restrict__ bg) {
    pdl_trigger();
    pdl_wait();
    const float* proj = pdl_fresh(proj_in);
    const int lane = threadIdx.x & 31, hh = blockIdx.y * 4 + (threadIdx.x >> 5);       // neighbouring warps: neighbouring channels
    const int t0 = blockIdx.x * CONV_RUN, t1 = min(T, t0 + CONV_RUN);
    const int C = 2 * G * dk + H * dv;
    if (hh > 2 * G + H) return;
    if (hh == 2 * G + H) {
        for (int i = lane; i < (t1 - t0) * H; i += 32) {
            const int t = t0 + i / H, h = i % H;
            const float beta = sigmoid_f(proj[(size_t)t * ps + ob + h]);
            if (a_log == nullptr) {
                bg[(size_t)t * H + h] = beta;
            } else {
                bg[(size_t)t * 2 * H + h] = beta;
                const float dt = softplus_f(proj[(size_t)t * ps + oa + h] + load_param(dt_bias, dt_bf16, h));
                bg[(size_t)t * 2 * H + H + h] = expf(-expf(load_param(a_log, a_log_bf16, h)) * dt);
            }
        }
        return;
    }
    const bool unit = hh < 2 * G;
    const int n = unit ? dk : dv, c0 = unit ? hh * dk : 2 * G * dk + (hh - 2 * G) * dv;
    float w[CONV_TAPS][M], x[CONV_TAPS][M];            // lag j: tap and input of j tokens back (lags from K on: zero)
#pragma unroll
    for (int j = 0; j < CONV_TAPS; ++j)
#pragma unroll
        for (int m = 0; m < M; ++m) {
            const int d = lane + 32 * m;
            w[j][m] = j < K && d < n ? load_param(taps, taps_bf16, (size_t)(c0 + d) * K + (K - 1 - j)) : 0.f;
            x[j][m] = 0.f;
        }
    int seg = -1, s0 = 0, s1 = 0;
    float ahead[M];                                    // the next token's inputs, asked for before this one's are used
#pragma unroll
    for (int m = 0; m < M; ++m) ahead[m] = lane + 32 * m < n ? proj[(size_t)t0 * ps + c0 + lane + 32 * m] : 0.f;
    for (int t = t0; t < t1; ++t) {
        if (t >= s1) {                                 // the run's first token, or a segment's: the inputs before it
            seg = tok_seg[t], s0 = seg_start[seg], s1 = seg_start[seg + 1];
            const float* tl = tail + (size_t)slots[seg] * (K - 1) * C;
#pragma unroll
            for (int j = 0; j + 1 < CONV_TAPS; ++j) {  // becomes lag j + 1
                const int src = t - s0 - 1 - j;
#pragma unroll
                for (int m = 0; m < M; ++m) {
                    const int d = lane + 32 * m;
                    x[j][m] = j + 1 < K && d < n ? (src >= 0 ? proj[(size_t)(t - 1 - j) * ps + c0 + d] : tl[(size_t)(K - 1 + src) * C + c0 + d]) : 0.f;
                }
            }
        }
        float y[M], ss = 0.f;
#pragma unroll
        for (int m = 0; m < M; ++m) {
#pragma unroll
            for (int j = CONV_TAPS - 1; j > 0; --j) x[j][m] = x[j - 1][m];
            x[0][m] = ahead[m];
            if (t + 1 < t1) ahead[m] = lane + 32 * m < n ? proj[(size_t)(t + 1) * ps + c0 + lane + 32 * m] : 0.f;
            float acc = 0.f;
#pragma unroll
            for (int j = CONV_TAPS - 1; j >= 0; --j)
                if (j < K) acc += w[j][m] * x[j][m];
            y[m] = silu_f(acc);
            if (lane + 32 * m < n) ss += y[m] * y[m];
        }
        if (unit) {
            ss = warp_sum(ss);
            const float inv = (1.f / sqrtf(ss + unit_eps)) * (hh < G ? 1.f / sqrtf((float)dk) : 1.f);
#pragma unroll
            for (int m = 0; m < M; ++m) y[m] *= inv;
        }
#pragma unroll
        for (int m = 0; m < M; ++m)
            if (lane + 32 * m < n) qkv[(size_t)t * C + c0 + lane + 32 * m] = y[m];
    }
}

// tail[slot][r][c] <- the input (rows - r) tokens before the end of the request's tokens so far: from this
// step's rows where the step reaches that far back, else from the tail as it was (shifted).  One CTA per
// segment; a thread owns a column, and walks r upwards, so that what it still needs is never overwritten.
__global__ void state_tail_kernel(const float* __restrict__ src_in, long long ss, int width, float* __restrict__ tail,
                                  int rows, const int* __restrict__ seg_start, const int* __restrict__ slots) {
    pdl_trigger();
    pdl_wait();
    const float* src = pdl_fresh(src_in);
    const int seg = blockIdx.x, s0 = seg_start[seg], qlen = seg_start[seg + 1] - s0;
    float* tl = tail + (size_t)slots[seg] * rows * width;
    for (int c = threadIdx.x; c < width; c += blockDim.x)
        for (int r = 0; r < rows; ++r) {
            const int idx = qlen - rows + r;           // place in the segment of the token that row r holds afterwards
            tl[(size_t)r * width + c] = idx >= 0 ? src[(size_t)(s0 + idx) * ss + c] : tl[(size_t)(r + qlen) * width + c];
        }
}

// out[s][t][c] = x[t][c] + (x_prev[t][c] - x[t][c]) mu[s][c],  s < n;  x_prev of a segment's first token is prev[slot].
template <typename T>
__global__ void shift_mix_kernel(const float* __restrict__ x_in, int D, const float* prev,
                                 const void* __restrict__ mu, int mu_bf16, int n, const int* __restrict__ tok_seg,
                                 const int* __restrict__ seg_start, const int* __restrict__ slots, T* __restrict__ out,
                                 long long out_plane, int keep_prev) {
    pdl_trigger();
    pdl_wait();
    const float* x = pdl_fresh(x_in);
    const int t = blockIdx.x, seg = tok_seg[t];
    float* own = const_cast<float*>(prev) + (size_t)slots[seg] * D;
    const float* xp = t > seg_start[seg] ? x + (size_t)(t - 1) * D : own;
    for (int c = threadIdx.x; c < D; c += blockDim.x) {
        const float a = x[(size_t)t * D + c], d = xp[c] - a;
        for (int s = 0; s < n; ++s)
            out[(size_t)s * out_plane + (size_t)t * D + c] = from_float<T>(a + d * load_param(mu, mu_bf16, (size_t)s * D + c));
        if (keep_prev) own[c] = a;       // a step of single tokens: this token is its request's previous one from now on
    }
}

// w[t][c] <- exp(-exp(w[t][c] + w0[c])) in place: the decay of every key channel from its exponent, once for all
// the CTAs of the scan that read it (a step with many tokens; a decode step lets the scan do it).
__global__ void decay_from_exponent_kernel(float* __restrict__ w, long long ws, const void* __restrict__ w0, int w0_bf16, int A) {
    pdl_trigger();
    pdl_wait();
    float* row = pdl_fresh(w) + (size_t)blockIdx.y * ws;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < A; c += gridDim.x * blockDim.x)
        row[c] = expf(-expf(row[c] + load_param(w0, w0_bf16, c)));
}

// out[t][n] = epi(sum_r inner(low[t][r]) w2t[r][n] + b[n]): the second half of a low-rank product with what follows it,
// in one launch and float32 throughout.  inner: tanh (1) or nothing (0).  epi:
//   PRISM_LR_EXPEXP    exp(-exp(z))                          a per-channel decay from its double exponent
//   PRISM_LR_SOFTPLUS  exp(-exp(alog[n / per]) softplus(z))  a per-channel decay with one rate per group of `per` channels
//   PRISM_LR_SIGMOID   sigmoid(z)                            a gate
//   PRISM_LR_EXPSIG    exp(-rate sigmoid(z))                 a per-channel decay kept inside (exp(-rate), 1), rate a constant
//   PRISM_LR_SIGPOW    sigmoid(z)^rate                       a per-channel decay near one for a small constant rate
// b may be null.  A CTA takes 128 channels and sixteen tokens, so that every weight it reads serves sixteen tokens
// (whose inner values sit side by side in shared memory: four 128-bit loads per weight); w2t is the second matrix
// transposed, [R, N], so that neighbouring threads read neighbouring floats.  A step of few tokens is bound by the latency of the weights:
// they are asked for in L2 before the dependency wait and read sixteen at a time, by CTAs of up to eight tokens (TOK 8; R 64, N 2,048:
// 7.9 -> 5.3 us with the weights in L2, inside a decode step that has streamed others since 16 -> 8.5).
#define PRISM_LR_EXPEXP 0
#define PRISM_LR_SOFTPLUS 1
#define PRISM_LR_SIGMOID 2
#define PRISM_LR_EXPSIG 3
#define PRISM_LR_SIGPOW 4
template <int TOK>
__global__ void __launch_bounds__(128)
lowrank_decay_kernel(const float* __restrict__ low_in, long long ls, int R, const float* __restrict__ w2t,
                                     const void* __restrict__ w0, int w0_bf16, int N, int T, float* __restrict__ out,
                                     long long os, int inner, int epi, const void* __restrict__ alog, int alog_bf16, int per,
                                     float crate) {
    pdl_trigger();
    extern __shared__ __align__(16) float s[];         // [R][TOK]
    const int t0 = blockIdx.y * TOK, n = blockIdx.x * 128 + threadIdx.x;
    if (TOK == 8) {                                    // the weights' lines: 128 floats of each of R rows
        for (int i = threadIdx.x; i < 4 * R; i += 128) {
            const int c = blockIdx.x * 128 + i % 4 * 32;
            if (c < N) asm volatile("prefetch.global.L2 [%0];" ::"l"(w2t + (size_t)(i / 4) * N + c));
        }
    }
    pdl_wait();
    const float* low = pdl_fresh(low_in);
    for (int i = threadIdx.x; i < TOK * R; i += 128) {
        const int j = i / R, r = i - j * R;            // neighbouring threads read neighbouring entries of a token's row
        const float v = t0 + j < T ? low[(size_t)(t0 + j) * ls + r] : 0.f;
        s[r * TOK + j] = inner ? tanhf(v) : v;
    }
    __syncthreads();
    if (n >= N) return;
    float acc[TOK];
#pragma unroll
    for (int j = 0; j < TOK; ++j) acc[j] = 0.f;
    auto add = [&](int r, float w) {
#pragma unroll
        for (int j = 0; j < TOK; j += 4) {
            const float4 t4 = *reinterpret_cast<const float4*>(s + r * TOK + j);
            acc[j] += w * t4.x;
            acc[j + 1] += w * t4.y;
            acc[j + 2] += w * t4.z;
            acc[j + 3] += w * t4.w;
        }
    };
    if constexpr (TOK == 8) {
        // the last few too come in one round (8 tokens, a rank of 28: 4.7 us with its last twelve one after another, now 3.9)
        for (int r0 = 0; r0 < R; r0 += 16) {
            float w[16];
#pragma unroll
            for (int e = 0; e < 16; ++e) w[e] = r0 + e < R ? w2t[(size_t)(r0 + e) * N + n] : 0.f;
#pragma unroll
            for (int e = 0; e < 16; ++e)
                if (r0 + e < R) add(r0 + e, w[e]);
        }
    } else {
        for (int r = 0; r < R; ++r) add(r, w2t[(size_t)r * N + n]);
    }
    const float b = w0 != nullptr ? load_param(w0, w0_bf16, n) : 0.f;
    const float rate = epi == PRISM_LR_SOFTPLUS ? expf(load_param(alog, alog_bf16, n / per)) : 0.f;
#pragma unroll
    for (int j = 0; j < TOK; ++j)
        if (t0 + j < T) {
            const float z = acc[j] + b;
            out[(size_t)(t0 + j) * os + n] = epi == PRISM_LR_EXPEXP ? expf(-expf(z))
                                             : epi == PRISM_LR_SOFTPLUS ? expf(-rate * softplus_f(z))
                                             : epi == PRISM_LR_EXPSIG ? expf(-crate * sigmoid_f(z))
                                             : epi == PRISM_LR_SIGPOW ? expf(-crate * softplus_f(-z)) : sigmoid_f(z);
        }
}

// ex[t][h dk + i] = e_i = k_i / sqrt(sum_i k_i^2 + unit_eps) per head (the unit key), and
// ex[t][(H + h) dk + i] = sigmoid(a_i + ab[h dk + i]) e_i (the removal rate per channel times it): what the generalized
// delta rule takes out of its state.  k, a: float32 column blocks of one product (row stride ps).  One warp per (token, head).
__global__ void unit_removal_kernel(const float* __restrict__ k_in, const float* __restrict__ a_in, long long ps,
                                    const void* __restrict__ ab, int ab_bf16, float unit_eps, int Ttot, int H, int dk,
                                    float* __restrict__ ex) {
    pdl_trigger();
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const long long w = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (w >= (long long)Ttot * H) return;
    const int t = (int)(w / H), h = (int)(w % H);
    const float* k = pdl_fresh(k_in) + (size_t)t * ps + (size_t)h * dk;
    const float* a = pdl_fresh(a_in) + (size_t)t * ps + (size_t)h * dk;
    float ss = 0.f;
    for (int i = lane; i < dk; i += 32) ss += k[i] * k[i];
    ss = warp_sum(ss);
    const float inv = 1.f / sqrtf(ss + unit_eps);
    float* e = ex + (size_t)t * 2 * H * dk + (size_t)h * dk;
    for (int i = lane; i < dk; i += 32) {
        const float u = k[i] * inv;
        e[i] = u;
        e[(size_t)H * dk + i] = sigmoid_f(a[i] + (ab != nullptr ? load_param(ab, ab_bf16, (size_t)h * dk + i) : 0.f)) * u;
    }
}

// out[t][h dv + c] = o[t][h][c] / sqrt(mean_c(o[t][h]^2) + eps) * weight[widx] * act(gate[t][h dv + c]) * scale,
// act silu, or sigmoid (gate_sigmoid; the gate may then hold the sigmoid already: gate_sigmoid 2),
// widx = c (one weight for all heads) or h dv + c (per_head_weight); weight null: ones.  One warp per (token, head).
template <typename T>
__global__ void headnorm_gate_kernel(const float* __restrict__ o_in, const float* __restrict__ gate_in, long long gs,
                                     const void* __restrict__ weight, int weight_bf16, int per_head_weight, float eps,
                                     float scale, int Ttot, int H, int dv, T* __restrict__ out, long long os, int gate_sigmoid) {
    pdl_trigger();
    pdl_wait();
    const float* o = pdl_fresh(o_in);
    const float* gate = pdl_fresh(gate_in);
    const int lane = threadIdx.x & 31;
    const long long w = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (w >= (long long)Ttot * H) return;
    const int t = (int)(w / H), h = (int)(w % H);
    const float* row = o + ((size_t)t * H + h) * dv;
    const float* gr = gate + (size_t)t * gs + (size_t)h * dv;
    constexpr int AHEAD = 4;                           // entries a lane keeps: rows and gates of up to 128 are all on their way
                                                       // before the sum (2,048 tokens, 16 heads of 128: 26 -> 19 us)
    float x[AHEAD], g4[AHEAD];
    float ss = 0.f;
#pragma unroll
    for (int m = 0; m < AHEAD; ++m) {
        const int c = lane + 32 * m;
        x[m] = c < dv ? row[c] : 0.f;
        g4[m] = c < dv ? gr[c] : 0.f;
    }
#pragma unroll
    for (int m = 0; m < AHEAD; ++m) ss += x[m] * x[m];
    for (int c = lane + 32 * AHEAD; c < dv; c += 32) ss += row[c] * row[c];
    ss = warp_sum(ss);
    const float inv = 1.f / sqrtf(ss / (float)dv + eps);
    auto put = [&](int c, float v, float gz) {
        const float wv = weight != nullptr ? load_param(weight, weight_bf16, per_head_weight ? (size_t)h * dv + c : (size_t)c) : 1.f;
        const float g = gate_sigmoid == 2 ? gz : (gate_sigmoid ? sigmoid_f(gz) : silu_f(gz));
        out[(size_t)t * os + (size_t)h * dv + c] = from_float<T>(v * inv * wv * g * scale);
    };
#pragma unroll
    for (int m = 0; m < AHEAD; ++m)
        if (lane + 32 * m < dv) put(lane + 32 * m, x[m], g4[m]);
    for (int c = lane + 32 * AHEAD; c < dv; c += 32) put(c, row[c], gr[c]);
}

// bg[t][h] = softplus(z[t][h] + bias[h]) (a step size) and bg[t][H + h] = exp(-exp(a_log[h]) times it) (the decay it makes).
__global__ void step_sizes_kernel(const float* __restrict__ z_in, long long zs, const void* __restrict__ bias, int bias_bf16,
                                  const void* __restrict__ a_log, int a_log_bf16, int T, int H, float* __restrict__ bg) {
    pdl_trigger();
    pdl_wait();
    const float* z = pdl_fresh(z_in);
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < (long long)T * H; i += (long long)gridDim.x * blockDim.x) {
        const int t = (int)(i / H), h = (int)(i - (long long)t * H);
        const float dt = softplus_f(z[(size_t)t * zs + h] + load_param(bias, bias_bf16, h));
        bg[(size_t)t * 2 * H + h] = dt;
        bg[(size_t)t * 2 * H + H + h] = expf(-expf(load_param(a_log, a_log_bf16, h)) * dt);
    }
}

// Rows of `parts` equal parts of w entries each, normed part by part:
//   before:  y = x * act(gate);  out = y / sqrt(mean_part(y^2) + eps) * weight * scale
//   after:   out = x / sqrt(mean_part(x^2) + eps) * weight * act(gate) * scale
// x [T, parts w] float32 contiguous, gate float32 and out with row strides of their own, weight [parts w]; act silu, or
// sigmoid.  One CTA per (token, part); VEC 4 reads and writes four neighbouring entries at a time.
template <typename T, int VEC>
__global__ void part_norm_gate_kernel(const float* __restrict__ x_in, const float* __restrict__ gate_in, long long gs,
                                      const void* __restrict__ weight, int weight_bf16, float eps, float scale, int parts, int w,
                                      int before, int sigmoid_act, T* __restrict__ out, long long os) {
    extern __shared__ __align__(16) float row[];       // [w]
    __shared__ float scratch[33];
    pdl_trigger();
    pdl_wait();
    const int t = blockIdx.x, p = blockIdx.y;
    const float* x = pdl_fresh(x_in) + ((size_t)t * parts + p) * w;
    const float* gate = pdl_fresh(gate_in) + (size_t)t * gs + (size_t)p * w;
    T* o = out + (size_t)t * os + (size_t)p * w;
    float ss = 0.f;
    for (int c = threadIdx.x * VEC; c < w; c += blockDim.x * VEC) {
        float v[VEC], g[VEC];
        if (VEC == 4) {
            const float4 a = *reinterpret_cast<const float4*>(x + c);
            v[0] = a.x; v[1 % VEC] = a.y; v[2 % VEC] = a.z; v[3 % VEC] = a.w;
            if (before) {
                const float4 b = *reinterpret_cast<const float4*>(gate + c);
                g[0] = b.x; g[1 % VEC] = b.y; g[2 % VEC] = b.z; g[3 % VEC] = b.w;
            }
        } else {
            v[0] = x[c];
            if (before) g[0] = gate[c];
        }
#pragma unroll
        for (int k = 0; k < VEC; ++k) {
            if (before) v[k] *= sigmoid_act ? sigmoid_f(g[k]) : silu_f(g[k]);
            ss += v[k] * v[k];
            row[c + k] = v[k];
        }
    }
    ss = block_sum(ss, scratch);
    const float inv = scale / sqrtf(ss / (float)w + eps);
    for (int c = threadIdx.x * VEC; c < w; c += blockDim.x * VEC) {
        float g[VEC], y[VEC];
        if (!before) {
            if (VEC == 4) {
                const float4 b = *reinterpret_cast<const float4*>(gate + c);
                g[0] = b.x; g[1 % VEC] = b.y; g[2 % VEC] = b.z; g[3 % VEC] = b.w;
            } else {
                g[0] = gate[c];
            }
        }
#pragma unroll
        for (int k = 0; k < VEC; ++k) {
            y[k] = row[c + k] * inv * load_param(weight, weight_bf16, (size_t)p * w + c + k);
            if (!before) y[k] *= sigmoid_act ? sigmoid_f(g[k]) : silu_f(g[k]);
        }
        if (VEC == 4 && sizeof(T) == 2) {
            *reinterpret_cast<uint2*>(o + c) = make_uint2(pack_bf16(y[0], y[1 % VEC]), pack_bf16(y[2 % VEC], y[3 % VEC]));
        } else {
#pragma unroll
            for (int k = 0; k < VEC; ++k) o[c + k] = from_float<T>(y[k]);
        }
    }
}

// ---------------------------------------------------------------------------------------------------------
// The scan.  grid (heads, segments, column blocks); the L threads of a column are neighbouring lanes of a warp,
// each owns R rows - quads of four neighbouring rows, quad part + L m - of CPT neighbouring columns of S in
// registers, and they add up their partial dot products by shuffles.  The step's vectors come through shared memory
// TB tokens at a time with cp.async, the next blocks on their way while this one is worked on; a thread reads its
// quads of q, k (w, e, c) with 128-bit loads, once for its CPT columns.  The state is kept in memory as
// [slot][head][column][row], so that the threads of a column read neighbouring floats.
//
// What bounds it, and the split: a token's work on a column is a chain (the delta rules: dot product, shuffles,
// update), so few columns leave latency exposed; and every column of a thread wants the token's vectors through
// shared memory, 128 bytes a cycle and SM, so many columns are bound by that unless a thread has several.  Tokens are
// taken eight at a time in straight line code: a token's read-out stands behind the next one's dot products, where
// the chain waits for its shuffles, and the eight read-outs are added up across the lanes together (7 shuffles
// instead of 24; the additions are the same).  The results do not depend on CPT, on the blocks or on how a request
// was cut: every sum has one order.
//   SCAN_DELTA:  x [T, *] row stride xs: q of kv head g at qo + g dk, k at ko + g dk; v at vo + h dv;
//                bg [T, 2 H]: beta | g.
//   SCAN_BONUS:  r at qo + h dk, k at ko + h dk, v at vo + h dv, the decay's exponent ww [T, H dk] (row stride ws)
//                with w = exp(-exp(ww + w0)) formed in shared memory, w0 [H dk], bonus u [H dk].  The bonus term is
//                (sum_i r_i u_i k_i) v: one sum for all columns.
//   SCAN_CHANNEL: q, k, v as for SCAN_DELTA; the decay itself in ww [T, H dk] (row stride ws); bg [T, H]: beta.
//   SCAN_GENERAL: r, k, v as for SCAN_BONUS; the decay itself in ww; ex [T, 2 H dk]: the unit key e at h dk, c at (H + h) dk.
//   SCAN_RETAIN: q, k, v as for SCAN_BONUS; the decay of head h in w0[h].
//   SCAN_TOKEN: q, k, v as for SCAN_DELTA; bg [T, 2 H]: dt | g; D of head h in w0[h] (null: no such term).
//   SCAN_GATED: q, k, v as for SCAN_BONUS; the decay itself in ww [T, H dk].
// ---------------------------------------------------------------------------------------------------------
struct ScanArgs {
    const float* x;          // q | k | v (or r | k | v) rows
    long long xs;
    long long qo, ko, vo;
    const float* bg;         // DELTA: beta | g
    const float* ww;         // BONUS: the decay's exponent before w0
    long long ws;
    const void* w0;
    int w0_bf16;
    const void* u;
    int u_bf16;
    const float* ex;         // GENERAL: unit key | removal rate times unit key, [T, 2 H dk] (row stride es)
    long long es;
    float* state;            // [slots, H, dv, dk]
    const int* seg_start;
    const int* slots;
    float* out;              // [T, H, dv]
    int H, rep, dk, dkp, dv, cols, colsp, L, TB, NBUF;
    int vec;                 // every source row piece starts on 16 bytes and is whole quads long
    int w_ready;             // BONUS: ww holds the decay itself already (prism_decay_from_exponent)
};

__device__ __forceinline__ void cp_async_f(float* smem, const float* gmem, int floats) {      // 1 or 4 floats
    const unsigned dst = (unsigned)__cvta_generic_to_shared(smem);
    if (floats == 4) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(gmem));
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(dst), "l"(gmem));
}

// all but the newest `n` groups (at most 6) have landed
__device__ __forceinline__ void cp_async_wait_upto(int n) {
    switch (n) {
        case 1: cp_async_wait<1>(); break;
        case 2: cp_async_wait<2>(); break;
        case 3: cp_async_wait<3>(); break;
        case 4: cp_async_wait<4>(); break;
        case 5: cp_async_wait<5>(); break;
        case 6: cp_async_wait<6>(); break;
        default: cp_async_wait<0>();
    }
}

// sum over the L (a power of two, known when the kernel is compiled) neighbouring lanes that share a column
template <int L> __device__ __forceinline__ float column_sum(float v) {
    if (L > 16) v += __shfl_xor_sync(0xffffffffu, v, 16);
    if (L > 8) v += __shfl_xor_sync(0xffffffffu, v, 8);
    if (L > 4) v += __shfl_xor_sync(0xffffffffu, v, 4);
    if (L > 2) v += __shfl_xor_sync(0xffffffffu, v, 2);
    if (L > 1) v += __shfl_xor_sync(0xffffffffu, v, 1);
    return v;
}

// vectors over the key channels that a token brings: q (or r) and k, a decay per channel, a unit key and what it removes
__host__ __device__ constexpr int scan_vectors(int mode) {
    return (mode == PRISM_SCAN_DELTA || mode == PRISM_SCAN_RETAIN || mode == PRISM_SCAN_TOKEN) ? 2 : (mode == PRISM_SCAN_GENERAL ? 5 : 3);
}

// four neighbouring floats of shared memory as two pairs
__device__ __forceinline__ ulonglong2 quad(const float* p) { return *reinterpret_cast<const ulonglong2*>(p); }
// x . y over a thread's quads, four chains side by side
template <int Q> __device__ __forceinline__ float quad_dot(const uint64_t (&x)[2 * Q], const ulonglong2 (&y)[Q]) {
    uint64_t a = 0, b = 0;
#pragma unroll
    for (int m = 0; m < Q; ++m) {
        fma2(a, x[2 * m], y[m].x);
        fma2(b, x[2 * m + 1], y[m].y);
    }
    const float2 p = unpack2(a), r = unpack2(b);
    return (p.x + p.y) + (r.x + r.y);
}

__device__ __forceinline__ void quad(const float* p, float (&v)[4]) {
    const float4 x = *reinterpret_cast<const float4*>(p);
    v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w;
}

// Padding entries of `rows` tokens' places in shared memory (rows beyond dk that the column's threads cover, columns beyond
// the CTA's) are never written by the copies: zero them once.
__device__ __forceinline__ void zero_padding(float* sm, int rows, int per_tok, int NV, int dk, int dkp, int ncols, int colsp) {
    if (dkp == dk && colsp == ncols) return;
    const int pad = NV * (dkp - dk) + (colsp - ncols);
    for (int i = threadIdx.x; i < rows * pad; i += blockDim.x) {
        const int slot = i / pad, c = i - slot * pad;
        const int which = c / (dkp - dk > 0 ? dkp - dk : 1);
        const int at = (dkp > dk && which < NV) ? which * dkp + dk + (c - which * (dkp - dk)) : NV * dkp + ncols + (c - NV * (dkp - dk));
        sm[(size_t)slot * per_tok + at] = 0.f;
    }
}

// w <- exp(-exp(w + w0)) of head h for `nb` tokens, per_tok apart; one warp
__device__ __forceinline__ void decays_in_place(const ScanArgs& a, float* w, int per_tok, int nb, int h) {
    for (int idx = threadIdx.x & 31; idx < nb * a.dk; idx += 32) {
        const int tt = idx / a.dk, i = idx - tt * a.dk;
        float& z = w[(size_t)tt * per_tok + i];
        z = expf(-expf(z + load_param(a.w0, a.w0_bf16, (size_t)h * a.dk + i)));
    }
}

constexpr int SCAN_STEP_BLOCKS = 3;          // blocks of tokens in shared memory: in use, landed, on its way

// The scan of a step of few tokens a request: bound by the state's way in and out, so a thread has one column in as few
// registers as it takes (70 to 90 for 128 rows and more, so that five CTAs and more share an SM) and the producer a short
// loop a token.  48 heads of 128 x 128, delta rule, 64 single tokens: 84 us, by the kernel below 162 us.  Every product and
// sum is written out as the kernel below has it, so that a request's values do not depend on which of the two ran.
template <int MODE, int R, int L>
__global__ void scan_step_kernel(const ScanArgs a) {
    pdl_trigger();
    pdl_wait();
    extern __shared__ __align__(16) float sm[];
    constexpr int NV = scan_vectors(MODE), Q = R / 4, dkp = L * R, NBUF = SCAN_STEP_BLOCKS;
    const int h = blockIdx.x, seg = blockIdx.y, col0 = blockIdx.z * a.cols;
    const int s0 = a.seg_start[seg], qlen = a.seg_start[seg + 1] - s0;
    const int dk = a.dk, dv = a.dv, TB = a.TB;
    const int ncols = min(a.cols, dv - col0);
    const int CT = blockDim.x - 32;                    // the last warp brings the vectors in
    const bool producer = (int)threadIdx.x >= CT;
    const int part = threadIdx.x % L;
    const bool live = !producer && (int)threadIdx.x / L < ncols;
    const int lc = live ? threadIdx.x / L : 0, col = col0 + lc;
    const int kvh = h / a.rep;
    const int per_tok = NV * dkp + a.colsp + 4;
    const float* x = pdl_fresh(a.x);
    const float* bg = pdl_fresh(a.bg);
    const float* ww = pdl_fresh(a.ww);
    const float* ex = pdl_fresh(a.ex);
    zero_padding(sm, NBUF * TB, per_tok, NV, dk, dkp, ncols, a.colsp);
    float* ub = sm + (size_t)NBUF * TB * per_tok;      // BONUS: u [dkp]
    if (MODE == PRISM_SCAN_BONUS)
        for (int i = threadIdx.x; i < dkp; i += blockDim.x) ub[i] = i < dk ? load_param(a.u, a.u_bf16, (size_t)h * dk + i) : 0.f;
    __syncthreads();

    auto stage = [&](int b0, int buf) {                // asks for block b0 of the segment's tokens
        const int lane = threadIdx.x - CT;
        const int nb = min(TB, qlen - b0);
        float* dst0 = sm + (size_t)buf * TB * per_tok;
        const int unit = a.vec ? 4 : 1;
        const int nk = (dk + unit - 1) / unit, nc = (ncols + unit - 1) / unit;     // pieces per vector
        const size_t head_q = (size_t)((MODE == PRISM_SCAN_DELTA || MODE == PRISM_SCAN_CHANNEL || MODE == PRISM_SCAN_TOKEN) ? kvh : h) * dk;
        for (int tt = 0; tt < nb; ++tt) {
            const size_t t = (size_t)(s0 + b0 + tt);
            const float* xr = x + t * a.xs;
            float* dst = dst0 + (size_t)tt * per_tok;
            for (int c = lane; c < nk; c += 32) {
                cp_async_f(dst + c * unit, xr + a.qo + head_q + c * unit, unit);
                cp_async_f(dst + dkp + c * unit, xr + a.ko + head_q + c * unit, unit);
                if (NV > 2) cp_async_f(dst + 2 * dkp + c * unit, ww + t * a.ws + (size_t)h * dk + c * unit, unit);
                if (NV > 3) {
                    cp_async_f(dst + 3 * dkp + c * unit, ex + t * a.es + (size_t)h * dk + c * unit, unit);
                    cp_async_f(dst + 4 * dkp + c * unit, ex + t * a.es + (size_t)(a.H + h) * dk + c * unit, unit);
                }
            }
            for (int c = lane; c < nc; c += 32)
                cp_async_f(dst + NV * dkp + c * unit, xr + a.vo + (size_t)h * dv + col0 + c * unit, unit);
            if ((MODE == PRISM_SCAN_DELTA || MODE == PRISM_SCAN_TOKEN) && lane < 2)  // beta (or dt), then g
                cp_async_f(dst + NV * dkp + a.colsp + lane, bg + t * 2 * a.H + (size_t)lane * a.H + h, 1);
            if (MODE == PRISM_SCAN_CHANNEL && lane == 0)                             // beta
                cp_async_f(dst + NV * dkp + a.colsp, bg + t * a.H + h, 1);
        }
        cp_async_commit();
    };
    auto finish = [&](int b0, int buf) {               // the block has landed: the decay from its exponent
        if (MODE == PRISM_SCAN_BONUS && !a.w_ready) {
            __syncwarp();
            decays_in_place(a, sm + (size_t)buf * TB * per_tok + 2 * dkp, per_tok, min(TB, qlen - b0), h);
        }
    };

    float S[R];
    float* st = a.state + (((size_t)a.slots[seg] * a.H + h) * dv + col) * dk;
    if (producer) {
        stage(0, 0);
        if (TB < qlen) stage(TB, 1);
        else cp_async_commit();
        cp_async_wait<1>();
        finish(0, 0);
    } else {
#pragma unroll
        for (int m = 0; m < Q; ++m) {
            const int i = 4 * (part + L * m);
            if (live && a.vec && i + 3 < dk) {
                const float4 v = *reinterpret_cast<const float4*>(st + i);
                S[4 * m] = v.x, S[4 * m + 1] = v.y, S[4 * m + 2] = v.z, S[4 * m + 3] = v.w;
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j) S[4 * m + j] = (live && i + j < dk) ? st[i + j] : 0.f;
            }
        }
    }
    __syncthreads();
    const float keep = MODE == PRISM_SCAN_RETAIN ? load_param(a.w0, a.w0_bf16, h) : 0.f;
    const float skip = MODE == PRISM_SCAN_TOKEN && a.w0 != nullptr ? load_param(a.w0, a.w0_bf16, h) : 0.f;

    int buf = 0;
    for (int b0 = 0; b0 < qlen; b0 += TB, buf = buf + 1 == NBUF ? 0 : buf + 1) {
        const int nb = min(TB, qlen - b0);
        if (producer) {
            // the block after the next goes into the buffer freed at the last barrier; the next one is seen in
            const int nxt = buf + 1 == NBUF ? 0 : buf + 1, nxt2 = nxt + 1 == NBUF ? 0 : nxt + 1;
            if (b0 + 2 * TB < qlen) stage(b0 + 2 * TB, nxt2);
            else cp_async_commit();
            cp_async_wait<1>();
            if (b0 + TB < qlen) finish(b0 + TB, nxt);
            __syncthreads();
            continue;
        }
        for (int tt = 0; tt < nb; ++tt) {
            const float* row = sm + ((size_t)buf * TB + tt) * per_tok + 4 * part;      // this thread's quads of q (or r); k, .. dkp further on
            const float* vv = row - 4 * part + NV * dkp;
            const float v = vv[lc];
            float o = 0.f;
            if (MODE == PRISM_SCAN_BONUS) {
                float b[4] = {0.f, 0.f, 0.f, 0.f}, c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int m = 0; m < Q; ++m) {
                    float q[4], k[4], w[4], u[4];
                    quad(row + 4 * L * m, q), quad(row + dkp + 4 * L * m, k), quad(row + 2 * dkp + 4 * L * m, w);
                    quad(ub + 4 * (part + L * m), u);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        float& s = S[4 * m + j];
                        b[j] = fmaf(__fmul_rn(q[j], u[j]), k[j], b[j]);
                        c[j] = fmaf(s, q[j], c[j]);
                        s = fmaf(w[j], s, __fmul_rn(k[j], v));
                    }
                }
                o = fmaf((b[0] + b[1]) + (b[2] + b[3]), v, (c[0] + c[1]) + (c[2] + c[3]));
            } else {
                // a column's sum against the state before the update: S^T k, or e^T S
                float u = 0.f, g = 1.f;
                constexpr bool DELTAS = MODE == PRISM_SCAN_DELTA || MODE == PRISM_SCAN_CHANNEL;
                if (DELTAS || MODE == PRISM_SCAN_GENERAL) {
                    float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                    for (int m = 0; m < Q; ++m) {
                        float k[4], w[4];
                        quad(row + (DELTAS ? 1 : 3) * dkp + 4 * L * m, k);
                        if (MODE == PRISM_SCAN_CHANNEL) quad(row + 2 * dkp + 4 * L * m, w);
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            float& s = S[4 * m + j];
                            if (MODE == PRISM_SCAN_CHANNEL) s = __fmul_rn(s, w[j]);
                            c[j] = fmaf(s, k[j], c[j]);
                        }
                    }
                    u = column_sum<L>((c[0] + c[1]) + (c[2] + c[3]));
                }
                if (MODE == PRISM_SCAN_DELTA) g = vv[a.colsp + 1];
                if (DELTAS) u = vv[a.colsp] * fmaf(-g, u, v);                          // what is written along k
                if (MODE == PRISM_SCAN_GENERAL) u = -u;
                if (MODE == PRISM_SCAN_RETAIN) g = keep, u = v;
                if (MODE == PRISM_SCAN_TOKEN) g = vv[a.colsp + 1], u = __fmul_rn(vv[a.colsp], v);
                if (MODE == PRISM_SCAN_GATED) u = v;
                float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int m = 0; m < Q; ++m) {
                    float q[4], k[4], w[4], e[4];
                    quad(row + 4 * L * m, q), quad(row + dkp + 4 * L * m, k);
                    if (MODE == PRISM_SCAN_GATED || MODE == PRISM_SCAN_GENERAL) quad(row + 2 * dkp + 4 * L * m, w);
                    if (MODE == PRISM_SCAN_GENERAL) quad(row + 4 * dkp + 4 * L * m, e);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        float& s = S[4 * m + j];
                        if (MODE == PRISM_SCAN_CHANNEL) s = fmaf(k[j], u, s);
                        else if (MODE == PRISM_SCAN_GENERAL) s = fmaf(k[j], v, fmaf(w[j], s, __fmul_rn(e[j], u)));
                        else s = fmaf(MODE == PRISM_SCAN_GATED ? w[j] : g, s, __fmul_rn(k[j], u));
                        c[j] = fmaf(s, q[j], c[j]);
                    }
                }
                o = (c[0] + c[1]) + (c[2] + c[3]);
            }
            o = column_sum<L>(o);
            if (MODE == PRISM_SCAN_TOKEN) o = fmaf(skip, v, o);
            if (live && part == 0) a.out[((size_t)(s0 + b0 + tt) * a.H + h) * dv + col] = o;
        }
        __syncthreads();                               // the next block has landed, and this buffer is free
    }
    if (live) {
#pragma unroll
        for (int m = 0; m < Q; ++m) {
            const int i = 4 * (part + L * m);
            if (a.vec && i + 3 < dk) {
                *reinterpret_cast<float4*>(st + i) = make_float4(S[4 * m], S[4 * m + 1], S[4 * m + 2], S[4 * m + 3]);
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (i + j < dk) st[i + j] = S[4 * m + j];
            }
        }
    }
}

// The scan of a step with many tokens a request.  GROUPS: eight tokens at a time (R 8 and 16), with the registers that their
// straight line code wants; else token by token.
template <int MODE, int R, int L, int CPT, bool GROUPS>
__global__ void __launch_bounds__(160, GROUPS ? 1 : (R == 32 ? 3 : 5)) scan_kernel(const ScanArgs a) {
    pdl_trigger();
    pdl_wait();
    extern __shared__ __align__(16) float sm[];
    constexpr int NV = scan_vectors(MODE);       // vectors over the key channels per token
    constexpr int Q = R / 4;                                   // quads of rows a thread owns
    const int h = blockIdx.x, seg = blockIdx.y, col0 = blockIdx.z * a.cols;
    const int s0 = a.seg_start[seg], qlen = a.seg_start[seg + 1] - s0;
    const int dk = a.dk, dv = a.dv, TB = a.TB;
    constexpr int dkp = L * R;                                 // the rows a column's threads cover; beyond dk: zeros
    const int ncols = min(a.cols, dv - col0);
    // The CTA's last warp brings the step's vectors in (and, for the decayed sum, turns the decay's exponent into
    // the decay); the warps before it own the state.  Their threads beyond the CTA's columns run along (they
    // take part in the shuffles) and neither load nor store.
    const int CT = blockDim.x - 32;
    const bool producer = (int)threadIdx.x >= CT;
    const int part = threadIdx.x % L;
    const bool live = !producer && (int)threadIdx.x / L * CPT < ncols;      // CPT > 1: the columns are whole groups of CPT
    const int lc = live ? threadIdx.x / L * CPT : 0, col = col0 + lc;
    const int kvh = h / a.rep;                         // DELTA: the q/k head this head uses
    // shared, per token of a block:  first[dkp] (q or r) | second[dkp] (k) | further vectors [dkp] | v[colsp] | 4 scalars
    const int per_tok = NV * dkp + a.colsp + 4;
    const int NBUF = a.NBUF;                           // blocks of tokens in shared memory: one in use, the others landed or on their way
    const float* x = pdl_fresh(a.x);
    const float* bg = pdl_fresh(a.bg);
    const float* ww = pdl_fresh(a.ww);
    const float* ex = pdl_fresh(a.ex);

    zero_padding(sm, NBUF * TB, per_tok, NV, dk, dkp, ncols, a.colsp);
    __syncthreads();

    // the producer warp asks for block b0 of the segment's tokens into buffer `buf`: the lanes are dealt out to the
    // pieces of a token's vectors, and where those are fewer than 32 to several tokens, so that a vector of a token
    // costs an instruction or less ...
    const int unit = a.vec ? 4 : 1;
    const int nk = (dk + unit - 1) / unit, nc = (ncols + unit - 1) / unit;          // pieces per vector
    const int lane = threadIdx.x & 31;
    const int ktoks = nk <= 16 ? 32 / nk : 1, ctoks = nc <= 16 ? 32 / nc : 1;        // tokens side by side
    const int kt = ktoks > 1 ? lane / nk : 0, kc = lane - kt * nk;
    const int ct = ctoks > 1 ? lane / nc : 0, cc = lane - ct * nc;
    const bool one_piece = a.vec && nk <= 32;          // a lane brings one piece of a vector at most
    const size_t head_q = (size_t)((MODE == PRISM_SCAN_DELTA || MODE == PRISM_SCAN_CHANNEL || MODE == PRISM_SCAN_TOKEN) ? kvh : h) * dk;
    auto stage = [&](int b0, int buf) {
        const int nb = min(TB, qlen - b0);
        float* dst0 = sm + (size_t)buf * TB * per_tok;
        const size_t t = (size_t)(s0 + b0 + kt);
        const float* xq = x + t * a.xs + head_q + a.qo + kc * unit;
        const float* xk = x + t * a.xs + head_q + a.ko + kc * unit;
        const float* wr = NV > 2 ? ww + t * a.ws + (size_t)h * dk + kc * unit : nullptr;
        const float* er = NV > 3 ? ex + t * a.es + (size_t)h * dk + kc * unit : nullptr;
        const size_t c_at = NV > 3 ? (size_t)a.H * dk : 0;                            // from the unit key to what it removes
        const size_t xstep = (size_t)ktoks * a.xs, wstep = (size_t)ktoks * a.ws, estep = (size_t)ktoks * a.es;
        float* dst = dst0 + (size_t)kt * per_tok + kc * unit;
        if (one_piece) {
            if (kt < ktoks && kc < nk)
#pragma unroll 4
                for (int tt = kt; tt < nb; tt += ktoks) {
                    cp_async_f(dst, xq, 4);
                    cp_async_f(dst + dkp, xk, 4);
                    if (NV > 2) cp_async_f(dst + 2 * dkp, wr, 4);
                    if (NV > 3) {
                        cp_async_f(dst + 3 * dkp, er, 4);
                        cp_async_f(dst + 4 * dkp, er + c_at, 4);
                        er += estep;
                    }
                    xq += xstep, xk += xstep;
                    if (NV > 2) wr += wstep;
                    dst += ktoks * per_tok;
                }
        } else if (kt < ktoks) {
            for (int tt = kt; tt < nb; tt += ktoks) {
                for (int c = 0; c + kc < nk; c += 32) {
                    cp_async_f(dst + c * unit, xq + c * unit, unit);
                    cp_async_f(dst + dkp + c * unit, xk + c * unit, unit);
                    if (NV > 2) cp_async_f(dst + 2 * dkp + c * unit, wr + c * unit, unit);
                    if (NV > 3) {
                        cp_async_f(dst + 3 * dkp + c * unit, er + c * unit, unit);
                        cp_async_f(dst + 4 * dkp + c * unit, er + c_at + c * unit, unit);
                    }
                }
                xq += xstep, xk += xstep;
                if (NV > 2) wr += wstep;
                if (NV > 3) er += estep;
                dst += ktoks * per_tok;
            }
        }
        if (ct < ctoks)
            for (int tt = ct; tt < nb; tt += ctoks)
                for (int c = cc; c < nc; c += 32)
                    cp_async_f(dst0 + (size_t)tt * per_tok + NV * dkp + c * unit,
                               x + (size_t)(s0 + b0 + tt) * a.xs + a.vo + (size_t)h * dv + col0 + c * unit, unit);
        for (int tt = lane; tt < nb; tt += 32) {
            float* sc = dst0 + (size_t)tt * per_tok + NV * dkp + a.colsp;
            const size_t ts = (size_t)(s0 + b0 + tt);
            if (MODE == PRISM_SCAN_DELTA || MODE == PRISM_SCAN_TOKEN) {              // beta (or dt), then g
                cp_async_f(sc, bg + ts * 2 * a.H + h, 1);
                cp_async_f(sc + 1, bg + ts * 2 * a.H + a.H + h, 1);
            }
            if (MODE == PRISM_SCAN_CHANNEL) cp_async_f(sc, bg + ts * a.H + h, 1);    // beta
        }
        cp_async_commit();
    };
    // ... and, once the copies of that block have landed (the caller has waited), turns the decay's exponent into the decay
    auto finish = [&](int b0, int buf) {
        if (MODE == PRISM_SCAN_BONUS && !a.w_ready) {
            __syncwarp();
            decays_in_place(a, sm + (size_t)buf * TB * per_tok + 2 * dkp, per_tok, min(TB, qlen - b0), h);
        }
    };

    uint64_t S[CPT][R / 2], bonus[MODE == PRISM_SCAN_BONUS ? R / 2 : 1];
    float* st = a.state + (((size_t)a.slots[seg] * a.H + h) * dv + col) * dk;
    if (producer) {
        for (int i = 0; i < NBUF - 1; ++i) {
            if (i * TB < qlen) stage(i * TB, i);
            else cp_async_commit();
        }
        cp_async_wait_upto(NBUF - 2);
        finish(0, 0);
    } else {
#pragma unroll
        for (int m = 0; m < Q; ++m) {
            const int i = 4 * (part + L * m);
#pragma unroll
            for (int p = 0; p < CPT; ++p) {
                const float* sp = st + (size_t)p * dk + i;
                if (live && a.vec && i + 3 < dk) {
                    const float4 v = *reinterpret_cast<const float4*>(sp);
                    S[p][2 * m] = pack2(v.x, v.y);
                    S[p][2 * m + 1] = pack2(v.z, v.w);
                } else {
                    float v[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) v[j] = (live && i + j < dk) ? sp[j] : 0.f;
                    S[p][2 * m] = pack2(v[0], v[1]);
                    S[p][2 * m + 1] = pack2(v[2], v[3]);
                }
            }
            if (MODE == PRISM_SCAN_BONUS) {
                float v[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) v[j] = i + j < dk ? load_param(a.u, a.u_bf16, (size_t)h * dk + i + j) : 0.f;
                bonus[2 * m % (R / 2)] = pack2(v[0], v[1]);
                bonus[(2 * m + 1) % (R / 2)] = pack2(v[2], v[3]);
            }
        }
    }
    __syncthreads();
    const float keep = MODE == PRISM_SCAN_RETAIN ? load_param(a.w0, a.w0_bf16, h) : 0.f;      // the head's constant decay
    const float skip = MODE == PRISM_SCAN_TOKEN && a.w0 != nullptr ? load_param(a.w0, a.w0_bf16, h) : 0.f;

    auto read = [&](const ulonglong2 (&q)[Q], float (&o)[CPT]) {
        if (MODE == PRISM_SCAN_BONUS) return;
#pragma unroll
        for (int p = 0; p < CPT; ++p) o[p] = quad_dot<Q>(S[p], q);
    };
    // One token, whose vectors lie at f1: S moves on, and q is what reads it out (`read`: this thread's part of column p),
    // or, for the decayed sum with a bonus, o is read out at once.  `before`: the read-out of the token before (last_q
    // into last_o) is still due; it stands where the chain waits for its shuffles.
    auto token = [&](const float* f1, ulonglong2 (&q)[Q], float (&o)[CPT], bool before, const ulonglong2 (&last_q)[Q], float (&last_o)[CPT]) {
        const float* row = f1 + 4 * part;
        const float* vv = f1 + NV * dkp;
        ulonglong2 k[Q];
        float v[CPT];
#pragma unroll
        for (int m = 0; m < Q; ++m) k[m] = quad(row + dkp + 4 * L * m);
#pragma unroll
        for (int m = 0; m < Q; ++m) q[m] = quad(row + 4 * L * m);
        if (CPT == 4) {
            const float4 v4 = *reinterpret_cast<const float4*>(vv + lc);
            v[0] = v4.x, v[1 % CPT] = v4.y, v[2 % CPT] = v4.z, v[3 % CPT] = v4.w;
        } else if (CPT == 2) {
            const float2 v2 = *reinterpret_cast<const float2*>(vv + lc);
            v[0] = v2.x, v[1 % CPT] = v2.y;
        } else {
            v[0] = vv[lc];
        }
        if (MODE == PRISM_SCAN_DELTA || MODE == PRISM_SCAN_CHANNEL) {
            const float beta = vv[a.colsp], g = MODE == PRISM_SCAN_DELTA ? vv[a.colsp + 1] : 1.f;
            if (MODE == PRISM_SCAN_CHANNEL) {
                if (before) read(last_q, last_o);      // S is about to decay
#pragma unroll
                for (int m = 0; m < Q; ++m) {
                    const ulonglong2 w = quad(row + 2 * dkp + 4 * L * m);
#pragma unroll
                    for (int p = 0; p < CPT; ++p) {
                        S[p][2 * m] = mul2(S[p][2 * m], w.x);
                        S[p][2 * m + 1] = mul2(S[p][2 * m + 1], w.y);
                    }
                }
            }
            const uint64_t g2 = pack2(g, g);
            float ks[CPT];
#pragma unroll
            for (int p = 0; p < CPT; ++p) ks[p] = quad_dot<Q>(S[p], k);
            if (MODE == PRISM_SCAN_DELTA && before) read(last_q, last_o);
#pragma unroll
            for (int p = 0; p < CPT; ++p) ks[p] = column_sum<L>(ks[p]);
#pragma unroll
            for (int p = 0; p < CPT; ++p) {
                const float uu = beta * fmaf(-g, ks[p], v[p]);
                const uint64_t u2 = pack2(uu, uu);
#pragma unroll
                for (int m = 0; m < Q; ++m) {
                    if (MODE == PRISM_SCAN_DELTA) {    // the small product is the rounded one, not the decayed state
                        S[p][2 * m] = mad2(S[p][2 * m], g2, mul2(k[m].x, u2));
                        S[p][2 * m + 1] = mad2(S[p][2 * m + 1], g2, mul2(k[m].y, u2));
                    } else {
                        fma2(S[p][2 * m], k[m].x, u2);
                        fma2(S[p][2 * m + 1], k[m].y, u2);
                    }
                }
            }
        } else if (MODE == PRISM_SCAN_GENERAL) {
            float es[CPT];                             // e^T S of a column, from the state before the token
            {
                ulonglong2 e[Q];
#pragma unroll
                for (int m = 0; m < Q; ++m) e[m] = quad(row + 3 * dkp + 4 * L * m);
#pragma unroll
                for (int p = 0; p < CPT; ++p) es[p] = quad_dot<Q>(S[p], e);
            }
            if (before) read(last_q, last_o);
#pragma unroll
            for (int p = 0; p < CPT; ++p) es[p] = column_sum<L>(es[p]);
#pragma unroll
            for (int m = 0; m < Q; ++m) {
                const ulonglong2 w = quad(row + 2 * dkp + 4 * L * m), c = quad(row + 4 * dkp + 4 * L * m);
#pragma unroll
                for (int p = 0; p < CPT; ++p) {
                    // what is removed is the rounded product: it is smaller than k v wherever c is, and rounding k v instead,
                    // ahead of the shuffles, leaves 3 % (slow decays) to 8 % (decays of 0.55 to 1) more error
                    const uint64_t v2 = pack2(v[p], v[p]), e2 = pack2(-es[p], -es[p]);
                    S[p][2 * m] = mad2(w.x, S[p][2 * m], mul2(c.x, e2));
                    S[p][2 * m + 1] = mad2(w.y, S[p][2 * m + 1], mul2(c.y, e2));
                    fma2(S[p][2 * m], k[m].x, v2);
                    fma2(S[p][2 * m + 1], k[m].y, v2);
                }
            }
        } else if (MODE == PRISM_SCAN_BONUS) {
            uint64_t b0 = 0, b1 = 0;
#pragma unroll
            for (int m = 0; m < Q; ++m) {
                fma2(b0, mul2(q[m].x, bonus[2 * m % (R / 2)]), k[m].x);
                fma2(b1, mul2(q[m].y, bonus[(2 * m + 1) % (R / 2)]), k[m].y);
            }
            const float2 p0 = unpack2(b0), p1 = unpack2(b1);
            const float now = (p0.x + p0.y) + (p1.x + p1.y);
#pragma unroll
            for (int p = 0; p < CPT; ++p) o[p] = fmaf(now, v[p], quad_dot<Q>(S[p], q));
#pragma unroll
            for (int m = 0; m < Q; ++m) {
                const ulonglong2 w = quad(row + 2 * dkp + 4 * L * m);
#pragma unroll
                for (int p = 0; p < CPT; ++p) {
                    const uint64_t v2 = pack2(v[p], v[p]);
                    S[p][2 * m] = mad2(w.x, S[p][2 * m], mul2(k[m].x, v2));
                    S[p][2 * m + 1] = mad2(w.y, S[p][2 * m + 1], mul2(k[m].y, v2));
                }
            }
        } else {                                       // S <- (decay) S + k v^T, read out after it
            const float dt = MODE == PRISM_SCAN_TOKEN ? vv[a.colsp] : 1.f;
            const float g = MODE == PRISM_SCAN_TOKEN ? vv[a.colsp + 1] : keep;
            const uint64_t g2 = pack2(g, g);
            if (before) read(last_q, last_o);
#pragma unroll
            for (int m = 0; m < Q; ++m) {
                ulonglong2 w = make_ulonglong2(g2, g2);
                if (MODE == PRISM_SCAN_GATED) w = quad(row + 2 * dkp + 4 * L * m);
#pragma unroll
                for (int p = 0; p < CPT; ++p) {
                    const float t = MODE == PRISM_SCAN_TOKEN ? __fmul_rn(dt, v[p]) : v[p];
                    const uint64_t v2 = pack2(t, t);
                    S[p][2 * m] = mad2(w.x, S[p][2 * m], mul2(k[m].x, v2));
                    S[p][2 * m + 1] = mad2(w.y, S[p][2 * m + 1], mul2(k[m].y, v2));
                }
            }
        }
    };
    // token tt of the segment, whose vectors lie at f1
    auto store = [&](int tt, const float* f1, float (&o)[CPT]) {
        float* dst = a.out + ((size_t)(s0 + tt) * a.H + h) * dv + col;
        if (MODE == PRISM_SCAN_TOKEN)
#pragma unroll
            for (int p = 0; p < CPT; ++p) o[p] = fmaf(skip, f1[NV * dkp + lc + p], o[p]);
        if (CPT == 4) *reinterpret_cast<float4*>(dst) = make_float4(o[0], o[1 % CPT], o[2 % CPT], o[3 % CPT]);
        else if (CPT == 2) *reinterpret_cast<float2*>(dst) = make_float2(o[0], o[1 % CPT]);
        else dst[0] = o[0];
    };

    int buf = 0;
    for (int b0 = 0; b0 < qlen; b0 += TB, buf = buf + 1 == NBUF ? 0 : buf + 1) {
        const int nb = min(TB, qlen - b0);
        if (producer) {
            // while block b0 is worked on: ask for the block that goes into the buffer freed at the last barrier, and
            // see the next one in
            const int nxt = buf + 1 == NBUF ? 0 : buf + 1, freed = buf == 0 ? NBUF - 1 : buf - 1;
            if (b0 + (NBUF - 1) * TB < qlen) stage(b0 + (NBUF - 1) * TB, freed);
            else cp_async_commit();
            cp_async_wait_upto(NBUF - 2);
            if (b0 + TB < qlen) finish(b0 + TB, nxt);
            __syncthreads();
            continue;
        }
        const float* blk = sm + (size_t)buf * TB * per_tok;
        int tt = 0;
        if constexpr (GROUPS) {                        // L is 8
            for (; tt + 8 <= nb; tt += 8) {
                float o[8][CPT];
                ulonglong2 q[2][Q];
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    token(blk + (size_t)(tt + i) * per_tok, q[i & 1], o[i], i > 0, q[(i + 1) & 1], o[(i + 7) & 7]);
                read(q[1], o[7]);
                // the eight tokens' sums over the eight lanes of a column, each lane ends with one token's: the same
                // pairs as column_sum's, half of the values a level
                float r[CPT];
#pragma unroll
                for (int p = 0; p < CPT; ++p) {
                    float h4[4], h2[2];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float mine = part & 4 ? o[i + 4][p] : o[i][p], other = part & 4 ? o[i][p] : o[i + 4][p];
                        h4[i] = mine + __shfl_xor_sync(0xffffffffu, other, 4);
                    }
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const float mine = part & 2 ? h4[i + 2] : h4[i], other = part & 2 ? h4[i] : h4[i + 2];
                        h2[i] = mine + __shfl_xor_sync(0xffffffffu, other, 2);
                    }
                    const float mine = part & 1 ? h2[1] : h2[0], other = part & 1 ? h2[0] : h2[1];
                    r[p] = mine + __shfl_xor_sync(0xffffffffu, other, 1);
                }
                if (live) store(b0 + tt + part, blk + (size_t)(tt + part) * per_tok, r);
            }
        }
        for (; tt < nb; ++tt) {
            float o[CPT];
            ulonglong2 q[Q];
            token(blk + (size_t)tt * per_tok, q, o, false, q, o);
            read(q, o);
#pragma unroll
            for (int p = 0; p < CPT; ++p) o[p] = column_sum<L>(o[p]);
            if (live && part == 0) store(b0 + tt, blk + (size_t)tt * per_tok, o);
        }
        __syncthreads();                               // the next block has landed, and this buffer is free
    }
    if (live) {
#pragma unroll
        for (int m = 0; m < Q; ++m) {
            const int i = 4 * (part + L * m);
#pragma unroll
            for (int p = 0; p < CPT; ++p) {
                float* sp = st + (size_t)p * dk + i;
                const float2 lo = unpack2(S[p][2 * m]), hi = unpack2(S[p][2 * m + 1]);
                if (a.vec && i + 3 < dk) {
                    *reinterpret_cast<float4*>(sp) = make_float4(lo.x, lo.y, hi.x, hi.y);
                } else {
                    const float v[4] = {lo.x, lo.y, hi.x, hi.y};
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (i + j < dk) sp[j] = v[j];
                }
            }
        }
    }
}

static int launch_scan(void (*kern)(const ScanArgs), const ScanArgs& a, int vectors, int cpt, int S, cudaStream_t stream) {
    const int per_tok = vectors * a.dkp + a.colsp + 4;
    const size_t smem = ((size_t)a.NBUF * a.TB * per_tok + (a.u != nullptr ? a.dkp : 0)) * sizeof(float);      // BONUS: + u
    if (smem > 200 * 1024) return (int)cudaErrorInvalidValue;
    open_smem(kern, smem);
    dim3 grid(a.H, S, (a.dv + a.cols - 1) / a.cols);
    return (int)launch_kernel(kern, grid, dim3((a.cols / cpt * a.L + 31) / 32 * 32 + 32), smem, stream, a);      // + the producer warp
}

}  // namespace prism

PRISM_EXPORT int prism_conv_unit_gates(const float* proj, long long ps, int ob, int oa, const void* taps, int taps_dtype,
                                       int K, const float* tail, const void* a_log, int a_log_dtype, const void* dt_bias,
                                       int dt_dtype, const int* tok_seg, const int* seg_start, const int* slots, int T, int G,
                                       int H, int dk, int dv, float unit_eps, float* qkv, float* bg, int move_tail,
                                       cudaStream_t stream) {
    if (T <= 0) return 0;
    if (K < 1 || G < 1 || H < 1 || dk < 1 || dv < 1) return (int)cudaErrorInvalidValue;
    const int C = 2 * G * dk + H * dv;
    const size_t smem = (size_t)C * sizeof(float);
    if (smem > 200 * 1024) return (int)cudaErrorInvalidValue;
    // Runs of tokens: a warp's sixteen tokens one after another take 8 to 12 us whatever else there is, so only where the other
    // kernel, bound by its T C channels, takes longer, and where the warps' lanes are not mostly idle (a head has 1, 2 or 4 entries a
    // lane).  Six heads of 128: 512 tokens 8.3 us and 11.9 in runs, 1,024 11.7 and 12.7, 2,048 19.1 and 16.8; 48 of 128: 256 tokens
    // 19.2 and 15.0; 16 of 64: 512 tokens 8.8 and 9.0, 1,024 11.8 and 10.6.
    const int widest = dk > dv ? dk : dv, per_lane = widest <= 32 ? 1 : widest <= 64 ? 2 : 4;
    if (!move_tail && K <= prism::CONV_TAPS && widest <= 128 && (long long)T * C >= (widest <= 64 ? 600000 : 1200000) &&
        (2 * G + H) * 32 * per_lane <= 2 * C) {
        const dim3 grid((T + prism::CONV_RUN - 1) / prism::CONV_RUN, (2 * G + H + 1 + 3) / 4);
        auto run = [&](auto kernel) {
            return (int)prism::launch_kernel(kernel, grid, dim3(128), 0, stream, proj, ps, ob, oa, taps, taps_dtype == PRISM_DTYPE_BF16, K,
                                             tail, a_log, a_log_dtype == PRISM_DTYPE_BF16, dt_bias, dt_dtype == PRISM_DTYPE_BF16, tok_seg,
                                             seg_start, slots, T, G, H, dk, dv, unit_eps, qkv, bg);
        };
        return per_lane == 1 ? run(prism::conv_unit_gates_run_kernel<1>) : per_lane == 2 ? run(prism::conv_unit_gates_run_kernel<2>)
                            : run(prism::conv_unit_gates_run_kernel<4>);
    }
    auto kern = prism::conv_unit_gates_kernel;
    prism::open_smem(kern, smem);
    const int threads = C >= 2048 ? 1024 : (C >= 512 ? 256 : 128);          // a few channels a thread: their loads are one chain each
    return (int)prism::launch_kernel(kern, dim3(T), dim3(threads), smem, stream, proj, ps, ob, oa, taps,
                                     taps_dtype == PRISM_DTYPE_BF16, K, tail, a_log, a_log_dtype == PRISM_DTYPE_BF16, dt_bias,
                                     dt_dtype == PRISM_DTYPE_BF16, tok_seg, seg_start, slots, G, H, dk, dv, unit_eps, qkv, bg,
                                     move_tail);
}

PRISM_EXPORT int prism_state_tail(const float* src, long long src_stride, int width, float* tail, int rows,
                                  const int* seg_start, const int* slots, int S, cudaStream_t stream) {
    if (S <= 0 || rows <= 0 || width <= 0) return 0;
    return (int)prism::launch_kernel(prism::state_tail_kernel, dim3(S), dim3(width >= 1024 ? 256 : 128), 0, stream, src,
                                     src_stride, width, tail, rows, seg_start, slots);
}

PRISM_EXPORT int prism_shift_mix(const float* x, int D, const float* prev, const void* mu, int mu_dtype, int n,
                                 const int* tok_seg, const int* seg_start, const int* slots, int T, void* out, int out_dtype,
                                 long long out_plane, int keep_prev, cudaStream_t stream) {
    if (T <= 0 || n <= 0) return 0;
    const int threads = D >= 2048 ? 1024 : (D >= 512 ? 256 : 128);
    const int mb = mu_dtype == PRISM_DTYPE_BF16;
    if (out_dtype == PRISM_DTYPE_BF16)
        return (int)prism::launch_kernel(prism::shift_mix_kernel<__nv_bfloat16>, dim3(T), dim3(threads), 0, stream, x, D, prev, mu,
                                         mb, n, tok_seg, seg_start, slots, (__nv_bfloat16*)out, out_plane, keep_prev);
    return (int)prism::launch_kernel(prism::shift_mix_kernel<float>, dim3(T), dim3(threads), 0, stream, x, D, prev, mu, mb, n,
                                     tok_seg, seg_start, slots, (float*)out, out_plane, keep_prev);
}

PRISM_EXPORT int prism_decay_from_exponent(float* w, long long w_stride, const void* w0, int w0_dtype, int T, int A,
                                           cudaStream_t stream) {
    if (T <= 0 || A <= 0) return 0;
    if (T > 65535) return (int)cudaErrorInvalidValue;
    return (int)prism::launch_kernel(prism::decay_from_exponent_kernel, dim3((A + 255) / 256, T), dim3(256), 0, stream, w,
                                     w_stride, w0, w0_dtype == PRISM_DTYPE_BF16, A);
}

// low [T, R] float32 (row stride free), w2t [R, N] float32, w0 [N] or null; out [T, N] float32; inner 1: tanh of low;
// epi PRISM_LR_*; alog [N / per] for PRISM_LR_SOFTPLUS; crate: the constant rate of PRISM_LR_EXPSIG.
PRISM_EXPORT int prism_lowrank_decay(const float* low, long long low_stride, int R, const float* w2t, const void* w0,
                                     int w0_dtype, int N, int T, float* out, long long out_stride, int inner, int epi,
                                     const void* alog, int alog_dtype, int per, float crate, cudaStream_t stream) {
    if (epi == PRISM_LR_SOFTPLUS && (alog == nullptr || per < 1)) return (int)cudaErrorInvalidValue;
    if (T <= 0 || N <= 0) return 0;
    const int tok = T <= 8 && R >= 16 ? 8 : 16, token_tiles = (T + tok - 1) / tok;
    const size_t smem = (size_t)tok * R * sizeof(float);
    if (R < 1 || (size_t)16 * R * sizeof(float) > 200 * 1024 || token_tiles > 65535) return (int)cudaErrorInvalidValue;
    auto kern = tok == 8 ? prism::lowrank_decay_kernel<8> : prism::lowrank_decay_kernel<16>;
    prism::open_smem(kern, smem);
    return (int)prism::launch_kernel(kern, dim3((N + 127) / 128, token_tiles), dim3(128), smem,
                                     stream, low, low_stride, R, w2t, w0, w0_dtype == PRISM_DTYPE_BF16, N, T, out, out_stride, inner, epi, alog,
                                     alog_dtype == PRISM_DTYPE_BF16, per < 1 ? 1 : per, crate);
}

// k, a [T, H dk] float32 column blocks with row stride ps; ab [H dk] or null; ex [T, 2 H dk] float32 out.
PRISM_EXPORT int prism_unit_removal(const float* k, const float* a, long long ps, const void* ab, int ab_dtype, float unit_eps,
                                    int T, int H, int dk, float* ex, cudaStream_t stream) {
    if (T <= 0 || H <= 0 || dk <= 0) return 0;
    const int warps = 4;
    const long long total = (long long)T * H;
    return (int)prism::launch_kernel(prism::unit_removal_kernel, dim3((unsigned)((total + warps - 1) / warps)), dim3(warps * 32), 0,
                                     stream, k, a, ps, ab, ab_dtype == PRISM_DTYPE_BF16, unit_eps, T, H, dk, ex);
}

// z [T, H] float32 (row stride zs); bias, a_log [H]; bg [T, 2 H] float32 out.
PRISM_EXPORT int prism_step_sizes(const float* z, long long zs, const void* bias, int bias_dtype, const void* a_log, int a_log_dtype,
                                  int T, int H, float* bg, cudaStream_t stream) {
    if (T <= 0 || H <= 0) return 0;
    const long long blocks = ((long long)T * H + 255) / 256;
    return (int)prism::launch_kernel(prism::step_sizes_kernel, dim3((unsigned)(blocks < 1184 ? blocks : 1184)), dim3(256), 0, stream, z, zs,
                                     bias, bias_dtype == PRISM_DTYPE_BF16, a_log, a_log_dtype == PRISM_DTYPE_BF16, T, H, bg);
}

// x [T, parts * w] float32 contiguous; gate [T, parts * w] float32 (row stride gs); weight [parts * w]; out [T, parts * w] of
// out_dtype (row stride os); before 1: the gate multiplies before the norm, 0: after it; sigmoid_act 1: sigmoid, 0: silu.
PRISM_EXPORT int prism_part_norm_gate(const float* x, const float* gate, long long gs, const void* weight, int weight_dtype, float eps,
                                      float scale, int T, int parts, int w, int before, int sigmoid_act, void* out, int out_dtype,
                                      long long os, cudaStream_t stream) {
    using namespace prism;
    if (T <= 0 || parts <= 0 || w <= 0) return 0;
    const size_t smem = (size_t)w * sizeof(float);
    if (parts > 65535 || smem > 200 * 1024) return (int)cudaErrorInvalidValue;
    const bool vec = w % 4 == 0 && gs % 4 == 0 && os % 4 == 0 && (uintptr_t)x % 16 == 0 && (uintptr_t)gate % 16 == 0 &&
                     (uintptr_t)out % (out_dtype == PRISM_DTYPE_BF16 ? 8 : 16) == 0;
    const int per = vec ? w / 4 : w;
    const int threads = per >= 1024 ? 512 : (per >= 256 ? 256 : (per >= 128 ? 128 : (per >= 64 ? 64 : 32)));
    const int wb = weight_dtype == PRISM_DTYPE_BF16;
#define PRISM_PN(TT, V)                                                                                                   \
    do {                                                                                                                  \
        auto kern = part_norm_gate_kernel<TT, V>;                                                                         \
        open_smem(kern, smem);                                                                                            \
        return (int)launch_kernel(kern, dim3(T, parts), dim3(threads), smem, stream, x, gate, gs, weight, wb, eps, scale, \
                                  parts, w, before, sigmoid_act, (TT*)out, os);                                           \
    } while (0)
    if (out_dtype == PRISM_DTYPE_BF16) {
        if (vec) PRISM_PN(__nv_bfloat16, 4);
        PRISM_PN(__nv_bfloat16, 1);
    }
    if (vec) PRISM_PN(float, 4);
    PRISM_PN(float, 1);
#undef PRISM_PN
}

PRISM_EXPORT int prism_headnorm_gate(const float* o, const float* gate, long long gate_stride, const void* weight,
                                     int weight_dtype, int per_head_weight, float eps, float scale, int T, int H, int dv,
                                     void* out, int out_dtype, long long out_stride, int gate_sigmoid, cudaStream_t stream) {
    if (T <= 0 || H <= 0 || dv <= 0) return 0;
    const int warps = 4;
    const long long total = (long long)T * H;
    const int blocks = (int)((total + warps - 1) / warps);
    const int wb = weight_dtype == PRISM_DTYPE_BF16;
    if (out_dtype == PRISM_DTYPE_BF16)
        return (int)prism::launch_kernel(prism::headnorm_gate_kernel<__nv_bfloat16>, dim3(blocks), dim3(warps * 32), 0, stream, o,
                                         gate, gate_stride, weight, wb, per_head_weight, eps, scale, T, H, dv,
                                         (__nv_bfloat16*)out, out_stride, gate_sigmoid);
    return (int)prism::launch_kernel(prism::headnorm_gate_kernel<float>, dim3(blocks), dim3(warps * 32), 0, stream, o, gate,
                                     gate_stride, weight, wb, per_head_weight, eps, scale, T, H, dv, (float*)out, out_stride, gate_sigmoid);
}

// mode PRISM_SCAN_*; state [slots, H, dv, dk] float32; out [T, H, dv] float32; rep: heads per q/k head (DELTA).
// Returns cudaErrorInvalidValue for dk > 1024.
PRISM_EXPORT int prism_recurrent_scan(int mode, const float* x, long long x_stride, long long qo, long long ko, long long vo,
                                      const float* bg,
                                      const float* ww, long long ww_stride, const void* w0, int w0_dtype, const void* u,
                                      int u_dtype, float* state, const int* seg_start, const int* slots, int S, int T, int max_q_len,
                                      int H, int rep, int dk, int dv, float* out, int w_ready, const float* ex,
                                      long long ex_stride, cudaStream_t stream) {
    using namespace prism;
    if (S <= 0) return 0;
    if (H < 1 || rep < 1 || dk < 1 || dv < 1 || dk > 1024 || S > 65535) return (int)cudaErrorInvalidValue;
    ScanArgs a;
    a.x = x; a.xs = x_stride; a.qo = qo; a.ko = ko; a.vo = vo; a.bg = bg; a.ww = ww; a.ws = ww_stride;
    a.w0 = w0; a.w0_bf16 = w0_dtype == PRISM_DTYPE_BF16; a.u = u; a.u_bf16 = u_dtype == PRISM_DTYPE_BF16;
    a.state = state; a.seg_start = seg_start; a.slots = slots; a.out = out; a.H = H; a.rep = rep; a.dk = dk; a.dv = dv;
    a.w_ready = w_ready;
    a.ex = ex; a.es = ex_stride;
    if (mode == PRISM_SCAN_RETAIN && (w0 == nullptr || rep != 1)) return (int)cudaErrorInvalidValue;
    if (mode == PRISM_SCAN_GENERAL && (ex == nullptr || ww == nullptr || rep != 1)) return (int)cudaErrorInvalidValue;
    if ((mode == PRISM_SCAN_TOKEN && bg == nullptr) || (mode == PRISM_SCAN_GATED && (ww == nullptr || rep != 1))) return (int)cudaErrorInvalidValue;
    const int R = dk <= 32 ? 4 : (dk <= 64 ? 8 : (dk <= 128 ? 16 : 32));
    int L = 1;
    while (L * R < dk) L *= 2;                          // at most 32
    if (R >= 8 && L < 8) L = 8;                        // the compiled pairs: more than 32 rows always take eight threads a column
    a.L = L;
    a.dkp = L * R;                                     // the rows the threads of a column cover; beyond dk: zeros
    const bool quads = dk % 4 == 0 && dv % 4 == 0 && x_stride % 4 == 0 && qo % 4 == 0 && ko % 4 == 0 && vo % 4 == 0 &&
                       (uintptr_t)x % 16 == 0 && (uintptr_t)state % 16 == 0 && (uintptr_t)out % 16 == 0 &&
                       (scan_vectors(mode) == 2 || (ww_stride % 4 == 0 && (uintptr_t)ww % 16 == 0)) &&
                       (mode != PRISM_SCAN_GENERAL || (ex_stride % 4 == 0 && (uintptr_t)ex % 16 == 0 && ((long long)H * dk) % 4 == 0));
    // Columns a CTA: the fewest of 4 to 64 whose CTAs fit the 148 SMs once, since a second CTA on an SM shares its
    // schedulers and shared memory while the chain of tokens takes as long (2,048 tokens, delta rule, 16 heads of 128:
    // 16 columns 296 us, 8 columns on two CTAs an SM 346 us; 32 heads: 32 columns 370 us, 16 columns 587 us).  More than
    // 4 x 4 of them give a thread several, so that the token's vectors are read fewer times.  The modes with three
    // vectors and more do better where each warp has twice the columns a thread and a CTA of its own (2,048 columns,
    // general, 1,024 tokens: 212 us, 16 columns as four warps 230 us; bonus, 2,048 tokens: 178 and 255 us), the others
    // not (delta: 330 and 296 us).  A few tokens a request are bound by the state's way in and out: one column a thread.
    int cpt = 1, threads = 128;
    auto ctas = [&](int cols) { return (long long)H * S * ((dv + cols - 1) / cols); };
    // Many tokens: requests of more than 16 on average, or one whose chain of tokens (some 0.2 us each are gained) is worth more
    // than the states of all of them lose in few and heavy CTAs.  16 heads of 128 x 128, delta rule, by the two kernels: 512
    // tokens beside 32 single ones 284 and 190 us, 40 beside 63 58 and 112 us.  States of 50 MB and more stream from HBM and want more
    // CTAs where two vectors a token leave little else to do (64 requests of 17 tokens, 48 heads: retain 452 and 575 us, gated 660
    // and 610).  Beyond 128 rows only five vectors a token are worth it (8 heads of 256 x 256, general: 512 tokens 363 and 291 us,
    // 64 requests of 17 450 and 570; delta, 16 requests of 64: 224 and 294).
    const long long states = (long long)S * H * dk * dv;
    const bool many = quads && max_q_len >= 16 &&
                      (R == 32 ? scan_vectors(mode) == 5 && 30000LL * max_q_len > states
                               : T > (scan_vectors(mode) == 2 && states > 12000000 ? 32LL : 16LL) * S || 80000LL * max_q_len > states);
    const bool groups = many && (R == 8 || R == 16);
    if (groups) {
        int want = 4;
        while (want < 64 && ctas(want) > 148) want *= 2;
        cpt = want <= 16 ? 1 : (want == 32 ? 2 : 4);
        if (scan_vectors(mode) > 2 && (want == 16 || want == 32)) cpt *= 2, want /= 2;
        threads = want / cpt * L;
    } else {
        while (threads > 32 && ctas(threads / L) < 148) threads /= 2;
    }
    int cols = threads / L < 1 ? 1 : threads / L * cpt;
    if (cols > dv) cols = dv;
    if (cols >= 4) cols = cols / 4 * 4;
    a.cols = cols;
    a.colsp = (cols + 3) / 4 * 4;
    a.vec = quads && cols % 4 == 0;
    const int per_tok = scan_vectors(mode) * a.dkp + a.colsp + 4;
    int tb = (24 * 1024 / 4) / per_tok;
    tb = tb < 1 ? 1 : (tb >= 16 ? 16 : (many && tb >= 8 ? 8 : tb));
    a.TB = tb > max_q_len ? (max_q_len < 1 ? 1 : max_q_len) : tb;      // a decode step stages one token, and CTAs are small
    a.NBUF = SCAN_STEP_BLOCKS;
    if (many) {
        // blocks on their way cover the latency of memory at some 100 ns a token; 100 KB leave room for two CTAs an SM
        const int blocks = (max_q_len + a.TB - 1) / a.TB;
        // (up to 32 rows a CTA is small, and where several share an SM the others cover it)
        a.NBUF = (R == 4 && ctas(cols) > 296 ? 36 : 100) * 1024 / (a.TB * per_tok * 4);
        a.NBUF = a.NBUF > 8 ? 8 : a.NBUF;
        if (a.NBUF > blocks + 1) a.NBUF = blocks + 1;
        if (a.NBUF < 3) a.NBUF = 3;
    }
    // rows a thread and threads a column, both known to the compiler: (4, 1..8) up to 32 rows, (8, 8), (16, 8), (32, 8..32)
#define PRISM_SCAN_GO(K) return launch_scan(K, a, scan_vectors(mode), cpt, S, stream)
#define PRISM_SCAN_EIGHT(M, RR)                                                                      \
    do {                                                                                             \
        if (!groups) PRISM_SCAN_GO((scan_step_kernel<M, RR, 8>));                                    \
        if (cpt == 4) PRISM_SCAN_GO((scan_kernel<M, RR, 8, 4, true>));                               \
        if (cpt == 2) PRISM_SCAN_GO((scan_kernel<M, RR, 8, 2, true>));                               \
        PRISM_SCAN_GO((scan_kernel<M, RR, 8, 1, true>));                                             \
    } while (0)
#define PRISM_SCAN_ONE(M, RR, LL)                                                                    \
    do {                                                                                             \
        if constexpr (RR == 4 || scan_vectors(M) == 5)                                               \
            if (many) PRISM_SCAN_GO((scan_kernel<M, RR, LL, 1, false>));                             \
        PRISM_SCAN_GO((scan_step_kernel<M, RR, LL>));                                                \
    } while (0)
#define PRISM_SCAN(M)                                                                                \
    do {                                                                                             \
        if (R == 8) PRISM_SCAN_EIGHT(M, 8);                                                          \
        if (R == 16) PRISM_SCAN_EIGHT(M, 16);                                                        \
        if (R == 4 && L == 1) PRISM_SCAN_ONE(M, 4, 1);                                               \
        if (R == 4 && L == 2) PRISM_SCAN_ONE(M, 4, 2);                                               \
        if (R == 4 && L == 4) PRISM_SCAN_ONE(M, 4, 4);                                               \
        if (R == 4) PRISM_SCAN_ONE(M, 4, 8);                                                         \
        if (L == 8) PRISM_SCAN_ONE(M, 32, 8);                                                        \
        if (L == 16) PRISM_SCAN_ONE(M, 32, 16);                                                      \
        PRISM_SCAN_ONE(M, 32, 32);                                                                   \
    } while (0)
    if (mode == PRISM_SCAN_DELTA) PRISM_SCAN(PRISM_SCAN_DELTA);
    if (mode == PRISM_SCAN_BONUS) PRISM_SCAN(PRISM_SCAN_BONUS);
    if (mode == PRISM_SCAN_CHANNEL) PRISM_SCAN(PRISM_SCAN_CHANNEL);
    if (mode == PRISM_SCAN_GENERAL) PRISM_SCAN(PRISM_SCAN_GENERAL);
    if (mode == PRISM_SCAN_RETAIN) PRISM_SCAN(PRISM_SCAN_RETAIN);
    if (mode == PRISM_SCAN_TOKEN) PRISM_SCAN(PRISM_SCAN_TOKEN);
    if (mode == PRISM_SCAN_GATED) PRISM_SCAN(PRISM_SCAN_GATED);
#undef PRISM_SCAN
#undef PRISM_SCAN_ONE
#undef PRISM_SCAN_EIGHT
#undef PRISM_SCAN_GO
    return (int)cudaErrorInvalidValue;
}
