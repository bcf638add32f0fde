// True float32 matrix product for the 32-bit path:  C = A @ W^T (+ bias),
// A [M, K] row-major, W [N, K] row-major (the [out, in] layout of the model
// file, andre-fu/prism engine/weight_pool.py:46-70; F.linear at
// engine/executor.py:109,122,125,127,130).  CUDA-core FFMA only: no tensor
// cores, no TF32.
//
// Every kernel here adds an output's products in one order, which depends on
// K alone: K is cut into slices of 32, slice c belongs to class c % 8, a class
// is one chain of fused multiply-adds over its slices in ascending order, and
// the eight classes' sums are added in ascending order.  So a value does not
// depend on M, on the row's place in the batch, on the grid or on the kernel,
// and a product can still be spread over eight threads (few rows: the lanes of
// one warp) or eight CTAs (few tiles: a cluster) where one chain per output
// would leave the GPU idle.
//
// Few rows (M <= 16) are bound by the stream of weights: measured at 3 rows, K 896, N 151,936 (545 MB) 2.4 ms with one tile
// kernel for every M, 0.09 ms here.
#include "f32x2.cuh"

namespace prism {
namespace f32gemm {

constexpr int SLICE = 32, CLASSES = 8, PERIOD = SLICE * CLASSES;
constexpr int FEW_WARPS = 8;                  // of a CTA that takes few rows, at most

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// `bytes` of the 16 (of the 4) are copied, the rest of the destination becomes zero
__device__ __forceinline__ void copy16(uint32_t dst, const float* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copy4(uint32_t dst, const float* src, int bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

// ---- few rows, a ring a CTA ------------------------------------------------------------------------------
// A CTA owns BN weight rows and all M <= MT rows of A and walks K in periods of 256 through a ring of shared memory stages that both
// go through, so that W is read once at any K (cp.async; the weights of the first stages are brought into L2 before the dependency
// wait: read they are after it, so that they may also be what an earlier kernel of the stream writes).  Thread =
// (class, column group): the eight classes of a column are eight neighbouring lanes.  A row's 16-byte pieces lie
// at (class, piece ^ class), so that the eight lanes read eight different bank groups.
// BN 8 where N is small (bound by latency: N 896 is 112 CTAs of two warps), else 32 with two columns a thread, which halves the
// reads of A.
template <int MT, int BN, int CPT, int STAGES, bool VEC>
__global__ void __launch_bounds__(BN / CPT * CLASSES)
shared_ring_kernel(const float* A, int lda, const float* W, int ldw, const void* __restrict__ bias,
                   int bias_bf16, float* C, int ldc, int M, int N, int K) {
    constexpr int THREADS = BN / CPT * CLASSES;
    constexpr int STAGE = (BN + MT) * PERIOD;
    extern __shared__ __align__(16) float smem[];
    const int tid = threadIdx.x, j = tid % CLASSES, cg = tid / CLASSES;
    const int n0 = blockIdx.x * BN;
    const int periods = (K + PERIOD - 1) / PERIOD;

    auto load = [&](const float* src, int ld, int rows, int limit, int row0, int period, float* dst) {
        // rows x 64 pieces of 16 bytes
        for (int idx = tid; idx < rows * (PERIOD / 4); idx += THREADS) {
            const int r = idx / (PERIOD / 4), piece = idx % (PERIOD / 4);
            const int cls = piece / 8, at = cls * 8 + ((piece % 8) ^ cls);
            const int k = period * PERIOD + piece * 4;
            const uint32_t d = smem_addr(dst + r * PERIOD + at * 4);
            const int have = row0 + r < limit ? min(max(K - k, 0), 4) : 0;
            const float* s = have ? src + (size_t)(row0 + r) * ld + k : src;
            if (VEC) {
                copy16(d, s, have * 4);
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e) copy4(d + 4 * e, e < have ? s + e : src, e < have ? 4 : 0);
            }
        }
    };

    pdl_trigger();
    // lines of 128 bytes: eight of a row a period
    for (int idx = tid; idx < BN * 8 * (STAGES - 1); idx += THREADS) {
        const int r = idx / (8 * (STAGES - 1)), k = idx % (8 * (STAGES - 1)) * 32;
        if (n0 + r < N && k < K) asm volatile("prefetch.global.L2 [%0];" ::"l"(W + (size_t)(n0 + r) * ldw + k));
    }
    pdl_wait();
    W = pdl_fresh(W), A = pdl_fresh(A);
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < periods) {
            load(W, ldw, BN, N, n0, s, smem + s * STAGE);
            load(A, lda, MT, M, 0, s, smem + s * STAGE + BN * PERIOD);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }

    float acc[MT][CPT];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int p = 0; p < CPT; ++p) acc[m][p] = 0.f;

    for (int t = 0; t < periods; ++t) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncthreads();
        const int next = t + STAGES - 1;
        if (next < periods) {
            float* st = smem + (next % STAGES) * STAGE;
            load(W, ldw, BN, N, n0, next, st);
            load(A, lda, MT, M, 0, next, st + BN * PERIOD);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float4* ws = reinterpret_cast<const float4*>(smem + (t % STAGES) * STAGE);
        const float4* xs = ws + BN * (PERIOD / 4);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int at = j * 8 + (i ^ j);
            float4 w[CPT];
#pragma unroll
            for (int p = 0; p < CPT; ++p) w[p] = ws[(cg + p * (BN / CPT)) * (PERIOD / 4) + at];
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                const float4 x = xs[m * (PERIOD / 4) + at];
#pragma unroll
                for (int p = 0; p < CPT; ++p) {
                    acc[m][p] = fmaf(x.x, w[p].x, acc[m][p]);
                    acc[m][p] = fmaf(x.y, w[p].y, acc[m][p]);
                    acc[m][p] = fmaf(x.z, w[p].z, acc[m][p]);
                    acc[m][p] = fmaf(x.w, w[p].w, acc[m][p]);
                }
            }
        }
    }
#pragma unroll
    for (int m = 0; m < MT; ++m) {
#pragma unroll
        for (int p = 0; p < CPT; ++p) {
            float v = __shfl_sync(0xffffffffu, acc[m][p], 0, CLASSES);
#pragma unroll
            for (int c = 1; c < CLASSES; ++c) v += __shfl_sync(0xffffffffu, acc[m][p], c, CLASSES);
            const int n = n0 + cg + p * (BN / CPT);
            if ((m * CPT + p) % CLASSES == j && m < M && n < N) {
                if (bias != nullptr) v += load_param(bias, bias_bf16, n);
                C[(size_t)m * ldc + n] = v;
            }
        }
    }
}

// all but the newest `stages - 1` groups (2 to 8 stages) have landed
__device__ __forceinline__ void few_wait(int stages) {
    switch (stages) {
        case 2: asm volatile("cp.async.wait_group 1;" ::: "memory"); break;
        case 3: asm volatile("cp.async.wait_group 2;" ::: "memory"); break;
        case 4: asm volatile("cp.async.wait_group 3;" ::: "memory"); break;
        case 5: asm volatile("cp.async.wait_group 4;" ::: "memory"); break;
        case 6: asm volatile("cp.async.wait_group 5;" ::: "memory"); break;
        case 7: asm volatile("cp.async.wait_group 6;" ::: "memory"); break;
        default: asm volatile("cp.async.wait_group 7;" ::: "memory"); break;
    }
}

// ---- few rows -----------------------------------------------------------------------------------------
// Bound by the stream of weights.  A warp takes 4 CPT columns at a time and walks their K in periods of 256 through a
// ring of its own (cp.async), straight on into the first periods of its next columns; no warp waits for another.  A CTA has a
// contiguous share of the columns, even to 4 CPT of them over the SMs, and keeps its rows of A whole in shared memory
// (XRES; a K too long for that sends them through the rings too).  Lane = (class, column): the eight classes of a column
// are eight neighbouring lanes.  A row's 16-byte pieces lie at (class, piece ^ class), so that the eight lanes read eight
// different bank groups.  The weights of the first stages are brought into L2 before the dependency wait; read they are after
// it, so that they may also be what an earlier kernel of the stream writes.  (One CTA an SM by its shared memory: told so, the compiler takes 69
// to 255 registers; left alone it kept to 64 and spilled, three rows of K 4,864 to N 896 15.7 us against 11.2.)
template <int MT, int CPT, bool VEC, bool XRES>
__global__ void __launch_bounds__(FEW_WARPS * 32, 1)
few_rows_kernel(const float* A, int lda, const float* W, int ldw, const void* __restrict__ bias,
                int bias_bf16, float* C, int ldc, int M, int N, int K, int stages) {
    constexpr int COLS = 4 * CPT, ROWS = COLS + (XRES ? 0 : MT);     // rows of a stage
    extern __shared__ __align__(16) float smem[];
    const int lane = threadIdx.x % 32, warp = threadIdx.x / 32, warps = blockDim.x / 32, j = lane % CLASSES, cg = lane / CLASSES;
    const int m0 = blockIdx.y * MT;
    const int periods = (K + PERIOD - 1) / PERIOD, mrows = min(MT, M - m0);
    const int groups = (N + COLS - 1) / COLS;
    const int g1 = (int)((long long)groups * (blockIdx.x + 1) / gridDim.x);
    const int g0 = (int)((long long)groups * blockIdx.x / gridDim.x) + warp;     // then every `warps`-th
    const int mine = g0 < g1 ? (g1 - g0 + warps - 1) / warps : 0;
    float* ring = smem + (XRES ? (size_t)periods * mrows * PERIOD : 0) + (size_t)warp * stages * ROWS * PERIOD;

    // the 64 pieces of a row's period, two a lane; the place of piece p
    auto place = [](int p) { return (p / 8) * 8 + ((p % 8) ^ (p / 8)); };
    const int at0 = place(lane) * 4, at1 = place(lane + 32) * 4;
    auto bring = [&](const float* row, int k, bool live, uint32_t d) {
        const int have = live ? min(max(K - k, 0), 4) : 0;
        const float* s = have ? row + k : row;
        if (VEC) {
            copy16(d, s, have * 4);
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) copy4(d + 4 * e, e < have ? s + e : row, e < have ? 4 : 0);
        }
    };
    auto bring_row = [&](const float* row, int k, bool live, float* dst) {
        bring(row, k + lane * 4, live, smem_addr(dst + at0));
        bring(row, k + (lane + 32) * 4, live, smem_addr(dst + at1));
    };
    int lg = g0, lt = 0, ls = 0, left = mine * periods;       // the next period to ask for and the stage it goes to
    auto ask = [&]() {
        if (left > 0) {
            float* dst = ring + (size_t)ls * ROWS * PERIOD;
            const int k = lt * PERIOD;
            if (VEC && k + PERIOD <= K && (lg + 1) * COLS <= N) {
                const float* s = W + (size_t)lg * COLS * ldw + k + lane * 4;
                const uint32_t d0 = smem_addr(dst + at0), d1 = smem_addr(dst + at1);
#pragma unroll
                for (int c = 0; c < COLS; ++c, s += ldw) {
                    copy16(d0 + c * PERIOD * 4, s, 16);
                    copy16(d1 + c * PERIOD * 4, s + 128, 16);
                }
            } else {
#pragma unroll 1
                for (int c = 0; c < COLS; ++c) {
                    const int n = lg * COLS + c;
                    bring_row(W + (size_t)min(n, N - 1) * ldw, k, n < N, dst + c * PERIOD);
                }
            }
            if (!XRES) {
#pragma unroll 1
                for (int m = 0; m < mrows; ++m) bring_row(A + (size_t)(m0 + m) * lda, k, true, dst + (COLS + m) * PERIOD);
            }
            if (++lt == periods) lt = 0, lg += warps;
            if (++ls == stages) ls = 0;
            --left;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    pdl_trigger();
    // lines of 128 bytes: eight of a row a period
    for (int idx = lane; idx < COLS * 8 * stages; idx += 32) {
        const int n = g0 * COLS + idx % COLS, k = idx / COLS * 32;
        if (mine && n < N && k < K) asm volatile("prefetch.global.L2 [%0];" ::"l"(W + (size_t)n * ldw + k));
    }
    pdl_wait();
    W = pdl_fresh(W), A = pdl_fresh(A);
    if (XRES) {                                       // lands with the first stage's group
        for (int idx = warp; idx < periods * mrows; idx += warps) {
            const int t = idx / mrows, m = idx - t * mrows;
            bring_row(A + (size_t)(m0 + m) * lda, t * PERIOD, true, smem + (size_t)idx * PERIOD);
        }
    }
    for (int s = 0; s < stages; ++s) ask();
    if (XRES) {
        few_wait(stages);
        __syncthreads();
    }

    int stage = 0;
    for (int g = g0; g < g1; g += warps) {
        float acc[MT][CPT];
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int p = 0; p < CPT; ++p) acc[m][p] = 0.f;
        for (int t = 0; t < periods; ++t) {
            few_wait(stages);
            __syncwarp();
            const float4* ws = reinterpret_cast<const float4*>(ring + (size_t)stage * ROWS * PERIOD);
            const float4* xs = XRES ? reinterpret_cast<const float4*>(smem + (size_t)t * mrows * PERIOD) : ws + COLS * (PERIOD / 4);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int at = j * 8 + (i ^ j);
                float4 w[CPT];
#pragma unroll
                for (int p = 0; p < CPT; ++p) w[p] = ws[(cg + 4 * p) * (PERIOD / 4) + at];
#pragma unroll
                for (int m = 0; m < MT; ++m) {
                    const float4 x = xs[(MT <= 4 ? m : min(m, mrows - 1)) * (PERIOD / 4) + at];
#pragma unroll
                    for (int p = 0; p < CPT; ++p) {
                        acc[m][p] = fmaf(x.x, w[p].x, acc[m][p]);
                        acc[m][p] = fmaf(x.y, w[p].y, acc[m][p]);
                        acc[m][p] = fmaf(x.z, w[p].z, acc[m][p]);
                        acc[m][p] = fmaf(x.w, w[p].w, acc[m][p]);
                    }
                }
            }
            __syncwarp();
            ask();                                    // into the stage that was just read
            if (++stage == stages) stage = 0;
        }
        // the classes' sums in ascending order; eight outputs at a time, lane j of a column ends with output j
        constexpr int OUT = MT * CPT;
#pragma unroll
        for (int o0 = 0; o0 < OUT; o0 += 8) {
            float v[8];
#pragma unroll
            for (int o = 0; o < 8; ++o) v[o] = o0 + o < OUT ? acc[(o0 + o < OUT ? o0 + o : 0) / CPT][(o0 + o) % CPT] : 0.f;
#pragma unroll
            for (int s = 4; s; s /= 2)
#pragma unroll
                for (int o = 0; o < 8; ++o)
                    if (!(o & s)) {
                        const bool up = j & s;
                        const float got = __shfl_xor_sync(0xffffffffu, up ? v[o] : v[o | s], s);
                        if (up) v[o] = got;
                        else v[o | s] = got;
                    }
            float sum = v[0];
#pragma unroll
            for (int c = 1; c < CLASSES; ++c) sum += v[c];
            const int o = o0 + j, m = o / CPT, n = g * COLS + cg + 4 * (o % CPT);
            if (o < OUT && m < mrows && n < N) {
                if (bias != nullptr) sum += load_param(bias, bias_bf16, n);
                C[(size_t)(m0 + m) * ldc + n] = sum;
            }
        }
    }
}

// ---- many rows --------------------------------------------------------------------------------------
// BM x BN outputs a CTA, TM x TN a thread, a slice of K or half of one a step (the next one on its way in registers), the
// multiply-adds in pairs of rows (fma.rn.f32x2).  Neighbouring lanes bring the neighbouring bytes of a row, and what they
// store transposed lies at row ^ TURN (k / 4), so that a warp's stores meet no bank twice and rows stay together in fours.
// (Lanes that brought a row each took 32 half-used sectors a load: 252 rows, N 9,728, K 896 193 us, now 130; the
// multiply-adds alone would take 61.  A 128-bit load from shared memory keeps the SM's path to the registers busy for four cycles
// whatever its lanes share, so the loads weigh nearly as much as the multiply-adds; a second copy of W with its columns swapped
// instead of the two moves a column took 164 us, 8 x 8 outputs a thread 136: fewer loads, but half the warps to cover them.)
// SPLIT: the eight classes of a tile are the eight CTAs of a cluster, whose sums meet through distributed shared memory.
template <int BM, int BN, int STEP, bool SPLIT> constexpr int many_smem() { return (2 * STEP * (BM + BN) + (SPLIT ? BM * BN : 0)) * 4; }

template <int BM, int BN, int TM, int TN, int STEP, bool SPLIT, bool VEC>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
many_rows_kernel(const float* A, int lda, const float* W, int ldw, const void* __restrict__ bias,
                 int bias_bf16, float* C, int ldc, int M, int N, int K) {
    constexpr int THREADS = (BM / TM) * (BN / TN), OWN = SPLIT ? 1 : CLASSES;       // classes of this CTA
    constexpr int P = STEP / 4, TURN = 32 / P;                       // 16-byte pieces of a row a step
    constexpr int LA = BM * P / THREADS, LW = BN * P / THREADS;      // pieces a thread brings
    static_assert(BM % 32 == 0 && BN % 32 == 0 && TM % 4 == 0 && TN % 4 == 0 && LA * THREADS == BM * P && LW * THREADS == BN * P &&
                  (STEP == SLICE || STEP == SLICE / 2), "");
    extern __shared__ __align__(16) float smem[];
    float* as = smem;                              // [2][STEP][BM]
    float* ws = smem + 2 * STEP * BM;              // [2][STEP][BN]
    float* sums = ws + 2 * STEP * BN;              // [BM][BN] of a split tile
    const int tid = threadIdx.x, tx = tid % (BN / TN), ty = tid / (BN / TN);
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int slices = (K + SLICE - 1) / SLICE;
    const int first = SPLIT ? (int)blockIdx.z : 0;                  // a cluster is (1, 1, 8): its rank is the class

    pdl_trigger();
    pdl_wait();
    A = pdl_fresh(A);
    W = pdl_fresh(W);

    float4 ra[LA], rw[LW];
    auto piece = [&](const float* src, int ld, int row, int limit, int k) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row < limit && k < K) {
            const float* s = src + (size_t)row * ld + k;
            if (VEC && k + 4 <= K) {
                v = *reinterpret_cast<const float4*>(s);
            } else {
                v.x = s[0];
                if (k + 1 < K) v.y = s[1];
                if (k + 2 < K) v.z = s[2];
                if (k + 3 < K) v.w = s[3];
            }
        }
        return v;
    };
    auto fetch = [&](int k0) {
#pragma unroll
        for (int i = 0; i < LA; ++i) {
            const int idx = tid + i * THREADS;
            ra[i] = piece(A, lda, m0 + idx / P, M, k0 + idx % P * 4);
        }
#pragma unroll
        for (int i = 0; i < LW; ++i) {
            const int idx = tid + i * THREADS;
            rw[i] = piece(W, ldw, n0 + idx / P, N, k0 + idx % P * 4);
        }
    };
    auto put = [&](int b) {
#pragma unroll
        for (int i = 0; i < LA; ++i) {
            const int idx = tid + i * THREADS, p = idx % P;
            float* d = as + (b * STEP + 4 * p) * BM + ((idx / P) ^ (TURN * p));
            d[0] = ra[i].x, d[BM] = ra[i].y, d[2 * BM] = ra[i].z, d[3 * BM] = ra[i].w;
        }
#pragma unroll
        for (int i = 0; i < LW; ++i) {
            const int idx = tid + i * THREADS, p = idx % P;
            float* d = ws + (b * STEP + 4 * p) * BN + ((idx / P) ^ (TURN * p));
            d[0] = rw[i].x, d[BN] = rw[i].y, d[2 * BN] = rw[i].z, d[3 * BN] = rw[i].w;
        }
    };

    uint64_t acc[TM / 2][TN];                      // two rows each
    float total[SPLIT ? 1 : TM][SPLIT ? 1 : TN];
#pragma unroll
    for (int i = 0; i < TM / 2; ++i)
#pragma unroll
        for (int q = 0; q < TN; ++q) acc[i][q] = 0;
    for (auto& t : total)
        for (auto& v : t) v = 0.f;
    // row of accumulator i, column of accumulator q (fours lie together)
    auto row = [&](int i) { return ty * 4 + i / 4 * (BM / (TM / 4)) + i % 4; };
    auto column = [&](int q) { return tx * 4 + q / 4 * (BN / (TN / 4)) + q % 4; };
    auto close = [&](int cl) {                     // the sums of class cl are complete
        if constexpr (!SPLIT) {
#pragma unroll
            for (int i = 0; i < TM / 2; ++i)
#pragma unroll
                for (int q = 0; q < TN; ++q) {
                    const float2 v = unpack2(acc[i][q]);
                    total[2 * i][q] = cl == 0 ? v.x : total[2 * i][q] + v.x;
                    total[2 * i + 1][q] = cl == 0 ? v.y : total[2 * i + 1][q] + v.y;
                    acc[i][q] = 0;
                }
        } else {
#pragma unroll
            for (int i = 0; i < TM / 2; ++i)
#pragma unroll
                for (int q = 0; q < TN; q += 4) {
                    const float2 v[4] = {unpack2(acc[i][q]), unpack2(acc[i][q + 1]), unpack2(acc[i][q + 2]), unpack2(acc[i][q + 3])};
                    *reinterpret_cast<float4*>(sums + row(2 * i) * BN + column(q)) = make_float4(v[0].x, v[1].x, v[2].x, v[3].x);
                    *reinterpret_cast<float4*>(sums + row(2 * i + 1) * BN + column(q)) = make_float4(v[0].y, v[1].y, v[2].y, v[3].y);
                }
        }
    };
    // The CTA's classes follow one another, a class's slices in ascending order, a slice in one step or two (the second only
    // where K reaches into it).
    int cls = first, c = first, h = 0, b = 0;
    if (c < slices) {
        fetch(c * SLICE);
        put(0);
        __syncthreads();
        while (true) {
            int ncls = cls, nc = c, nh = 0;
            if (STEP < SLICE && h == 0 && c * SLICE + STEP < K) {
                nh = 1;
            } else {
                nc += CLASSES;
                while (nc >= slices && ++ncls < first + OWN) nc = ncls;
            }
            const bool more = nc < slices;
            if (more) fetch(nc * SLICE + nh * STEP);
#pragma unroll
            for (int k = 0; k < STEP; ++k) {
                const float* ak = as + (b * STEP + k) * BM + ((ty * 4) ^ (TURN * (k / 4)));
                const float* wk = ws + (b * STEP + k) * BN + ((tx * 4) ^ (TURN * (k / 4)));
                ulonglong2 a[TM / 4];
#pragma unroll
                for (int i = 0; i < TM / 4; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(ak + i * (BM / (TM / 4)));
#pragma unroll
                for (int q = 0; q < TN; q += 4) {
                    const float4 w = *reinterpret_cast<const float4*>(wk + q / 4 * (BN / (TN / 4)));
                    const uint64_t w2[4] = {pack2(w.x, w.x), pack2(w.y, w.y), pack2(w.z, w.z), pack2(w.w, w.w)};
#pragma unroll
                    for (int i = 0; i < TM / 4; ++i)
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            fma2(acc[2 * i][q + e], a[i].x, w2[e]);
                            fma2(acc[2 * i + 1][q + e], a[i].y, w2[e]);
                        }
                }
            }
            if (!more || ncls != cls)
                for (int cl = cls; cl < (more ? ncls : first + OWN); ++cl) close(cl);      // empty classes add their zero too
            if (!more) break;
            put(b ^ 1);
            __syncthreads();
            b ^= 1, c = nc, cls = ncls, h = nh;
        }
    } else {
        for (int cl = first; cl < first + OWN; ++cl) close(cl);
    }
    const bool quads = N % 4 == 0 && ldc % 4 == 0 && (uintptr_t)C % 16 == 0;
    auto store = [&](int m, int n, float4 v) {
        if (m >= M || n >= N) return;
        if (bias != nullptr) {
            v.x += load_param(bias, bias_bf16, n);
            if (n + 1 < N) v.y += load_param(bias, bias_bf16, n + 1);
            if (n + 2 < N) v.z += load_param(bias, bias_bf16, n + 2);
            if (n + 3 < N) v.w += load_param(bias, bias_bf16, n + 3);
        }
        float* d = C + (size_t)m * ldc + n;
        if (quads) {
            *reinterpret_cast<float4*>(d) = v;
        } else {
            d[0] = v.x;
            if (n + 1 < N) d[1] = v.y;
            if (n + 2 < N) d[2] = v.z;
            if (n + 3 < N) d[3] = v.w;
        }
    };
    if constexpr (!SPLIT) {
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int q = 0; q < TN; q += 4)
                store(m0 + row(i), n0 + column(q), make_float4(total[i][q], total[i][q + 1], total[i][q + 2], total[i][q + 3]));
    } else {
        asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
        // this CTA adds up an eighth of the tile's rows
        for (int idx = tid; idx < BM / CLASSES * (BN / 4); idx += THREADS) {
            const int r = first * (BM / CLASSES) + idx / (BN / 4), n = idx % (BN / 4) * 4;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int cl = 0; cl < CLASSES; ++cl) {
                uint32_t remote;
                float4 x;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_addr(sums + r * BN + n)), "r"(cl));
                asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(x.x), "=f"(x.y), "=f"(x.z), "=f"(x.w) : "r"(remote) : "memory");
                if (cl == 0) v = x;
                else v.x += x.x, v.y += x.y, v.z += x.z, v.w += x.w;
            }
            store(m0 + r, n0 + n, v);
        }
        asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
    }
}

struct Call {
    const float* A;
    int lda;
    const float* W;
    int ldw;
    const void* bias;
    int bb;
    float* C;
    int ldc, M, N, K;
    cudaStream_t stream;
};

template <int MT, int BN, int CPT, int STAGES, bool VEC> int shared_ring(const Call& c) {
    constexpr int smem = STAGES * (BN + MT) * PERIOD * 4;
    auto kern = shared_ring_kernel<MT, BN, CPT, STAGES, VEC>;
    if (smem > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return (int)e;
    }
    return (int)launch_kernel(kern, dim3((c.N + BN - 1) / BN), dim3(BN / CPT * CLASSES), smem, c.stream, c.A, c.lda, c.W, c.ldw, c.bias,
                              c.bb, c.C, c.ldc, c.M, c.N, c.K);
}

// Shared memory of a CTA: what its rings may take while the rows of A leave room (110 KB instead, for a second CTA, is 4 to 8 % slower on
// average over 2,400 shapes: two stages where three fit), the same where those rows go through the rings, where two
// CTAs are to share an SM, and what there is
constexpr int FEW_SMEM = 160 * 1024, FEW_SMEM_THROUGH = 220 * 1024, FEW_SMEM_TWO = 110 * 1024, FEW_SMEM_MOST = 226 * 1024;
constexpr int FEW_X_MOST = 160 * 1024;         // rows of A that are kept whole, in bytes

// MT rows a CTA, 4 CPT columns a warp
template <int MT, int CPT, bool VEC, bool XRES> int few(const Call& c, int budget = XRES ? FEW_SMEM : FEW_SMEM_THROUGH) {
    const int groups = (c.N + 4 * CPT - 1) / (4 * CPT), periods = (c.K + PERIOD - 1) / PERIOD, blocks = (c.M + MT - 1) / MT;
    const int x = XRES ? periods * min(c.M, MT) * PERIOD * 4 : 0, per_warp = (4 * CPT + (XRES ? 0 : MT)) * PERIOD * 4;
    // as many warps as share a CTA's columns evenly
    const int most = min(FEW_WARPS, (FEW_SMEM_MOST - x) / (2 * per_warp)), each = max(2, (groups + 147) / 148), rounds = (each + most - 1) / most;
    const int warps = (each + rounds - 1) / rounds;
    const int ctas = min(148, (groups + warps - 1) / warps);
    const int stages = max(2, min(8, (budget - x) / (per_warp * warps))), smem = x + stages * per_warp * warps;
    auto kern = few_rows_kernel<MT, CPT, VEC, XRES>;
    // the limit belongs to the function, not to the call: one value, so that no thread's call lowers it under another's
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, FEW_SMEM_MOST);
    if (e != cudaSuccess) return (int)e;
    return (int)launch_kernel(kern, dim3(ctas, blocks), dim3(warps * 32), smem, c.stream, c.A, c.lda, c.W, c.ldw, c.bias,
                              c.bb, c.C, c.ldc, c.M, c.N, c.K, stages);
}

// Rows of A that do not fit whole, cut into blocks that do, where the blocks' CTAs all run side by side: each reads W, but few columns are
// soon read and few CTAs leave the SMs idle (16 rows, N 256, K 8,960: 23.5 us in four blocks, 58.0 through the rings); -1 where not
template <int MT> int side_by_side(const Call& c, long long row) {
    const long long columns = (long long)((c.M + MT - 1) / MT) * c.N, x = min(c.M, MT) * row;
    if (x <= FEW_X_MOST && columns <= 148 * 8) return few<MT, 1, true, true>(c);
    if (x <= 94 * 1024 && columns <= 148 * 16) return few<MT, 1, true, true>(c, FEW_SMEM_TWO);
    if (x <= FEW_X_MOST && columns <= 148 * 16 && c.M > 4) return few<MT, 2, true, true>(c);
    if constexpr (MT > 1) return side_by_side<MT == 3 ? 2 : MT / 2>(c, row);
    return -1;
}

// Which of the two, and with how many columns a lane: from 2,394 shapes of 1 to 16 rows, 8 to 151,936 columns and K 260 to 40,960, weights
// mostly from memory, and 444 whose rows start off 16-byte boundaries (microseconds).  The first that holds:
// - N whose CTAs of eight columns all run at once (`PLACES`: their rings bound how many an SM holds) has a ring a CTA where K is too
//   short to pay for bringing all of A first (8 rows, N 896: K 640 5.2 and 5.2 by warps, K 4,864 25.8 and 19.6), where the rows are
//   twelve and more (16 rows, N 54, K 2,044: 15.4 and 16.7) or copies are single entries;
// - rows of A that do not fit whole: blocks of them side by side (above); nine rows and more in two blocks, one after the other, as long as
//   eight fit and the columns are many (two streams of W, but eight rows leave the SM's shared memory the time for them; 16 rows, N 18,944, K 4,864:
//   142.6, once 159.4); else through the warps' rings, W once at any K (16 rows, N 4,600, K 18,944: 153.6, a ring a CTA 158.6 with 32 columns; 3 rows,
//   N 4,200, K 40,960: 104.0 and 220.9); single entries go through a ring a CTA;
// - just below 148 x 64 columns CTAs of 32 columns, two an SM, leave no SM idle, while the warps' shares are uneven
//   (1 row, N 9,400, K 896: 6.9, by warps 7.2);
// - else a ring a warp.  More columns a lane make the reads of A serve more products (8 rows, N 18,944, K 896: 25.8 with one, 18.7 with
//   two, 17.7 with four), but fewer share few columns more evenly (8 rows, N 3,300, K 896: 7.3, 7.2, 10.7) and leave more warps
//   beside much of A.  Four take too many registers beyond eight rows and too many bytes a stage beside more than 98 KB of A; one and two
//   rows gain from them with few columns and a short K only (1 row, N 9,728, K 384: 4.7 with two, 4.3 with four).
// Three rows have a form of their own: that of four reads a row of A more (10 to 14 % slower below 4,736 columns, 3 to 6 % above where K
// is below 1,000).
template <int MT, bool VEC> int few_k(const Call& c) {
    constexpr int CTA_MT = MT == 3 ? 4 : MT;                                           // a ring a CTA has no form of three rows
    constexpr int PLACES = VEC || MT > 4 ? 148 * 8 * (MT <= 2 ? 4 : MT <= 4 ? 3 : MT <= 8 ? 2 : 1) : 148 * 32 - 1;
    constexpr int SHORT = MT == 1 ? 1792 : MT == 3 || MT == 4 ? 640 : 1280;
    const long long row = ((long long)c.K + PERIOD - 1) / PERIOD * PERIOD * 4, x = row * c.M;       // bytes of A in shared memory
    const bool fits = x <= (MT == 8 && !VEC ? 128 * 1024 : FEW_X_MOST);
    if (c.N <= PLACES && (!VEC || (fits && (c.K < SHORT || c.M > 11)))) return shared_ring<CTA_MT, 8, 1, 5, VEC>(c);
    if constexpr (!VEC) {
        if (!fits) return shared_ring<CTA_MT, 32, 2, 3, VEC>(c);
    } else {
        if (!fits) {
            const int rc = side_by_side<MT>(c, row);
            if (rc >= 0) return rc;
            if constexpr (MT == 16) {
                if (c.N >= 148 * 32 && 8 * row <= FEW_X_MOST)
                    return c.N >= 148 * 64 && 8 * row <= 98 * 1024 ? few<8, 4, true, true>(c) : few<8, 2, true, true>(c);
            }
            return c.N <= 148 * (MT <= 4 ? 28 : MT <= 8 ? 14 : 16) ? few<MT, 1, true, false>(c) : few<MT, 2, true, false>(c);
        }
        if constexpr (MT <= 4) {
            if (c.N <= 148 * 64 && c.N > 148 * (MT > 2 ? 60 : c.K < 1280 ? 40 : 48)) return shared_ring<CTA_MT, 32, 2, 3, VEC>(c);
        }
    }
    if constexpr (MT <= 8) {
        if (c.N >= 148 * 64 && (MT > 2 ? x <= 98 * 1024 : c.N <= 148 * 84 && c.K <= 1280)) return few<MT, 4, VEC, true>(c);
    }
    const int one = 148 * (MT == 1 ? 32 : MT <= 8 ? 28 : 16);
    return c.N <= one || (MT <= 2 && x > 144 * 1024) ? few<MT, 1, VEC, true>(c) : few<MT, 2, VEC, true>(c);
}

template <bool VEC> int few_m(const Call& c) {
    if (c.M <= 1) return few_k<1, VEC>(c);
    if (c.M <= 2) return few_k<2, VEC>(c);
    if (c.M <= 3) return few_k<3, VEC>(c);
    if (c.M <= 4) return few_k<4, VEC>(c);
    if (c.M <= 8) return few_k<8, VEC>(c);
    return few_k<16, VEC>(c);
}

template <int BM, int BN, int TM, int TN, int STEP, bool SPLIT, bool VEC> int many(const Call& c) {
    constexpr int smem = many_smem<BM, BN, STEP, SPLIT>();
    static_assert(smem <= 48 * 1024, "");
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3((BM / TM) * (BN / TN));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = c.stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = SPLIT ? CLASSES : 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
    constexpr long long MOST = 65535LL * BM;       // rows of a launch: what a grid's y takes
    for (long long m = 0; m < c.M; m += MOST) {
        const int rows = (int)(c.M - m < MOST ? c.M - m : MOST);
        cfg.gridDim = dim3((c.N + BN - 1) / BN, (rows + BM - 1) / BM, SPLIT ? CLASSES : 1);
        const cudaError_t e = cudaLaunchKernelEx(&cfg, many_rows_kernel<BM, BN, TM, TN, STEP, SPLIT, VEC>, c.A + m * c.lda, c.lda, c.W, c.ldw,
                                                 c.bias, c.bb, c.C + m * c.ldc, c.ldc, rows, c.N, c.K);
        if (e != cudaSuccess) return (int)e;
    }
    return 0;
}

template <bool VEC> int pick(const Call& c) {
    auto tiles = [&](int bm, int bn) { return (long long)((c.M + bm - 1) / bm) * ((c.N + bn - 1) / bn); };
    // A short K (few of the eight classes have a slice) leaves the few rows' lanes and the cluster's CTAs idle: small tiles,
    // while they are no more than ten an SM (252 rows, N 2,048, K 32: 4.4 us, cluster 13.1; 512 rows, N 8,192, K 32: 14.3 us, tiles
    // of 64 x 64 11.8), by half a slice where K ends in the first (K 8, up to 1,500 tiles: 0.83 to 0.92 of the time).  Few rows take longer the more rows and
    // columns they have, the tiles the longer K is (12 rows, N 4,096, K 64: 4.2 us by tiles, 13.6 by rows; 4 rows, N 512, K 128: 6.2 and 2.4).
    int rows = 1;
    while (rows < c.M && rows < 32) rows *= 2;
    if (c.K <= (rows == 32 ? 3 * SLICE : (c.N < 1500 ? 3 : c.N < 4736 ? 10 : 12) * rows)) {
        if (tiles(32, 32) > 1500) return many<64, 64, 8, 4, 16, false, VEC>(c);
        return c.K <= SLICE / 2 ? many<32, 32, 4, 4, 16, false, VEC>(c) : many<32, 32, 4, 4, 32, false, VEC>(c);
    }
    if (c.M <= 16) return few_m<VEC>(c);
    // From 4,600 shapes of 17 to 2,048 rows, K 4 to 20,000.  A cluster shares the K of a tile of 64 x 64 where the tiles alone would not
    // fill the SMs some five times over.  It is worth less the fewer of its CTAs' slices are whole rounds of the classes (512 rows, N 4,096, 512 tiles: K 512,
    // 16 slices, 64.1 us and 62.0 unsplit, K 544, 17 slices, 79.4 and 65.5) and the shorter K is, for its two barriers (K 288 57.0 and 36.6).
    const int slices = (c.K + SLICE - 1) / SLICE, deep = (slices + CLASSES - 1) / CLASSES;
    const long long t64 = tiles(64, 64), full = slices >= 4 * CLASSES ? 900 : (150LL * slices / deep - 400) * min(c.K, 640) / 640;
    if (t64 >= (full > 301 ? full : 301) && (t64 > 400 || c.K <= 128 || c.K > 384)) return many<64, 64, 8, 4, 16, false, VEC>(c);
    // Tiles of 32 x 32 walk a short K alone: their time grows with K, the cluster's with its CTAs (1,000 rows, N 1,000, 256 tiles: K 192
    // 0.69 of the cluster's time, K 384 0.88, K 512 1.10; 512 rows, N 600, 80 tiles: K 128 0.84, K 192 1.08)
    if (c.M > 32 && slices <= 12 && t64 > (slices <= 4 ? 18 : min(222, 37 * (slices - 2)))) return many<32, 32, 4, 4, 32, false, VEC>(c);
    // Split tiles, by how many CTAs of 64 x 64 an SM gets (`whole`; of 32 x 64: `half`, at some 0.55 of the time each).  Half tiles of
    // whole slices where no SM gets two of them, or more than two but three of 64 x 64 at most: half the barriers, and more bytes on their way from
    // few CTAs (242 rows, N 707, K 5,900: 85.4 us, 99.8 in tiles of 64 x 64; 900 shapes of up to 55 tiles: 0.8 to 0.9 of the time).  At four, 256
    // threads a tile (296 rows, N 868, K 14,312: 246 us, 301 with 128).  From there on the SMs are full, and whole tiles read less; half tiles
    // where they share the SMs more evenly, or those of 64 x 64 leave a fifth of them idle (178 rows, N 278, K 2,309, 120 CTAs: 26.0 us, half tiles
    // 34.5; 43 rows, N 604, K 11,256, 80 CTAs: 89.3 and 76.7).
    const long long whole = (t64 * CLASSES + 147) / 148, half = (tiles(32, 64) * CLASSES + 147) / 148;
    if (half == 1 || (c.M > 32 && half > 2 && whole <= 3)) return many<32, 64, 4, 4, 32, true, VEC>(c);
    if (c.M > 32 && whole == 4) return many<64, 64, 4, 4, 16, true, VEC>(c);
    return c.M <= 32 || (half == 2 && t64 < 15) || (whole <= 6 && 55 * half < 100 * whole) ? many<32, 64, 4, 4, 16, true, VEC>(c)
                                                                                                 : many<64, 64, 8, 4, 16, true, VEC>(c);
}

}  // namespace f32gemm
}  // namespace prism

PRISM_EXPORT int prism_sgemm_nt(const float* A, int lda, const float* W, int ldw, const void* bias,
                                int bias_dtype, float* C, int ldc, int M, int N, int K,
                                cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    const prism::f32gemm::Call c{A, lda, W, ldw, bias, bias_dtype == PRISM_DTYPE_BF16, C, ldc, M, N, K, stream};
    // 16-byte copies where every row starts on a 16-byte boundary
    const bool vec = ((uintptr_t)A | (uintptr_t)W) % 16 == 0 && (M == 1 || lda % 4 == 0) && (N == 1 || ldw % 4 == 0);
    return vec ? prism::f32gemm::pick<true>(c) : prism::f32gemm::pick<false>(c);
}
