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
// Few rows (M <= 16) are bound by the stream of weights: measured at 3 rows,
// K 896, N 151,936 (545 MB) 2.4 ms with one tile kernel for every M, 0.11 ms here.
#include "f32x2.cuh"

namespace prism {
namespace f32gemm {

constexpr int SLICE = 32, CLASSES = 8, PERIOD = SLICE * CLASSES;

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// `bytes` of the 16 (of the 4) are copied, the rest of the destination becomes zero
__device__ __forceinline__ void copy16(uint32_t dst, const float* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copy4(uint32_t dst, const float* src, int bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

// ---- few rows -----------------------------------------------------------------------------------------
// A CTA owns BN weight rows and all M <= MT rows of A and walks K in periods of 256 through a ring of shared
// memory stages (cp.async; the weights of the first stages are brought into L2 before the dependency wait: read they are
// after it, so that they may also be what an earlier kernel of the stream writes).  Thread =
// (class, column group): the eight classes of a column are eight neighbouring lanes.  A row's 16-byte pieces lie
// at (class, piece ^ class), so that the eight lanes read eight different bank groups.
// BN 8 where N is small (N 896: 112 CTAs), else 32 with two columns a thread, which halves the reads of A.
template <int MT, int BN, int CPT, int STAGES, bool VEC>
__global__ void __launch_bounds__(BN / CPT * CLASSES)
few_rows_kernel(const float* A, int lda, const float* W, int ldw, const void* __restrict__ bias,
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

template <int MT, int BN, int CPT, int STAGES, bool VEC> int few(const Call& c) {
    constexpr int smem = STAGES * (BN + MT) * PERIOD * 4;
    auto kern = few_rows_kernel<MT, BN, CPT, STAGES, VEC>;
    if (smem > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return (int)e;
    }
    return (int)launch_kernel(kern, dim3((c.N + BN - 1) / BN), dim3(BN / CPT * CLASSES), smem, c.stream, c.A, c.lda, c.W, c.ldw, c.bias,
                              c.bb, c.C, c.ldc, c.M, c.N, c.K);
}

// BN 8 keeps every SM busy down to N of about a thousand; from 148 x 32 columns on wider CTAs fill the GPU too
template <int MT, bool VEC> int few_n(const Call& c) {
    return c.N >= 4736 ? few<MT, 32, 2, 3, VEC>(c) : few<MT, 8, 1, 5, VEC>(c);
}

template <bool VEC> int few_m(const Call& c) {
    if (c.M <= 1) return few_n<1, VEC>(c);
    if (c.M <= 2) return few_n<2, VEC>(c);
    if (c.M <= 4) return few_n<4, VEC>(c);
    if (c.M <= 8) return few_n<8, VEC>(c);
    return few_n<16, VEC>(c);
}

template <int BM, int BN, int TM, int TN, int STEP, bool SPLIT, bool VEC> int many(const Call& c) {
    constexpr int smem = many_smem<BM, BN, STEP, SPLIT>();
    static_assert(smem <= 48 * 1024, "");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((c.N + BN - 1) / BN, (c.M + BM - 1) / BM, SPLIT ? CLASSES : 1);
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
    return (int)cudaLaunchKernelEx(&cfg, many_rows_kernel<BM, BN, TM, TN, STEP, SPLIT, VEC>, c.A, c.lda, c.W, c.ldw, c.bias, c.bb, c.C,
                                   c.ldc, c.M, c.N, c.K);
}

template <bool VEC> int pick(const Call& c) {
    auto tiles = [&](int bm, int bn) { return (long long)((c.M + bm - 1) / bm) * ((c.N + bn - 1) / bn); };
    // A short K (few of the eight classes have a slice) leaves the few rows' lanes and the cluster's CTAs idle: small tiles,
    // while they are no more than ten an SM (252 rows, N 2,048, K 32: 5.8 us, cluster 16.1; 512 rows, N 8,192, K 16: 14.7 us,
    // 128 x 64 13.1).  Few rows take longer the more rows and columns they have, the tiles the longer K is (12 rows, N 4,096, K 64:
    // 4.2 us by tiles, 13.6 by rows; 4 rows, N 512, K 128: 6.2 and 2.4).
    int rows = 1;
    while (rows < c.M && rows < 32) rows *= 2;
    if (c.K <= (rows == 32 ? 3 * SLICE : (c.N < 1500 ? 3 : c.N < 4736 ? 10 : 12) * rows))
        return tiles(32, 32) <= 1500 ? many<32, 32, 4, 4, 32, false, VEC>(c) : many<64, 64, 8, 4, 16, false, VEC>(c);
    if (c.M <= 16) return few_m<VEC>(c);
    // Where tiles of 64 x 64 would not fill the SMs some six times over, a cluster shares their K, as far as its CTAs have slices
    // (252 rows, N 9,728, K 896, 608 tiles: 130 us, unsplit 137; 512 rows, 1,216 tiles: 250 and 229).  Six of its CTAs fit an SM; where
    // one round holds all, half tiles may share the SMs more evenly, at some 0.55 of the time each (252 rows, K 4,864: N 896 83 us
    // against 104; K 896, N 1,152 26.6 and 25.6).
    if (tiles(64, 64) * PERIOD >= 900LL * (c.K < PERIOD ? c.K : PERIOD)) return many<64, 64, 8, 4, 16, false, VEC>(c);
    const long long whole = (tiles(64, 64) * CLASSES + 147) / 148, half = (tiles(32, 64) * CLASSES + 147) / 148;
    return c.M <= 32 || (whole <= 6 && 55 * half < 100 * whole) ? many<32, 64, 4, 4, 16, true, VEC>(c) : many<64, 64, 8, 4, 16, true, VEC>(c);
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
