// Batched float32 matrix products on the FMA pipe, shared by the exact linear projection and the unfused attention
// pieces with their backward pass: C(m,n) = alpha * sum_k A(m,k) B(k,n), every output one chain of fused multiply-adds
// in ascending k (four chains, one per quarter of the k range, where split_kernel takes it).
//
// Bound: the FP32 pipe (128 FMA per clock per SM: 74 TFLOP/s).  A thread owns 8 x 8 outputs as 8 x 4 packed pairs
// (fma.rn.f32x2 halves the issue slots, which leaves room for the shared-memory loads and the tile traffic); a warp
// 32 x 64 (or 64 x 32 where the product has only 32 columns).  Tiles of A and B cross shared memory as [k][m] and [k][n],
// double-buffered through registers: the global loads of slice i+1 are in flight under the products of slice i.
#pragma once
#include "common.cuh"

namespace grl {
namespace sgemm {

constexpr int BK = 16;

// One operand.  Element (outer, inner) of batch (b, h) lives at base[b*sb + h*sh + outer*ld + inner]; which of its two
// indices is the contiguous one is a template parameter of the kernel.  vec: rows start on 16-byte boundaries.
struct Operand {
    const float* base;
    long long sb, sh, ld;
    int vec;
};
struct Output {
    float* base;
    long long sb, sh, ld;
};
inline Operand operand(const float* base, long long sb, long long sh, long long ld) {
    const bool vec = ((uintptr_t)base % 16 == 0) && sb % 4 == 0 && sh % 4 == 0 && ld % 4 == 0;
    return Operand{base, sb, sh, ld, vec ? 1 : 0};
}

template <int BM_, int BN_>
struct Shape {
    static constexpr int BM = BM_, BN = BN_;
    static constexpr int WM = BN >= 64 ? 32 : 64, WN = BN >= 64 ? 64 : 32;      // outputs of a warp
    static constexpr int WARPS_N = BN / WN, WARPS = (BM / WM) * WARPS_N, THREADS = WARPS * 32;
    static constexpr int LANES_N = WN / 8;
    static constexpr int LDA = BM + 4, LDB = BN + 4;                            // floats per k row of a tile
    static constexpr int TILE = BK * (LDA + LDB);                               // floats per stage
    static constexpr int MIN_CTAS = 384 / THREADS > 8 ? 8 : THREADS == 256 ? 2 : 384 / THREADS;   // at least 12 warps an SM (<= 168 registers)
};

__device__ __forceinline__ float4 load4(const float* row, int i, int n, bool vec) {
    if (vec && i + 3 < n) return __ldg(reinterpret_cast<const float4*>(row + i));
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < n) v.x = __ldg(row + i);
    if (i + 1 < n) v.y = __ldg(row + i + 1);
    if (i + 2 < n) v.z = __ldg(row + i + 2);
    if (i + 3 < n) v.w = __ldg(row + i + 3);
    return v;
}

__device__ __forceinline__ void store4(float* dst, float4 v, int left, bool vec) {     // left: values that are inside the row
    if (vec && left > 3) {
        *reinterpret_cast<float4*>(dst) = v;
        return;
    }
    if (left > 0) dst[0] = v.x;
    if (left > 1) dst[1] = v.y;
    if (left > 2) dst[2] = v.z;
    if (left > 3) dst[3] = v.w;
}

// One k slice of an operand on its way from global to shared memory: EXT rows (m or n) x BK.  KC: the k index is the
// contiguous one (a thread's float4 is four k of one row and is stored transposed); otherwise the row index is.
// PAIR: a second tensor w of the same shape is read along, and what is stored is w * (v - dot) with one `dot` per row
// (KC) or per k -- the softmax backward, formed on the way to shared memory.
template <int EXT, int THREADS, bool KC, bool PAIR = false>
struct Fetch {
    static constexpr int VECS = EXT * BK / 4 / THREADS;
    static_assert(EXT * BK / 4 % THREADS == 0, "slice must divide over the threads");
    float4 v[VECS], w[PAIR ? VECS : 1];
    __device__ __forceinline__ void load(const float* base, const float* pair, long long ld, bool vec, int row0, int rows, int k0, int K,
                                         int tid) {
#pragma unroll
        for (int i = 0; i < VECS; ++i) {
            const int q = tid + i * THREADS;
            const int outer = KC ? row0 + q / (BK / 4) : k0 + q / (EXT / 4), inner = KC ? k0 + (q % (BK / 4)) * 4 : row0 + (q % (EXT / 4)) * 4;
            const bool in = outer < (KC ? rows : K);
            const long long off = (long long)outer * ld;
            v[i] = in ? load4(base + off, inner, KC ? K : rows, vec) : make_float4(0.f, 0.f, 0.f, 0.f);
            if constexpr (PAIR) w[i] = in ? load4(pair + off, inner, KC ? K : rows, vec) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
    __device__ __forceinline__ void store(float* tile, int LD, int tid, const float* dots, int row0, int rows, int k0, int K) const {
#pragma unroll
        for (int i = 0; i < VECS; ++i) {
            const int q = tid + i * THREADS;
            float4 x = v[i];
            if constexpr (PAIR) {
                const int outer = KC ? row0 + q / (BK / 4) : k0 + q / (EXT / 4);
                const float d = outer < (KC ? rows : K) ? dots[outer] : 0.f;
                x = make_float4(w[i].x * (x.x - d), w[i].y * (x.y - d), w[i].z * (x.z - d), w[i].w * (x.w - d));
            }
            if constexpr (KC) {
                float* p = tile + (q % (BK / 4)) * 4 * LD + q / (BK / 4);
                p[0] = x.x; p[LD] = x.y; p[2 * LD] = x.z; p[3 * LD] = x.w;
            } else {
                *reinterpret_cast<float4*>(tile + (q / (EXT / 4)) * LD + (q % (EXT / 4)) * 4) = x;
            }
        }
    }
};

// The 8 x 8 outputs of a thread: rows row(i), columns col(j).
template <typename SH>
struct Place {
    int m0, n0;         // first row / column of this thread inside the CTA's tile
    __device__ __forceinline__ Place(int tid) {
        const int warp = tid >> 5, lane = tid & 31;
        m0 = (warp / SH::WARPS_N) * SH::WM + (lane / SH::LANES_N) * 4;
        n0 = (warp % SH::WARPS_N) * SH::WN + (lane % SH::LANES_N) * 4;
    }
    __device__ __forceinline__ int row(int i) const { return m0 + (i & 3) + (i >> 2) * (SH::WM / 2); }
    __device__ __forceinline__ int col(int j) const { return n0 + (j & 3) + (j >> 2) * (SH::WN / 2); }
};

// acc[i][j/2] over k in [0, K): the main loop.  CAUSAL: rows of the product only see k <= m (slices that straddle the
// diagonal test every term; the caller passes the tile's own upper limit as K).  With `pair` A is pair * (a - dots).
// GROUPS > 1: the threads are one of several groups with a product of their own (group `g`, barrier g + 1).
template <typename SH, bool AKC, bool BKC, bool CAUSAL, bool PAIR, int GROUPS = 1>
__device__ __forceinline__ void mainloop(float2 (&acc)[8][4], float* smem, const float* a, const Operand& A, const float* b,
                                         const Operand& B, int m0, int n0, int M, int N, int K, const float* pair, const float* dots) {
    const int tid = GROUPS == 1 ? threadIdx.x : threadIdx.x % SH::THREADS;
    auto sync = [&]() {
        if constexpr (GROUPS == 1) __syncthreads();
        else asm volatile("bar.sync %0, %1;" ::"r"((int)threadIdx.x / SH::THREADS + 1), "n"(SH::THREADS) : "memory");
    };
    const Place<SH> at(tid);
    Fetch<SH::BM, SH::THREADS, AKC, PAIR> fa;
    Fetch<SH::BN, SH::THREADS, BKC> fb;
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = make_float2(0.f, 0.f);
    fa.load(a, pair, A.ld, A.vec, m0, M, 0, K, tid);
    fb.load(b, nullptr, B.ld, B.vec, n0, N, 0, K, tid);
    fa.store(smem, SH::LDA, tid, dots, m0, M, 0, K);
    fb.store(smem + BK * SH::LDA, SH::LDB, tid, nullptr, n0, N, 0, K);
    sync();
    const int slices = (K + BK - 1) / BK;
    for (int s = 0; s < slices; ++s) {
        const float* as = smem + (s & 1) * SH::TILE;
        const float* bs = as + BK * SH::LDA;
        if (s + 1 < slices) {
            fa.load(a, pair, A.ld, A.vec, m0, M, (s + 1) * BK, K, tid);
            fb.load(b, nullptr, B.ld, B.vec, n0, N, (s + 1) * BK, K, tid);
        }
        const bool diagonal = CAUSAL && (s + 1) * BK > m0;
        if (!diagonal) {
#pragma unroll
            for (int k = 0; k < BK; ++k) {
                float av[8];
                float2 bv[4];
                *reinterpret_cast<float4*>(av) = *reinterpret_cast<const float4*>(as + k * SH::LDA + at.m0);
                *reinterpret_cast<float4*>(av + 4) = *reinterpret_cast<const float4*>(as + k * SH::LDA + at.m0 + SH::WM / 2);
                *reinterpret_cast<float4*>(bv) = *reinterpret_cast<const float4*>(bs + k * SH::LDB + at.n0);
                *reinterpret_cast<float4*>(bv + 2) = *reinterpret_cast<const float4*>(bs + k * SH::LDB + at.n0 + SH::WN / 2);
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[i][j] = __ffma2_rn(make_float2(av[i], av[i]), bv[j], acc[i][j]);
            }
        } else {
            for (int k = 0; k < BK; ++k) {
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float av = as[k * SH::LDA + at.row(i)];
                    if (s * BK + k <= m0 + at.row(i)) {
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                            acc[i][j] = __ffma2_rn(make_float2(av, av), *reinterpret_cast<const float2*>(bs + k * SH::LDB + at.col(2 * j)), acc[i][j]);
                    }
                }
            }
        }
        if (s + 1 < slices) {
            float* ns = smem + ((s + 1) & 1) * SH::TILE;
            fa.store(ns, SH::LDA, tid, dots, m0, M, (s + 1) * BK, K);
            fb.store(ns + BK * SH::LDA, SH::LDB, tid, nullptr, n0, N, (s + 1) * BK, K);
        }
        sync();
    }
}

// Write alpha * acc (+ bias) to C, rows < M and columns < N only.
template <typename SH>
__device__ __forceinline__ void store_tile(const float2 (&acc)[8][4], float* c, long long ld, int m0, int n0, int M, int N, float alpha,
                                           const float* bias) {
    const Place<SH> at(threadIdx.x);
    const bool vec = ((uintptr_t)c % 16 == 0) && ld % 4 == 0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int n = n0 + at.col(4 * h);
        if (n >= N) continue;
        const float4 bv = bias ? load4(bias, n, N, (uintptr_t)bias % 16 == 0) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int m = m0 + at.row(i);
            if (m >= M) continue;
            const float2 x = acc[i][2 * h], y = acc[i][2 * h + 1];
            const float4 v = make_float4(x.x * alpha + bv.x, x.y * alpha + bv.y, y.x * alpha + bv.z, y.y * alpha + bv.w);
            store4(c + (long long)m * ld + n, v, N - n, vec);
        }
    }
}

template <typename SH, bool AKC, bool BKC, bool CAUSAL, bool EARLY>
__global__ void __launch_bounds__(SH::THREADS, SH::MIN_CTAS) kernel(Operand A, Operand B, Output C, const float* bias, int M, int N, int K, int H,
                                                      float alpha) {
    __shared__ __align__(16) float smem[2 * SH::TILE];
    const int z = blockIdx.z, b = z / H, h = z % H;
    const int m0 = blockIdx.y * SH::BM, n0 = blockIdx.x * SH::BN;
    float2 acc[8][4];
    mainloop<SH, AKC, BKC, CAUSAL, false>(acc, smem, A.base + b * A.sb + h * A.sh, A, B.base + b * B.sb + h * B.sh, B, m0, n0, M, N,
                                   CAUSAL ? min(K, m0 + SH::BM) : K, nullptr, nullptr);
    store_tile<SH>(acc, C.base + b * C.sb + h * C.sh, C.ld, m0, n0, M, N, alpha, bias);
    if constexpr (EARLY) pdl_wait();
}

// 64 x 64 tiles with the K range cut over four groups of threads, whose partial tiles are added in ascending order.  One group
// alone is two warps an SM where there is one tile for each: the chain of load, barrier and products of a slice is the time
// then (128 x 768 x 3072: 64 us), and it is four times shorter this way.  Backward, us, whole / split: 1 x 4 heads x 1024 x 64 140 / 86,
// 2 x 12 x 512 x 64 164 / 102, 1 x 8 x 256 x 64 41 / 25, 1 x 4 x 700 x 32 129 / 47.
constexpr int kSplit = 4;
template <typename SH> struct Split {
    static constexpr int REGION = 2 * SH::TILE;         // floats a group has
    static constexpr int THREADS = SH::THREADS * kSplit, SMEM = kSplit * REGION * (int)sizeof(float);
    static constexpr int MIN_CTAS = THREADS > 128 ? 1 : 2;      // eight warps an SM with every register they ask for (32 columns at 168
                                                                // registers spilled: 84 us for 47 of the last figure above)
};
// One tile; operands, `pair` and `dots` as in mainloop, all of this batch.
template <typename SH, bool AKC, bool BKC, bool PAIR>
__device__ __forceinline__ void split_tile(float* dyn, const float* a0, const Operand& A, const float* b0, const Operand& B, float* c, long long ldc,
                                           const float* bias, int m0, int n0, int M, int N, int K, float alpha, const float* pair,
                                           const float* dots) {
    constexpr int REGION = Split<SH>::REGION;
    static_assert(REGION >= SH::THREADS * 64, "a partial tile reuses its group's stages");
    const int g = threadIdx.x / SH::THREADS, tid = threadIdx.x % SH::THREADS;
    const int slices = (K + BK - 1) / BK, k0 = g * slices / kSplit * BK, k1 = min(K, (g + 1) * slices / kSplit * BK);
    const long long ka = AKC ? k0 : k0 * A.ld;
    float2 acc[8][4];
    mainloop<SH, AKC, BKC, false, PAIR, kSplit>(acc, dyn + g * REGION, a0 + ka, A, b0 + (BKC ? k0 : k0 * B.ld), B, m0, n0, M, N, k1 - k0,
                                                PAIR ? pair + ka : nullptr, PAIR && !AKC ? dots + k0 : dots);
    float2* mine = reinterpret_cast<float2*>(dyn + g * REGION) + tid;
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) mine[(i * 4 + j) * SH::THREADS] = acc[i][j];
    __syncthreads();
    // group g finishes rows 2g and 2g + 1 of every thread's eight
    const Place<SH> at(tid);
    const bool vec = ((uintptr_t)c % 16 == 0) && ldc % 4 == 0;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int i = 2 * g + q, m = m0 + at.row(i);
        if (m >= M) continue;
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
            const int n = n0 + at.col(4 * hh);
            float2 x = make_float2(0.f, 0.f), y = x;
#pragma unroll
            for (int p = 0; p < kSplit; ++p) {
                const float2* part = reinterpret_cast<const float2*>(dyn + p * REGION) + tid;
                x = __fadd2_rn(x, part[(i * 4 + 2 * hh) * SH::THREADS]);
                y = __fadd2_rn(y, part[(i * 4 + 2 * hh + 1) * SH::THREADS]);
            }
            const float4 bv = bias ? load4(bias, n, N, (uintptr_t)bias % 16 == 0) : make_float4(0.f, 0.f, 0.f, 0.f);
            store4(c + (long long)m * ldc + n, make_float4(x.x * alpha + bv.x, x.y * alpha + bv.y, y.x * alpha + bv.z, y.y * alpha + bv.w), N - n, vec);
        }
    }
}

template <typename SH, bool AKC, bool BKC, bool EARLY>
__global__ void __launch_bounds__(Split<SH>::THREADS, Split<SH>::MIN_CTAS)
split_kernel(Operand A, Operand B, Output C, const float* bias, int M, int N, int K, int H, float alpha) {
    extern __shared__ __align__(16) float dyn[];
    const int z = blockIdx.z, b = z / H, h = z % H;
    split_tile<SH, AKC, BKC, false>(dyn, A.base + b * A.sb + h * A.sh, A, B.base + b * B.sb + h * B.sh, B, C.base + b * C.sb + h * C.sh, C.ld, bias,
                                    blockIdx.y * SH::BM, blockIdx.x * SH::BN, M, N, K, alpha, nullptr, nullptr);
    if constexpr (EARLY) pdl_wait();
}

// Which tile: the widest one whose grid still gives every SM two CTAs; 64 rows otherwise, so that a small product
// spreads over more SMs.  32 columns only where the product has no more (half of a 64-column tile would be padding).
inline int tile_rows(int M, int N, int batch, int bn, int sms) {
    const long long big = (long long)((M + 127) / 128) * ((N + bn - 1) / bn) * batch;
    return big >= 2LL * sms ? 128 : 64;
}

// From two slices on: backward of 4 x 12 heads x 128 x 128 53.5 us whole, 41.2 split; 1 x 1 x 64 x 64 22.7 and 17.5.
inline bool split_pays(int K) { return K > BK; }

// EARLY: the launch starts under the kernel before it on the stream, of which it needs nothing but the end (see launch_pdl).
template <bool AKC, bool BKC, bool CAUSAL = false, bool EARLY = false>
int launch(grl_device* dev, const Operand& A, const Operand& B, const Output& C, const float* bias, int M, int N, int K, int batch,
           int H, float alpha, const char* name, int rows_hint = 0) {
    cudaError_t err = cudaSuccess;
    auto go = [&](auto shape) {
        using SH = decltype(shape);
        dim3 grid((N + SH::BN - 1) / SH::BN, (M + SH::BM - 1) / SH::BM, batch * H);
        if constexpr (EARLY) err = launch_pdl(kernel<SH, AKC, BKC, CAUSAL, true>, grid, SH::THREADS, 0, dev->stream, A, B, C, bias, M, N, K, H, alpha);
        else kernel<SH, AKC, BKC, CAUSAL, false><<<grid, SH::THREADS, 0, dev->stream>>>(A, B, C, bias, M, N, K, H, alpha);
    };
    auto go_small = [&](auto shape) {
        using SH = decltype(shape);
        if (CAUSAL || !split_pays(K)) return go(shape);
        auto kern = split_kernel<SH, AKC, BKC, EARLY>;
        err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Split<SH>::SMEM);
        if (err) return;
        dim3 grid((N + SH::BN - 1) / SH::BN, (M + SH::BM - 1) / SH::BM, batch * H);
        if constexpr (EARLY) err = launch_pdl(kern, grid, Split<SH>::THREADS, Split<SH>::SMEM, dev->stream, A, B, C, bias, M, N, K, H, alpha);
        else kern<<<grid, Split<SH>::THREADS, Split<SH>::SMEM, dev->stream>>>(A, B, C, bias, M, N, K, H, alpha);
    };
    const int sms = dev->prop.multiProcessorCount;
    if (N <= 32) go_small(Shape<64, 32>());
    else if (N > 64 && !rows_hint && tile_rows(M, N, batch * H, 128, sms) == 128) go(Shape<128, 128>());
    else if ((rows_hint ? rows_hint : tile_rows(M, N, batch * H, 64, sms)) == 128) go(Shape<128, 64>());
    else go_small(Shape<64, 64>());
    GRL_CUDA(err);
    GRL_LAUNCHED(name);
    return GRL_OK;
}

}  // namespace sgemm
}  // namespace grl
