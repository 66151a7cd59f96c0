// Linear projection y = x W^T + b on the Blackwell tensor cores (bf16 operands, fp32 accumulation and
// output), plus the exact fp32 form.
//
// Replaces ops::linear (cpp/src/ops/linear.cpp:20-82, shader fnn-linear) and the fused QKV projection
// (shaders/fused-qkv-projection.glsl:40-74: the same product with the packed [W_q; W_k; W_v] weight),
// i.e. the steps on either side of attention.  x is (M, K) row-major, W (N, K) row-major -- both K-major,
// which is what tcgen05.mma wants from shared memory -- and y (M, N).
//
// Two kernels:
//  linear_pair_kernel   products that fill the GPU: two SMs share one 256 x BN tile of y (cta_group::2), persistent.
//  linear_split_kernel  everything smaller, above all the few rows of a decode step, where the one pass over W bounds the
//                       time: W rows are the 128 rows of the product, x rows its columns, and the K range is cut over the
//                       CTAs of a cluster, which add their partial tiles through distributed shared memory.
// Every mbarrier wait is bounded.
#include "common.cuh"
#include "sgemm.cuh"
#include "sm100_ptx.cuh"
#include "tmem_ops.cuh"

namespace grl {
namespace lin {

using namespace sm100;

constexpr int BK = 64;             // one 128-byte swizzle row of bf16
constexpr int kThreads = 256;      // warp 0 TMA, warp 1 MMA, warp 2 TMEM, warp 3 idle, warps 4-7 epilogue (TMEM lanes 0..127)
constexpr int kPairThreads = 384;  // pair kernel: warps 8-11 are epilogue as well
constexpr int kSmemMax = 227 * 1024;

struct Args {
    const float* bias;     // (N) or NULL
    float* y;              // (M, N)
    int32_t* status;
    int M, N, K;
    int tile_rows;         // split kernel: x rows per tile (a multiple of 16, at most 256)
    int stages, splits;    // split kernel: ring stages, CTAs of a cluster along K
    int tma_store;         // pair kernel: rows of y start on 16-byte boundaries
    long long wait_limit;
};

__device__ __forceinline__ bool wait(uint32_t bar, uint32_t parity, volatile int* abort, const Args& a, int which) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    for (;;) {
        if (mbar_try_wait(bar, parity)) return true;
        if (*abort) return false;
        if (clock64() - t0 > a.wait_limit) {
            *abort = 1;
            if (a.status && atomicCAS(a.status, 0, GRL_ERR_TIMEOUT) == 0) {
                a.status[1] = (5 << 28) | which;
                a.status[2] = blockIdx.x;
                a.status[3] = blockIdx.y;
            }
            return false;
        }
    }
}

__device__ __forceinline__ bool wait_warp(uint32_t bar, uint32_t parity, volatile int* abort, const Args& a, int which) {
    return __all_sync(0xffffffffu, wait(bar, parity, abort, a, which));
}

__device__ __forceinline__ uint32_t instr_desc(int m, int n) {   // D f32, A and B bf16, both K-major
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// ---- the pair kernel.  A 128 x 128 tile per SM reads its operands from shared memory as fast as the tensor core eats them
// (64 cycles of reads and 64 of TMA writes per 64 cycles of products), which held a one-SM kernel at 1.0 PFLOP/s; a pair
// reads each half of W's tile once for both SMs.  A CTA stages its 128 rows of x and BN/2 rows of W; the even CTA's thread
// issues the products for both; the accumulator (128 lanes x BN columns in each SM) is double-buffered, so that one tile's
// epilogue runs under the next tile's products.  4096 x 4096 x 4096: 157 us in 128 x 128 tiles of one SM each, 117 us in pairs
// (1.17 PFLOP/s), cold L2.
template <int BN_>
struct Pair {
    static constexpr int BN = BN_, A_BYTES = 128 * BK * 2, B_BYTES = BN / 2 * BK * 2, STAGE = A_BYTES + B_BYTES;
    static constexpr int OUT_BYTES = 8 * 4096;                      // a 32 x 32 float box a warp on its way out
    static constexpr int NST = (kSmemMax - 2048 - OUT_BYTES) / STAGE;      // 6 or 8
    static constexpr int SMEM_OUT = NST * STAGE, SMEM_BAR = SMEM_OUT + OUT_BYTES, SMEM = SMEM_BAR + 256 + 1024;
};

template <int BN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1)
linear_pair_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmY,
                   const Args a) {
    using P = Pair<BN>;
    constexpr int NST = P::NST;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t* smem = smem_raw + (base - raw);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = cluster_ctarank();
    const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const int tiles_m = (a.M + 255) / 256, tiles_n = (a.N + BN - 1) / BN, tiles = tiles_m * tiles_n;
    const int n_k = (a.K + BK - 1) / BK;

    const uint32_t bars = base + P::SMEM_BAR;
    auto full = [&](int s) { return bars + (uint32_t)s * 8u; };
    auto empty = [&](int s) { return bars + (uint32_t)(NST + s) * 8u; };
    auto acc_full = [&](int i) { return bars + (uint32_t)(2 * NST + i) * 8u; };
    auto acc_empty = [&](int i) { return bars + (uint32_t)(2 * NST + 2 + i) * 8u; };
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + P::SMEM_BAR + (2 * NST + 4) * 8);
    volatile int* abort = reinterpret_cast<volatile int*>(smem + P::SMEM_BAR + (2 * NST + 4) * 8 + 4);

    if (tid == 0) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmX)) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmW)) : "memory");
        for (int s = 0; s < NST; ++s) { mbar_init(full(s), 1); mbar_init(empty(s), 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(acc_full(i), 1); mbar_init(acc_empty(i), 16); }     // 8 epilogue warps of 2 CTAs
        *abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_smem();
    }
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();                    // the peer's barriers exist
    tc_fence_after();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(tmem_slot);
    pdl_wait();

    // Tiles in groups of eight rows of tiles, walked column by column: the pairs at work at one time share both operands' tiles
    // in L2.
    auto place = [&](int t, int& tm, int& tn) {
        const int g = t / (8 * tiles_n), rows = min(8, tiles_m - 8 * g), r = t - g * 8 * tiles_n;
        tm = 8 * g + r % rows;
        tn = r / rows;
    };

    if (warp == 0) {
        if (lane == 0) {
            int it = 0;
            bool ok = true;
            for (int t = pair; t < tiles && ok; t += pairs) {
                int tm, tn;
                place(t, tm, tn);
                const int m0 = tm * 256 + (int)rank * 128, n0 = tn * BN + (int)rank * (BN / 2);
                for (int k = 0; k < n_k; ++k, ++it) {
                    const int s = it % NST, ph = it / NST;
                    if (ph > 0 && !wait(empty(s), (ph - 1) & 1, abort, a, NST + s)) { ok = false; break; }
                    const uint32_t dst = base + (uint32_t)s * P::STAGE, bar = cluster_map(full(s), 0);
                    if (rank == 0) mbar_expect_tx(full(s), 2 * P::STAGE);        // both CTAs' copies signal the even CTA
                    tma_load_2d_pair(dst, &tmX, k * BK, m0, bar);
                    tma_load_2d_pair(dst + P::A_BYTES, &tmW, k * BK, n0, bar);
                }
            }
            if (*abort && rank == 0) {     // copies already issued must land before the shared memory is released
                const long long t0 = clock64();
                for (int i = max(0, it - NST); i < it; ++i)
                    while (!mbar_try_wait(full(i % NST), (i / NST) & 1) && clock64() - t0 < a.wait_limit) {}
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {
            const uint32_t idesc = instr_desc(256, BN);
            int it = 0, n = 0;
            bool ok = true;
            for (int t = pair; t < tiles && ok; t += pairs, ++n) {
                const int acc = n & 1;
                if (n >= 2 && !wait_warp(acc_empty(acc), ((n >> 1) - 1) & 1, abort, a, 2 * NST + 2 + acc)) break;
                tc_fence_after();
                const uint32_t d = tmem + (uint32_t)acc * 256u;
                for (int k = 0; k < n_k; ++k, ++it) {
                    const int s = it % NST, ph = it / NST;
                    ok = wait_warp(full(s), ph & 1, abort, a, s);
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t a_lo = desc_lo(base + (uint32_t)s * P::STAGE, 16), b_lo = desc_lo(base + (uint32_t)s * P::STAGE + P::A_BYTES, 16);
#pragma unroll
                    for (int ks = 0; ks < BK / 16; ++ks)
                        mma_ss_pair(d, a_lo + (uint32_t)(ks * 32 >> 4), b_lo + (uint32_t)(ks * 32 >> 4), idesc, (k | ks) != 0);
                    mma_commit_pair(empty(s));       // in both CTAs: the stage is free once these products have read it
                }
                if (ok) mma_commit_pair(acc_full(acc));
            }
        }
    } else if (warp >= 4) {
        // ------------------------------------------------------------------ epilogue: TMEM -> (+ bias) -> global
        // Two warps take the same 32 lanes, every other 32 columns each: with one the epilogue, not the products, was the time of a
        // tile of short K (4096 x 128 x 4097 66 us).
        const int w = warp & 3, half = (warp - 4) >> 2;
        const uint32_t box = base + P::SMEM_OUT + (uint32_t)(warp - 4) * 4096u;
        int n = 0;
        for (int t = pair; t < tiles; t += pairs, ++n) {
            const int acc = n & 1;
            int tm, tn;
            place(t, tm, tn);
            if (!wait_warp(acc_full(acc), (n >> 1) & 1, abort, a, 2 * NST + acc)) break;
            if (t + pairs >= tiles) pdl_trigger();        // the next kernel may launch under the last epilogues
            tc_fence_after();
            const int row0 = tm * 256 + (int)rank * 128 + w * 32;
            const uint32_t t_addr = tmem + (uint32_t)acc * 256u + ((uint32_t)(w * 32) << 16);
#pragma unroll 1
            for (int c = half; c < BN / 32; c += 2) {
                uint32_t r[32];
                tmem_ld_x32_sync(t_addr + c * 32, r);
                const int col = tn * BN + c * 32;
                if (c + 2 >= BN / 32) {        // this warp's last read of this accumulator: the next tile's products may overwrite it
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_cluster(cluster_map(acc_empty(acc), 0));
                }
                if (row0 >= a.M || col >= a.N) continue;
                if (a.bias) {
                    const float bl = col + lane < a.N ? __ldg(a.bias + col + lane) : 0.f;
#pragma unroll
                    for (int e = 0; e < 32; ++e) r[e] = __float_as_uint(__uint_as_float(r[e]) + __shfl_sync(0xffffffffu, bl, e));
                }
                // 32 rows x 128 bytes under the 128-byte swizzle
                if (a.tma_store && lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                __syncwarp();
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    sts128(box + lane * 128 + ((q ^ (lane & 7)) << 4), make_uint4(r[4 * q], r[4 * q + 1], r[4 * q + 2], r[4 * q + 3]));
                if (a.tma_store) {
                    fence_async_smem();
                    __syncwarp();
                    if (lane == 0) {
                        tma_store_2d(&tmY, box, col, row0);
                        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                    }
                } else {       // rows of y off 16-byte boundaries: the warp stores 32 consecutive floats of one row at a time
                    __syncwarp();
                    const int rows = min(32, a.M - row0);
                    float* dst = a.y + (size_t)row0 * a.N + col + lane;
                    if (col + lane < a.N) {
#pragma unroll 16
                        for (int rr = 0; rr < 32; ++rr) {
                            const float v = lds32f(box + rr * 128 + (((lane >> 2) ^ (rr & 7)) << 4) + (lane & 3) * 4);
                            if (rr < rows) dst[(size_t)rr * a.N] = v;
                        }
                    }
                }
            }
        }
        if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    __syncwarp();
    cluster_sync();                    // neither CTA leaves while the other may still signal or read it
    tc_fence_after();
    if (warp == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
}

// ---- the split kernel.  Tile: 128 rows of W x tile_rows rows of x, y^T of it in TMEM (lane = column n of y, TMEM column = row m),
// so that few rows of x waste no product rows and a warp's store of one m is 32 consecutive floats of y.  Bound by the pass
// over W: two CTAs an SM keep about 200 KB in flight.
__global__ void __launch_bounds__(kThreads, 2)
linear_split_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW, const Args a) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t* smem = smem_raw + (base - raw);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int NST = a.stages, NT = a.tile_rows;
    const int w_bytes = 128 * BK * 2, stage_bytes = w_bytes + NT * BK * 2;
    const int part = a.splits > 1 ? (int)cluster_ctarank() : 0;
    const int n0 = (int)(blockIdx.x / a.splits) * 128, m0 = blockIdx.y * NT;
    const int n_k = (a.K + BK - 1) / BK, k0 = part * n_k / a.splits, k1 = (part + 1) * n_k / a.splits;
    const int tmem_cols = NT <= 32 ? 32 : NT <= 64 ? 64 : NT <= 128 ? 128 : 256;

    const uint32_t bars = base;        // barriers first (1 KiB), then the ring
    const uint32_t ring = base + 1024;
    auto full = [&](int s) { return bars + (uint32_t)s * 8u; };
    auto empty = [&](int s) { return bars + (uint32_t)(NST + s) * 8u; };
    const uint32_t acc_full = bars + 2 * NST * 8;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + (2 * NST + 1) * 8);
    volatile int* abort = reinterpret_cast<volatile int*>(smem + (2 * NST + 1) * 8 + 4);

    if (tid == 0) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmX)) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmW)) : "memory");
        for (int s = 0; s < NST; ++s) { mbar_init(full(s), 1); mbar_init(empty(s), 1); }
        mbar_init(acc_full, 1);
        *abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_smem();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(tmem_slot);
    pdl_wait();

    bool good = true;
    if (warp == 0) {
        if (lane == 0) {
            int issued = 0;
            for (int k = k0; k < k1; ++k) {
                const int i = k - k0, s = i % NST, ph = i / NST;
                if (ph > 0 && !wait(empty(s), (ph - 1) & 1, abort, a, NST + s)) break;
                const uint32_t dst = ring + (uint32_t)(s * stage_bytes);
                mbar_expect_tx(full(s), stage_bytes);
                tma_load_2d(dst, &tmW, k * BK, n0, full(s));
                tma_load_2d(dst + w_bytes, &tmX, k * BK, m0, full(s));
                issued = i + 1;
            }
            if (*abort) {     // copies already issued must land before the shared memory is released
                const long long t0 = clock64();
                for (int i = max(0, issued - NST); i < issued; ++i)
                    while (!mbar_try_wait(full(i % NST), (i / NST) & 1) && clock64() - t0 < a.wait_limit) {}
            }
        }
    } else if (warp == 1) {
        {
            const uint32_t idesc = instr_desc(128, NT);
            bool ok = true;
            for (int k = k0; k < k1 && ok; ++k) {
                const int i = k - k0, s = i % NST, ph = i / NST;
                ok = wait_warp(full(s), ph & 1, abort, a, s);
                if (!ok) break;
                tc_fence_after();
                const uint32_t w_lo = desc_lo(ring + (uint32_t)(s * stage_bytes), 16), x_lo = desc_lo(ring + (uint32_t)(s * stage_bytes + w_bytes), 16);
#pragma unroll
                for (int ks = 0; ks < BK / 16; ++ks)
                    mma_ss2(tmem, w_lo + (uint32_t)(ks * 32 >> 4), x_lo + (uint32_t)(ks * 32 >> 4), idesc, (i | ks) != 0);
                mma_commit(empty(s));                 // the stage is free once these products have read it
            }
            if (ok) mma_commit(acc_full);
        }
    } else if (warp >= 4) {
        good = wait_warp(acc_full, 0, abort, a, 2 * NST);
        pdl_trigger();        // the next kernel may launch under the epilogues; earlier it would take slots and sit unevenly
        tc_fence_after();
        const int w = warp & 3, n = n0 + w * 32 + lane;
        const uint32_t t_addr = tmem + ((uint32_t)(w * 32) << 16);
        const float b = a.bias && n < a.N ? __ldg(a.bias + n) : 0.f;
        float* part_tile = reinterpret_cast<float*>(smem + 1024) + w * 32 + lane;     // [m][128]; the ring is idle by now
        const int rows = min(NT, a.M - m0);
        if (good) {
            for (int c = 0; c < rows; c += 32) {
                uint32_t r[32];
                tmem_ld_x32_sync(t_addr + c, r);
#pragma unroll
                for (int e = 0; e < 32; ++e) {
                    if (c + e >= rows) break;
                    if (a.splits > 1) part_tile[(c + e) * 128] = __uint_as_float(r[e]);
                    else if (n < a.N) a.y[(size_t)(m0 + c + e) * a.N + n] = __uint_as_float(r[e]) + b;
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tmem_cols) : "memory");
    if (a.splits > 1) {
        __syncwarp();
        // every CTA of the cluster adds up its share of the rows, parts in ascending k
        cluster_sync();
        const int rows = min(NT, a.M - m0), lo = part * rows / a.splits, hi = (part + 1) * rows / a.splits;
        const bool vec = a.N % 4 == 0 && (uintptr_t)a.y % 16 == 0;
        if (!*abort) {
            for (int q = lo * 32 + tid; q < hi * 32; q += kThreads) {        // four columns of one row, all parts in flight
                float4 v[8];
#pragma unroll
                for (int p = 0; p < 8; ++p)
                    if (p < a.splits) v[p] = ld_cluster_f32x4(cluster_map(base + 1024u + (uint32_t)q * 16u, (uint32_t)p));
                float4 t = v[0];
#pragma unroll
                for (int p = 1; p < 8; ++p)
                    if (p < a.splits) { t.x += v[p].x; t.y += v[p].y; t.z += v[p].z; t.w += v[p].w; }
                const int n = n0 + (q & 31) * 4;
                if (a.bias) {
                    const float4 b = sgemm::load4(a.bias, n, a.N, (uintptr_t)a.bias % 16 == 0);
                    t.x += b.x; t.y += b.y; t.z += b.z; t.w += b.w;
                }
                float* dst = a.y + (size_t)(m0 + (q >> 5)) * a.N + n;
                if (vec && n + 3 < a.N) *reinterpret_cast<float4*>(dst) = t;
                else {
                    if (n < a.N) dst[0] = t.x;
                    if (n + 1 < a.N) dst[1] = t.y;
                    if (n + 2 < a.N) dst[2] = t.z;
                    if (n + 3 < a.N) dst[3] = t.w;
                }
            }
        }
        __syncwarp();
        cluster_sync();        // a CTA leaves only when nobody reads its part any more
    }
}

// Exact fp32 form for small products: a warp takes one row of W (one output column) and multiplies it with up to eight rows of
// x, all in 16-byte pieces (x stays in L1).  As long as its warps are one wave on the GPU this beats the 64 x 64 tiles of
// sgemm.cuh, of which there are too few then: 9 x 768 x 3000 14.4 us (tiles 26.7), 64 x 256 x 1024 12.3 (12.3), 48 x 700 x 700
// 14.4 (24.6); past the wave 32 x 768 x 3000 34.9 (26.7).
constexpr int kGemvRows = 8;
constexpr int kGemvWarps = 56;     // per SM, of the 64 it holds
template <int MR>
__global__ void __launch_bounds__(256) linear_f32_rows_kernel(const float* __restrict__ x, const float* __restrict__ w,
                                                              const float* __restrict__ bias, float* __restrict__ y, int M, int K, int N,
                                                              int vec) {
    const int n = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (n >= N) return;
    x += (size_t)blockIdx.y * MR * K;
    y += (size_t)blockIdx.y * MR * N;
    M -= blockIdx.y * MR;
    const float* wr = w + (size_t)n * K;
    float acc[MR];
#pragma unroll
    for (int m = 0; m < MR; ++m) acc[m] = 0.f;
#pragma unroll 4
    for (int k = lane * 4; k < K; k += 128) {
        const float4 a = sgemm::load4(wr, k, K, vec);
#pragma unroll
        for (int m = 0; m < MR; ++m) {
            if (m >= M) break;
            const float4 b = sgemm::load4(x + (size_t)m * K, k, K, vec);
            acc[m] = fmaf(a.x, b.x, acc[m]); acc[m] = fmaf(a.y, b.y, acc[m]);
            acc[m] = fmaf(a.z, b.z, acc[m]); acc[m] = fmaf(a.w, b.w, acc[m]);
        }
    }
    const float bn = bias ? bias[n] : 0.f;
#pragma unroll
    for (int m = 0; m < MR; ++m) {
        if (m >= M) break;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc[m] += __shfl_xor_sync(0xffffffffu, acc[m], o);
        if (lane == 0) y[(size_t)m * N + n] = acc[m] + bn;
    }
}

static int linear_f32(grl_device* dev, const float* x, const float* w, const float* bias, float* y, int M, int K, int N) {
    const long long warps = (long long)((M + kGemvRows - 1) / kGemvRows) * ((N + 7) / 8) * 8;
    if (M > kGemvRows && warps > (long long)kGemvWarps * dev->prop.multiProcessorCount)
        return sgemm::launch<true, true>(dev, sgemm::operand(x, 0, 0, K), sgemm::operand(w, 0, 0, K), sgemm::Output{y, 0, 0, N}, bias, M,
                                         N, K, 1, 1, 1.f, "linear_f32");
    const int vec = K % 4 == 0 && (uintptr_t)x % 16 == 0 && (uintptr_t)w % 16 == 0;
    const dim3 grid((unsigned)((N + 7) / 8), (unsigned)((M + kGemvRows - 1) / kGemvRows));
    if (M == 1) linear_f32_rows_kernel<1><<<grid, 256, 0, dev->stream>>>(x, w, bias, y, M, K, N, vec);
    else if (M <= 4) linear_f32_rows_kernel<4><<<grid, 256, 0, dev->stream>>>(x, w, bias, y, M, K, N, vec);
    else linear_f32_rows_kernel<kGemvRows><<<grid, 256, 0, dev->stream>>>(x, w, bias, y, M, K, N, vec);
    GRL_LAUNCHED("linear_f32_rows_kernel");
    return GRL_OK;
}

static int make_map(grl_device* dev, CUtensorMap* tm, const void* ptr, int rows, int cols, int box_rows, int box_cols, int elem_bytes) {
    TmapKey k{};
    k.ptr = ptr; k.rank = 2; k.swizzle_128b = 1; k.bytes = elem_bytes == 4 ? 4 : 0;
    k.dims[0] = (uint64_t)cols; k.dims[1] = (uint64_t)rows; k.strides[0] = (uint64_t)cols * elem_bytes;
    k.box[0] = (uint32_t)box_cols; k.box[1] = (uint32_t)box_rows;
    return get_tensor_map(dev, k, tm);
}

template <int BN>
static int launch_pair(grl_device* dev, const void* x, const void* w, Args a) {
    using P = Pair<BN>;
    CUtensorMap tx, tw, ty;
    int rc = make_map(dev, &tx, x, a.M, a.K, 128, BK, 2);
    if (!rc) rc = make_map(dev, &tw, w, a.N, a.K, BN / 2, BK, 2);
    a.tma_store = a.N % 4 == 0 && (uintptr_t)a.y % 16 == 0;
    ty = tx;
    if (!rc && a.tma_store) rc = make_map(dev, &ty, a.y, a.M, a.N, 32, 32, 4);
    if (rc) return rc;
    static bool attr_set[64] = {};
    if (!attr_set[dev->ordinal & 63]) {
        GRL_CUDA(cudaFuncSetAttribute(linear_pair_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, P::SMEM));
        attr_set[dev->ordinal & 63] = true;
    }
    const int tiles = (a.M + 255) / 256 * ((a.N + BN - 1) / BN), pairs = dev->prop.multiProcessorCount / 2;
    GRL_CUDA(launch_pdl(linear_pair_kernel<BN>, 2 * (tiles < pairs ? tiles : pairs), kPairThreads, P::SMEM, dev->stream, tx, tw, ty, a));
    GRL_LAUNCHED("linear_pair_kernel");
    return GRL_OK;
}

// Stands in for linear_split_kernel when max_active_clusters is asked: the occupancy of a kernel that allocates TMEM is given
// as one CTA an SM whatever it allocates.
__global__ void __launch_bounds__(kThreads, 2) placement_probe() {}

static int launch_split(grl_device* dev, const void* x, const void* w, Args a) {
    // x rows per tile: all of them up to 128 (W is then read once), tiles of 128 beyond
    a.tile_rows = a.M <= 128 ? (a.M + 15) / 16 * 16 : 128;
    const int n_k = (a.K + BK - 1) / BK;
    const int tiles = (a.N + 127) / 128 * ((a.M + a.tile_rows - 1) / a.tile_rows);
    const int stage = (128 + a.tile_rows) * BK * 2;
    // three CTAs an SM while each still has three stages (two beyond 64 rows): one's start and end run under the others' copies
    const int per_sm = a.tile_rows <= 64 ? 3 : 2;
    a.stages = (kSmemMax / per_sm - 3072) / stage;
    if (a.stages > n_k) a.stages = n_k;
    int smem = a.stages * stage;
    if (smem < a.tile_rows * 512) smem = a.tile_rows * 512;      // the partial tile of a split
    smem += 2048;
    static bool attr_set[64] = {};
    if (!attr_set[dev->ordinal & 63]) {
        GRL_CUDA(cudaFuncSetAttribute(linear_split_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax));
        GRL_CUDA(cudaFuncSetAttribute(placement_probe, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax));
        attr_set[dev->ordinal & 63] = true;
    }
    // K cut as far as one wave of clusters goes (a cluster too many is a second wave: 32 x 4096 x 12288 in clusters of 3 at two
    // CTAs an SM took 31 us for 22), at least four slices a CTA (measured, us at 1 / 2 / 4 / 8 parts: 32 x 4096 x 4096
    // 28 / 18.6 / 13.1 / 11.2, 32 x 4096 x 12288 32 / 22.9 / 21.5 / 26.8, 128 x 4096 x 4096 33 / 23.5 / 17.5 / 16.5)
    a.splits = 8;
    while (a.splits > 1 && (n_k < 4 * a.splits || tiles > max_active_clusters(dev, (const void*)placement_probe, kThreads, smem, a.splits))) a.splits /= 2;
    CUtensorMap tx, tw;
    int rc = make_map(dev, &tx, x, a.M, a.K, a.tile_rows, BK, 2);
    if (!rc) rc = make_map(dev, &tw, w, a.N, a.K, 128, BK, 2);
    if (rc) return rc;
    dim3 grid((a.N + 127) / 128 * a.splits, (a.M + a.tile_rows - 1) / a.tile_rows);
    GRL_CUDA(launch_pdl_cluster(linear_split_kernel, grid, kThreads, smem, dev->stream, a.splits, tx, tw, a));
    GRL_LAUNCHED("linear_split_kernel");
    return GRL_OK;
}

}  // namespace lin
}  // namespace grl

using namespace grl;

extern "C" int grl_linear(grl_device* dev, const void* x, const void* w, const float* bias, float* y, int m, int k, int n,
                          int in_dtype) {
    GRL_REQUIRE(dev && x && w && y, "NULL argument");
    GRL_REQUIRE(m > 0 && k > 0 && n > 0, "bad shape (%d,%d,%d)", m, k, n);
    GRL_REQUIRE(in_dtype == GRL_F32 || in_dtype == GRL_BF16, "unknown in_dtype");
    DeviceGuard g(dev->ordinal);
    if (in_dtype == GRL_F32)
        return lin::linear_f32(dev, static_cast<const float*>(x), static_cast<const float*>(w), bias, y, m, k, n);
    GRL_REQUIRE(k % 8 == 0, "the tensor-core projection needs the inner dimension to be a multiple of 8 (got %d): rows must "
                            "start on 16-byte boundaries for TMA", k);
    GRL_REQUIRE(((uintptr_t)x % 16 == 0) && ((uintptr_t)w % 16 == 0) && ((uintptr_t)y % 8 == 0), "x, w must be 16-byte aligned");
    lin::Args a{};
    a.bias = bias; a.y = y; a.status = dev->d_status; a.M = m; a.N = n; a.K = k; a.wait_limit = dev->wait_limit_cycles;
    dev->status_dirty = true;
    // The pair kernel wants more than one of its two 128-row halves and tiles for half the pairs; below that the split kernel
    // has more SMs at work.  It also takes a short K whose rows of y are off 16-byte boundaries: the time is that of the stores
    // then, which its accumulators (lane = column of y) need no transpose for: us, pair / split, 4096 x 64 x 12287 113 / 63, 4096 x 128 x
    // 4097 41 / 28, 4096 x 256 x 4097 43 / 37, but 4096 x 600 x 2047 25 / 31; as long as its tiles are one wave of two CTAs an SM, a K
    // up to 640 as well: 576 x 640 x 6598 19.0 / 12.2, 2000 x 304 x 2001 13.3 / 11.0, 200 x 400 x 4999 9.2 / 9.6.
    const int pairs = dev->prop.multiProcessorCount / 2;
    auto waves = [&](int bn) { return ((long long)((m + 255) / 256) * ((n + bn - 1) / bn) + pairs - 1) / pairs; };
    const bool one_wave = (long long)((m + 127) / 128) * ((n + 127) / 128) <= 4 * pairs;
    if (m <= 128 || (n % 4 != 0 && (k <= 256 || (k <= 640 && one_wave))) || (long long)((m + 255) / 256) * ((n + 127) / 128) < pairs / 2)
        return lin::launch_split(dev, x, w, a);
    // the tile whose waves cost least: a wave of 256 / 192 / 128 columns took 29.7 / 26.3 / 22.7 us at K = 4096 (narrower tiles are
    // bound by shared memory).  A wave of short K is bound by its stores instead, where these costs are not the right ones: with K from
    // 64 to 1024 the choice is within 3 % of the best tile at three in four of 35 shapes and 3 to 7 % behind it, mostly 192 columns, at the others
    // (us, chosen / 192: 4096 x 256 x 2560 25.6 / 23.7, 4096 x 512 x 6144 42.8 / 40.1, 4096 x 128 x 6144 35.4 / 33.0).
    const long long c256 = waves(256) * 297, c192 = waves(192) * 263, c128 = waves(128) * 227;
    if (c256 <= c192 && c256 <= c128) return lin::launch_pair<256>(dev, x, w, a);
    return c192 <= c128 ? lin::launch_pair<192>(dev, x, w, a) : lin::launch_pair<128>(dev, x, w, a);
}
