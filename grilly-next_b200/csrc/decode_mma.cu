// GQA decode over the paged bf16 cache, head_dim 128 or 64, pages of 64, 32 or 16 tokens: the fast path.
//
// Replaces shaders/gqa-attention.glsl:34-130 like decode_splitkv.cu, for the geometry of the
// benchmark configurations.  One CTA owns (split, kv head, sequence); producer warps (one over the bf16 cache) stream
// whole (page, kv head) slabs -- 16 KiB of K and 16 KiB of V, each contiguous in HBM -- into a
// shared-memory ring with TMA (128-byte swizzle, mbarrier complete_tx); compute
// warps in groups of four (one group over the bf16 cache) each take 16 of a stage's 64 tokens and run QK^T and PV on tensor cores
// (mma.sync m16n8k16, the group's query heads padded to the 16-row operand, q split into
// bf16 hi+lo so that its fp32 precision survives), with a private fp32 online softmax in the
// exp2 domain.  K and V cross HBM -> SM exactly once; the compute warps' partials are merged in
// shared memory and leave the CTA as (O un-normalised, m, l), the layout lse_merge_kernel reads.  Warps, ring stages and the order of
// their waits in each of the three forms: decode_ring.h.  Splits of one head that fit a
// thread-block cluster merge through its shared memory instead, and a launch sets up its ring and barriers under the kernel before
// it.  Append + decode step: 1 sequence x 8 kv heads x 1001 tokens 19.4 us before, 9.9 now (latency); 32 x 8 x 4096 93 and 85 us
// (HBM); 1 x 8 x 131072 104 and 94 us (HBM; the decode alone 90), quantised 107 and 59 us (instructions: 444 a 16-token slice).
//
// The same kernel, in two forms for the quantised cache (GRL_FP8_INT4: FP8-E4M3 keys, INT4 values, one float16 scale
// per 32 key elements, cpp/src/ops/kv_cache.cpp:272-399 and :500-577): four compute and two producer warps, two CTAs an SM, or twelve
// and four, one CTA an SM.  It streams 12.5 KiB per (page, kv head) instead
// of 32 and dequantises in registers: key bytes become f16 by three integer operations per pair (every code is an
// exact f16 once divided by 256), the four scale groups of a head accumulate separately and are combined with 1/scale per
// token; value nibbles become f16 by one logic operation and one subtraction per pair (1024 + n or 64 + n in the
// mantissa, minus the offset and the code's bias), with 1/scale folded into P.  The contraction indices of both
// products are permuted so that every operand register is a plain 32-bit piece of what was loaded.
#include <cuda.h>
#include <cuda_fp16.h>

#include <type_traits>

#include "common.cuh"
#include "decode_plan.h"
#include "decode_ring.h"

namespace grl {
namespace dmma {

constexpr int P = 64;               // tokens per ring stage: one 64-token page, or two / four smaller ones side by side
constexpr int D = 128;              // head_dim of the quantised instance (the bf16 instances carry theirs as HD)
// The shared-memory ring of an instance.  After the ring: 256 bytes of barriers and flags, 128 of block table a producer, 256 a compute
// warp over the quantised cache (1/scale of its 16 tokens x 4 groups), 1 KiB of slack for the 1024-byte alignment of the ring.
template <int FORM, int HD> struct Ring {
    static constexpr int SLAB = P * HD * 2;             // 64 tokens of K (or V) for one kv head: 16 KiB at head_dim 128
    static constexpr int STAGE = 2 * SLAB;              // K then V
};
constexpr int QK_BYTES = P * D;          // 8 KiB of key bytes per 64 tokens of a kv head
constexpr int QV_BYTES = P * D / 2;      // 4 KiB of packed value nibbles
struct QuantRing {
    static constexpr int SLAB = 0;
    static constexpr int STAGE = 13 * 1024;  // keys at 0, values at 8 KiB, scales at 12 KiB
};
template <> struct Ring<QUANT_PAIR, 128> : QuantRing {};
template <> struct Ring<QUANT_WIDE, 128> : QuantRing {};
template <int FORM, int HD> struct Smem {
    static constexpr int BAR = Stages<FORM, HD>::NST * Ring<FORM, HD>::STAGE;
    static constexpr int TOTAL = BAR + 256 + 128 * Warps<FORM>::PROD + (FORM != BF16 ? 256 * Warps<FORM>::COMPUTE : 0) + 1024;
};
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kEmpty = -1e30f;

struct Args {
    const int32_t* block_table;
    const int32_t* seq_lens;
    const uint8_t* v_q;         // quantised cache: the value pool (plain bulk copies; the key pool goes through tmK)
    const uint16_t* scales;     // quantised cache: float16 bit patterns, (rows, D/32)
    const float* q;
    float* part;
    float* out;
    int32_t* status;
    int B, Hq, Hkv, max_pages, n_splits, group;
    int page, ppt;          // tokens per page (64, 32 or 16) and pages per 64-token stage
    float scale;
    int direct;
    // fused merge: the last CTA of a (sequence, kv head) to arrive merges the head's splits
    int fuse;               // 0: leave the splits to lse_merge_kernel
    int32_t* counters;      // arrival counters, zero between launches; [kDoneSlot] counts finished heads
    float* partial_out;     // != NULL: merged rows leave un-normalised as [O | m | l]
    float* scores_out;      // != NULL: (B*Hq, scores_ld) scaled scores, natural-log domain
    int scores_ld;
    PeerExchange x;         // x.world > 1: the merged rows are exchanged with the peers and merged again
    long long wait_limit;   // cycle budget of every mbarrier wait
    int alone;              // 1: one CTA an SM, and the next kernel starts after this one (decode_plan)
    int cluster;            // > 1: CTAs of a thread-block cluster; that many splits of a head merge through its shared memory
    int pps_hint;           // stages per split of a sequence of the longest length: what the first block-table read assumes
};
constexpr int kAloneSmem = 116 * 1024;      // dynamic shared memory of which an SM (228 KiB, 1 KiB reserved a CTA) does not hold two
constexpr int kDoneSlot = grl_device::kCounterSlots;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// The same test, but the thread may stay suspended in hardware for up to hint_ns while the phase is incomplete: a
// waiter that is far ahead of what it waits for then takes no issue slots.
__device__ __forceinline__ bool mbar_try_wait_suspend(uint32_t bar, uint32_t parity, uint32_t hint_ns) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(bar), "r"(parity), "r"(hint_ns) : "memory");
    return ok != 0;
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* tm, int c0, int c1, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(tm)), "r"(c0), "r"(c1), "r"(bar) : "memory");
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void cluster_sync() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_map(uint32_t addr, int rank) {   // this address in the shared memory of CTA `rank`
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ float4 ld_cluster_f32x4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ float ld_cluster_f32(uint32_t addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}
// D += A * B with A rows 8..15 all zero (a1 = a3 = 0): the query heads of one GQA group fill rows 0..7.
__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a2, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%5}, {%7,%8}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(0u), "r"(a2), "r"(b0), "r"(b1));
}
// Plain (untiled) bulk copy global -> shared, 16-byte aligned on both sides, completing on an mbarrier.
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(__cvta_generic_to_global(src)), "r"(bytes), "r"(bar) : "memory");
}
// All sixteen rows of A live (the transposed value product: rows are head_dim elements, columns query heads).
__device__ __forceinline__ void mma_f16_full(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                             uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// The same with C zero.
__device__ __forceinline__ void mma_f16_zero(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ uint32_t pack_f16(float lo, float hi) {
    __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}
// FP8-E4M3 codes to f16x2 by integer operations (the conversion instruction runs on the slow special-function
// pipe).  A code s eeee mmm becomes the f16 s 0eeee mmm0000000, which is the code's value (the reference's decoder,
// kv_cache.cpp:540-552: 2^(e-7) (1 + m/8), or m 2^-9 for e = 0) divided by 256, denormals included; the factor is
// folded into q.  Bytes (0, 2) of a word make one register, bytes (1, 3) the other: the byte permute puts each code
// under a copy of its sign, the shift brings exponent and mantissa into place and the sign to bit 15, the mask
// clears what the shift dragged along.
__device__ __forceinline__ uint32_t prmt(uint32_t w, uint32_t selector) {   // a selector digit >= 8 replicates the byte's sign
    uint32_t r;
    asm("prmt.b32 %0, %1, %1, %2;" : "=r"(r) : "r"(w), "r"(selector));
    return r;
}
__device__ __forceinline__ uint32_t e4m3_pair02_f16x2(uint32_t w) { return (prmt(w, 0xA280u) << 7) & 0xBF80BF80u; }
__device__ __forceinline__ uint32_t e4m3_pair13_f16x2(uint32_t w) { return (prmt(w, 0xB391u) << 7) & 0xBF80BF80u; }
// Value codes to f16x2 (low half: even token of the pair, high half: odd token): the nibble is placed in the mantissa of
// 1024 (bits 0-3) or of 64 (bits 4-7) by one three-input operation (mask and literal: the compiler makes two of it), and the
// offset plus the code's bias of 8 is subtracted, which is exact in f16.
__device__ __forceinline__ uint32_t and_or(uint32_t w, uint32_t mask, uint32_t bits) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(w), "r"(mask), "r"(bits));
    return r;
}
__device__ __forceinline__ uint32_t nib_lo(uint32_t w) {
    const uint32_t v = and_or(w, 0x000F000Fu, 0x64006400u), off = 0x64086408u;    // 1032, 1032
    __half2 r = __hsub2(*reinterpret_cast<const __half2*>(&v), *reinterpret_cast<const __half2*>(&off));
    return *reinterpret_cast<uint32_t*>(&r);
}
__device__ __forceinline__ uint32_t nib_hi(uint32_t w) {
    const uint32_t v = and_or(w, 0x00F000F0u, 0x54005400u), off = 0x54805480u;    // 72, 72
    __half2 r = __hsub2(*reinterpret_cast<const __half2*>(&v), *reinterpret_cast<const __half2*>(&off));
    return *reinterpret_cast<uint32_t*>(&r);
}
// 1/scale from the stored float16 bit pattern, as the reference's decode forms it (kv_cache.cpp:517-533): bits moved
// into a float32, not converted; a scale that is not positive gives 1.
__device__ __forceinline__ float inv_scale_bits(uint32_t h) {
    // exponent and mantissa under the float32 exponent field are the value times 2^-112, subnormal scales included
    const float sc = __uint_as_float((h & 0x7FFFu) << 13) * 5.192296858534828e+33f;
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(sc));     // within an ulp of the reference's quotient
    return (h - 1u) < 0x7FFFu ? r : 1.0f;
}
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}

struct Ctx {
    uint32_t bars;
    volatile int* abort;
    int32_t* status;
    long long limit;
};
// relaxed: the waiter is ahead of its consumers by the whole ring (the producer lane): it waits suspended instead of
// competing for issue slots with the compute warp that shares its scheduler.
__device__ __forceinline__ bool wait_bar(const Ctx& c, int bar, uint32_t parity, bool relaxed = false) {
    const uint32_t addr = c.bars + bar * 8;
    if (mbar_try_wait(addr, parity)) return true;
    const long long t0 = clock64();
    for (;;) {
        if (relaxed ? mbar_try_wait_suspend(addr, parity, 20000u) : mbar_try_wait(addr, parity)) return true;
        if (*c.abort) return false;
        if (clock64() - t0 > c.limit) {
            *c.abort = 1;
            if (c.status && atomicCAS(c.status, 0, GRL_ERR_TIMEOUT) == 0) {
                c.status[1] = (2 << 28) | bar;
                c.status[2] = blockIdx.x;
                c.status[3] = blockIdx.y | (blockIdx.z << 16);
            }
            return false;
        }
    }
}

// byte offset inside a slab of element (token row, column d): two 64-column halves, 128-byte swizzle
__device__ __forceinline__ uint32_t slab_off(int row, int d) {
    return (uint32_t)((d >> 6) * (P * 128) + row * 128 + ((((d & 63) >> 3) ^ (row & 7)) << 4));
}

template <int FORM, int HD>
__global__ void __launch_bounds__(Warps<FORM>::THREADS, Warps<FORM>::CTAS)
decode_mma_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, const Args a) {
    constexpr bool QUANT = FORM != BF16;
    static_assert(HD == 128 || (HD == 64 && !QUANT), "head_dim 128, or 64 over the bf16 cache");
    static_assert(FORM == QUANT_WIDE || Smem<FORM, HD>::TOTAL <= kAloneSmem, "the wider allocation holds the ring");
    constexpr int D = HD;
    constexpr int NST = Stages<FORM, HD>::NST, STAGE = Ring<FORM, HD>::STAGE, SMEM_BAR = Smem<FORM, HD>::BAR;
    constexpr int SLAB = Ring<FORM, HD>::SLAB;
    constexpr int COMPUTE = Warps<FORM>::COMPUTE, PROD = Warps<FORM>::PROD, kThreads = Warps<FORM>::THREADS;
    static_assert(2 * NST * 8 + 16 <= 256, "barrier block");
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_addr = smem_u32(smem_raw);
    const uint32_t base = (raw_addr + 1023u) & ~1023u;
    uint8_t* smem = smem_raw + (base - raw_addr);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int split = blockIdx.x, kvh = blockIdx.y, b = blockIdx.z;
    const int32_t* bt = a.block_table + (size_t)b * a.max_pages;

    int* abort_flag = reinterpret_cast<int*>(smem + SMEM_BAR + 2 * NST * 8);
    Ctx ctx{base + SMEM_BAR, abort_flag, a.status, a.wait_limit};
    auto full = [&](int s) { return ctx.bars + (uint32_t)s * 8u; };
    auto empty = [&](int s) { return ctx.bars + (uint32_t)(NST + s) * 8u; };
    if (tid == 0) {
        for (int s = 0; s < NST; ++s) { mbar_init(full(s), 1); mbar_init(empty(s), 4); }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmK)) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmV)) : "memory");
    }
    __syncthreads();
    // everything above ran beside the kernel before this one (the append of the step's token); nothing below may
    pdl_wait();
    const int32_t raw_len = a.seq_lens[b];
    // the split's first block-table entries, read beside the length on the guess that this sequence is the longest
    const int bt_guess = split * a.pps_hint * a.ppt;
    int32_t* bt_s = reinterpret_cast<int32_t*>(smem + SMEM_BAR + 256 + 128 * (warp >= COMPUTE ? warp - COMPUTE : 0));      // 32 entries a producer
    if (warp >= COMPUTE) bt_s[lane] = bt[min(bt_guess + lane, a.max_pages - 1)];
    const int len = max(0, min(raw_len, a.max_pages * a.page));   // never past the block table
    const int n_pages = (len + P - 1) / P;        // 64-token stages ("pages" below)
    const int pps = (n_pages + a.n_splits - 1) / a.n_splits;
    const int p_begin = min(n_pages, split * pps), p_end = min(n_pages, (split + 1) * pps);

    const int g = lane >> 2, t4 = lane & 3;      // mma row / column-pair index of this lane
    float o[D / 8][4];
    float m_run = kEmpty, l_run = 0.f;
#pragma unroll
    for (int i = 0; i < D / 8; ++i) { o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f; }

    if (warp >= COMPUTE) {
        // ------------------------------------------------------------------ producers
        __syncwarp();
        int issued = 0;
        const int pr = warp - COMPUTE;
        auto issue = [&](uint32_t dst, int page, int j, int s) {
            const int blk = page * a.Hkv + kvh;
            if constexpr (QUANT) {
                // rows of 128 key bytes under the 128-byte swizzle; a page's value and scale blocks are contiguous
                tma_load_2d(dst + j * a.page * 128, &tmK, 0, blk * a.page, full(s));
                bulk_load(dst + QK_BYTES + j * a.page * (D / 2), a.v_q + (size_t)blk * a.page * (D / 2), a.page * (D / 2), full(s));
                bulk_load(dst + QK_BYTES + QV_BYTES + j * a.page * (D / 16), a.scales + (size_t)blk * a.page * (D / 32),
                          a.page * (D / 16), full(s));
            } else {
#pragma unroll
                for (int c0 = 0; c0 < D; c0 += 64) {        // 64-column boxes (128 bytes: the swizzle span)
                    tma_load_2d(dst + (c0 / 64) * (P * 128) + j * a.page * 128, &tmK, c0, blk * a.page, full(s));
                    tma_load_2d(dst + SLAB + (c0 / 64) * (P * 128) + j * a.page * 128, &tmV, c0, blk * a.page, full(s));
                }
            }
        };
        constexpr uint32_t TOKEN_BYTES = QUANT ? D + D / 2 + D / 16 : D * 4;
        bool ok = true;
        // the pages of stage p that hold tokens of the sequence (all of them but in the last stage); rows of the stage that no copy
        // fills keep what they held: their tokens are past the length and masked
        auto pages_of = [&](int p) { return min(a.ppt, (len - p * P + a.page - 1) / a.page); };
        if (a.ppt <= 2) {
            // One or two pages a stage: lane 0 alone, in a shorter loop for one page a stage where that chain bounds the stream of
            // a CTA alone on its SM (131072 tokens x 8 heads, append + decode 97.8 -> 94.2 us; two CTAs an SM, 32 x 8 x 4096, 85.0 -> 85.6).
            auto page_of = [&](int i) { return (unsigned)(i - bt_guess) < 32u ? bt_s[i - bt_guess] : bt[i]; };
            auto walk = [&](auto one) {
                for (int p = p_begin + pr; p < p_end; p += PROD) {
                    const int i = p - p_begin, s = i % NST, it = i / NST;
                    if (it > 0 && !wait_bar(ctx, NST + s, (it - 1) & 1, true)) break;
                    if constexpr (decltype(one)::value) {
                        mbar_expect_tx(full(s), P * TOKEN_BYTES);
                        issue(base + (uint32_t)s * STAGE, page_of(p), 0, s);
                    } else {
                        const int np = pages_of(p);
                        mbar_expect_tx(full(s), (uint32_t)np * a.page * TOKEN_BYTES);
                        for (int j = 0; j < np; ++j) issue(base + (uint32_t)s * STAGE, page_of(p * a.ppt + j), j, s);
                    }
                    issued = i + 1;
                }
            };
            if (lane == 0) {
                if (a.ppt == 1 && (a.alone || FORM == QUANT_WIDE)) walk(std::true_type{});
                else walk(std::false_type{});
            }
        } else {
            // Four pages a stage: lane l holds the block-table entry of page first + l and issues that page's copies; the next 32
            // entries are read while these are used up (16-token pages, 131072 tokens x 8 heads: 143 -> 115 us, append + decode).
            int first = p_begin * a.ppt;
            int entry = first == bt_guess ? bt_s[lane] : bt[min(first + lane, a.max_pages - 1)];
            int entry_next = bt[min(first + 32 + lane, a.max_pages - 1)];
            for (int p = p_begin + pr; p < p_end; p += PROD) {
                const int i = p - p_begin, s = i % NST, it = i / NST;
                if (p * a.ppt - first >= 32) {
                    first += 32;
                    entry = entry_next;
                    entry_next = bt[min(first + 32 + lane, a.max_pages - 1)];
                }
                ok = lane != 0 || it == 0 || wait_bar(ctx, NST + s, (it - 1) & 1, true);
                if (!__all_sync(0xffffffffu, ok)) break;
                const int np = pages_of(p);
                if (lane == 0) mbar_expect_tx(full(s), (uint32_t)np * a.page * TOKEN_BYTES);
                __syncwarp();
                const int j = lane - (p * a.ppt - first);
                if (j >= 0 && j < np) issue(base + (uint32_t)s * STAGE, entry, j, s);
                __syncwarp();
                issued = i + 1;
            }
        }
        if (lane == 0) bt_s[0] = issued;
    } else if constexpr (QUANT) {
        // ------------------------------------------------------------------ compute over the quantised cache
        // Element permutation of the two products.  QK^T: k-step (grp, w) of lane (g, t4) covers elements
        // 32 grp + 8 t4 + 4 w + {0,2 | 1,3} = one 32-bit word of key bytes.  PV runs transposed (rows elements,
        // columns heads): row g | g + 8 of tile (grp, j) is element 32 grp + 4 g + 2 j | + 1, and the k index
        // pairs (2 t4, 2 t4 + 1 | + 8) are the token pairs (8 warp + 2 t4 | + 1) of the value block (quant_v_off).
        // Tokens: column n of score tile nt is token 2 n + nt of the warp's 16 (so that a half-warp's key loads hit
        // all banks once), and a lane's four scores are the four consecutive tokens 4 t4 .. 4 t4 + 3.
        const int qh0 = kvh * a.group;
        // A of a group's two k-steps is one operand: rows 0..7 the query heads of step w = 0, rows 8..15 those of w = 1.  A product's
        // other half goes unused, as the rows beyond the heads did before, and no operand needs a zero register moved in beside the
        // two live ones: with the nibbles' three-input operation 505 -> 444 instructions a slice, append + decode of 131072 tokens x
        // 8 heads 64.4 -> 59.6 us, 32 sequences x 4096 67.5 -> 61.8.
        uint32_t qf[4][4];
        {
            const float sc = a.scale * kLog2e * 256.f;      // the key registers hold code / 256
            const float* qrow = a.q + ((size_t)b * a.Hq + qh0 + g) * D;
            const bool live = g < a.group;
#pragma unroll
            for (int ks = 0; ks < 8; ++ks) {
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                if (live) v = *reinterpret_cast<const float4*>(qrow + 32 * (ks >> 1) + 8 * t4 + 4 * (ks & 1));
                qf[ks >> 1][ks & 1] = pack_f16(v.x * sc, v.z * sc);            // with the key codes of bytes 0 and 2 of the word
                qf[ks >> 1][2 + (ks & 1)] = pack_f16(v.y * sc, v.w * sc);      // bytes 1 and 3
            }
        }
        float* inv_w = reinterpret_cast<float*>(smem + SMEM_BAR + 256 + 128 * PROD) + warp * 64;   // [16 tokens][4 groups]
        bool ok = true;
        constexpr int GROUPS = Warps<FORM>::GROUPS;
        const int slice = warp & 3;             // which 16 tokens of a stage
        int s = (warp >> 2) - GROUPS;           // ring slot; the parity of its phase
        uint32_t parity = 0;
        for (int p = p_begin + (warp >> 2); p < p_end; p += GROUPS) {
            s += GROUPS;
            if (s >= NST) { s -= NST; parity ^= 1u; }
            // one try first: the bounded wait's clock and branches only where the slot is not there yet
            if (!__all_sync(0xffffffffu, mbar_try_wait(ctx.bars + s * 8, parity)))
                ok = __all_sync(0xffffffffu, wait_bar(ctx, s, parity));
            if (!ok) break;
            const uint8_t* kst = smem + s * STAGE;
            const uint8_t* vst = kst + QK_BYTES;
            const uint8_t* sst = vst + QV_BYTES;
            const int tok0 = p * P + 16 * slice;
            if (tok0 < len) {
                {   // 1/scale of this warp's tokens: lane -> token lane/2, groups 2*(lane&1) and the next; 0 past the end
                    const int tl = lane >> 1, g2 = (lane & 1) * 2;
                    const uint32_t hh = *reinterpret_cast<const uint32_t*>(sst + ((16 * slice + tl) * 4 + g2) * 2);
                    const bool live_t = tok0 + tl < len;
                    // token 4 q + 2 e + nt goes to [q][group][2 nt + e]
                    float* dst = inv_w + (tl >> 2) * 16 + g2 * 4 + (tl & 1) * 2 + ((tl >> 1) & 1);
                    dst[0] = live_t ? inv_scale_bits(hh & 0xFFFFu) : 0.f;
                    dst[4] = live_t ? inv_scale_bits(hh >> 16) : 0.f;
                }
                __syncwarp();
                float2 inv[2][4];           // [nt][group], of the lane's two tokens of tile nt
#pragma unroll
                for (int grp = 0; grp < 4; ++grp) {
                    const float4 v = *reinterpret_cast<const float4*>(inv_w + t4 * 16 + grp * 4);
                    inv[0][grp] = make_float2(v.x, v.y);
                    inv[1][grp] = make_float2(v.z, v.w);
                }
                // The two token pairs of this lane, 16 value bytes (all four groups) each (its tokens 4 t4 .. 4 t4 + 3 of the slice:
                // pairs 2 t4 and 2 t4 + 1; the 16-byte pieces of a pair are stored XOR-swizzled by the pair index, which keeps the
                // eight lanes of a quarter-warp on different banks), read ahead of the scores (131072 tokens x 8 heads 59.5 -> 58.9 us)
                const int pr = 8 * slice + 2 * t4;
                const uint4 va = *reinterpret_cast<const uint4*>(vst + pr * 128 + ((g ^ (pr & 7)) << 4));
                const uint4 vb = *reinterpret_cast<const uint4*>(vst + (pr + 1) * 128 + ((g ^ ((pr + 1) & 7)) << 4));
                // ---- S = q K^T for 16 tokens, one accumulator per scale group, combined with 1/scale
                float2 sc[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
                for (int nt = 0; nt < 2; ++nt) {
                    const int row = 16 * slice + 2 * g + nt;     // column n of tile nt is token 2 n + nt of the slice
#pragma unroll
                    for (int grp = 0; grp < 4; ++grp) {
                        const int chunk = (2 * grp + (t4 >> 1)) ^ (row & 7);
                        const uint2 kb = *reinterpret_cast<const uint2*>(kst + row * 128 + chunk * 16 + (t4 & 1) * 8);
                        float c0[4], c1[4];
                        mma_f16_zero(c0, qf[grp], e4m3_pair02_f16x2(kb.x), e4m3_pair13_f16x2(kb.x));
                        mma_f16_zero(c1, qf[grp], e4m3_pair02_f16x2(kb.y), e4m3_pair13_f16x2(kb.y));
                        sc[nt] = __ffma2_rn(make_float2(c0[0], c0[1]), inv[nt][grp], sc[nt]);
                        sc[nt] = __ffma2_rn(make_float2(c1[2], c1[3]), inv[nt][grp], sc[nt]);
                    }
                }
                float sacc[2][2] = {{sc[0].x, sc[0].y}, {sc[1].x, sc[1].y}};
                // ---- online softmax for head row g.  Only the last tile of a sequence has tokens past its end: they
                // get the "empty" score there, so the common path carries no per-token predicate
                if (tok0 + 16 > len) {
#pragma unroll
                    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                        for (int e = 0; e < 2; ++e)
                            if (tok0 + 4 * t4 + 2 * e + nt >= len) sacc[nt][e] = kEmpty;
                }
                if (a.scores_out && g < a.group) {
                    float* srow = a.scores_out + ((size_t)b * a.Hq + qh0 + g) * a.scores_ld + tok0 + 4 * t4;
#pragma unroll
                    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                        for (int e = 0; e < 2; ++e)
                            if (tok0 + 4 * t4 + 2 * e + nt < len) srow[2 * e + nt] = sacc[nt][e] * 0.6931471805599453f;
                }
                float mx = fmaxf(fmaxf(sacc[0][0], sacc[0][1]), fmaxf(sacc[1][0], sacc[1][1]));
                if (__any_sync(0xffffffffu, mx > m_run)) {      // a new maximum: seldom, after the first few tiles
                    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
                    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
                    const float m_new = fmaxf(m_run, mx);
                    const float corr = ex2(m_run - m_new);
                    l_run *= corr;
                    m_run = m_new;
                    // the accumulator columns of this lane are heads 2 t4 and 2 t4 + 1: their factors live in other lanes
                    const float ca = __shfl_sync(0xffffffffu, corr, 8 * t4), cb = __shfl_sync(0xffffffffu, corr, 8 * t4 + 4);
#pragma unroll
                    for (int n = 0; n < 8; ++n) { o[n][0] *= ca; o[n][2] *= ca; o[n][1] *= cb; o[n][3] *= cb; }
                }
                float2 pv[2];
#pragma unroll
                for (int nt = 0; nt < 2; ++nt) pv[nt] = make_float2(ex2(sacc[nt][0] - m_run), ex2(sacc[nt][1] - m_run));    // 0 for an "empty" score
                l_run += (pv[0].x + pv[0].y) + (pv[1].x + pv[1].y);
                // ---- O^T += V^T (P / scale)^T: rows are head_dim elements, columns heads, so all sixteen rows of the
                // product work and P is used as it comes out of S (pairs of tokens per head)
                const uint32_t xa[4] = {va.x, va.y, va.z, va.w}, xb[4] = {vb.x, vb.y, vb.z, vb.w};
#pragma unroll
                for (int grp = 0; grp < 4; ++grp) {
                    // B of the value product: k pairs are (even, odd) tokens of a pair = (tile 0, tile 1) of a column
                    const float2 w0 = __fmul2_rn(pv[0], inv[0][grp]), w1 = __fmul2_rn(pv[1], inv[1][grp]);
                    const uint32_t pa0 = pack_f16(w0.x, w1.x), pa2 = pack_f16(w0.y, w1.y);
                    const uint32_t x = xa[grp], y = xb[grp], xs = x >> 8, ys = y >> 8;
                    // nibble n of the even | odd token of a pair as f16x2: 1024 + n (low nibble) or 64 + n (high
                    // nibble) by one logic operation, then n - 8 exactly by one subtraction
                    // rows g | g + 8 of tile (grp, j) are elements 32 grp + 4 g + 2 j | + 1
                    mma_f16_full(o[2 * grp], nib_lo(x), nib_hi(x), nib_lo(y), nib_hi(y), pa0, pa2);
                    mma_f16_full(o[2 * grp + 1], nib_lo(xs), nib_hi(xs), nib_lo(ys), nib_hi(ys), pa0, pa2);
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(empty(s));
        }
        l_run += __shfl_xor_sync(0xffffffffu, l_run, 1);
        l_run += __shfl_xor_sync(0xffffffffu, l_run, 2);
    } else {
        // ------------------------------------------------------------------ compute: tokens [16*warp, 16*warp+16) of every page
        const int qh0 = kvh * a.group;
        // A fragments of q (rows = heads of the group, zero beyond), pre-scaled into the exp2 domain, hi + lo bf16
        uint32_t qhi[D / 16][2], qlo[D / 16][2];
        {
            const float sc = a.scale * kLog2e;
            const float* qrow = a.q + ((size_t)b * a.Hq + qh0 + g) * D;
            const bool live = g < a.group;
#pragma unroll
            for (int ks = 0; ks < D / 16; ++ks) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int d = 16 * ks + 8 * h + 2 * t4;
                    float x0 = 0.f, x1 = 0.f;
                    if (live) { const float2 v = *reinterpret_cast<const float2*>(qrow + d); x0 = v.x * sc; x1 = v.y * sc; }
                    const float h0 = __bfloat162float(__float2bfloat16_rn(x0)), h1 = __bfloat162float(__float2bfloat16_rn(x1));
                    qhi[ks][h] = pack_bf16(h0, h1);
                    qlo[ks][h] = pack_bf16(x0 - h0, x1 - h1);
                }
            }
        }
        bool ok = true;
        for (int p = p_begin; p < p_end && ok; ++p) {
            const int i = p - p_begin, s = i % NST, it = i / NST;
            ok = __all_sync(0xffffffffu, wait_bar(ctx, s, it & 1));
            if (!ok) break;
            const uint32_t kbase = base + (uint32_t)s * STAGE, vbase = kbase + SLAB;
            const int tok0 = p * P + 16 * warp;                 // first token of this warp's slice
            if (tok0 < len) {
                if (tok0 + 16 > len) {
                    // rows past the end of the sequence hold whatever the page held: zero them in V
                    // (their probabilities are zero, but 0 * NaN is not)
                    for (int c = lane; c < 16 * (D / 8); c += 32) {
                        const int r = 16 * warp + c / (D / 8), ch = c % (D / 8);
                        if (p * P + r >= len)
                            *reinterpret_cast<uint4*>(smem + s * STAGE + SLAB + slab_off(r, ch * 8)) = make_uint4(0, 0, 0, 0);
                    }
                    __syncwarp();
                }
                // ---- S = q K^T for 16 tokens: two 8-token n-tiles
                float sacc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
                const int mat = lane >> 3;
                {
                    const int row = 16 * warp + (lane & 7) + ((mat >> 1) << 3);
#pragma unroll
                    for (int ks = 0; ks < D / 16; ++ks) {
                        uint32_t kb[4];
                        ldmatrix_x4(kbase + slab_off(row, 16 * ks + ((mat & 1) << 3)), kb);
                        mma_16816(sacc[0], qhi[ks][0], qhi[ks][1], kb[0], kb[1]);
                        mma_16816(sacc[1], qhi[ks][0], qhi[ks][1], kb[2], kb[3]);
                        mma_16816(sacc[0], qlo[ks][0], qlo[ks][1], kb[0], kb[1]);
                        mma_16816(sacc[1], qlo[ks][0], qlo[ks][1], kb[2], kb[3]);
                    }
                }
                // ---- online softmax for head row g (lanes with the same g share the row)
                float mx = kEmpty;
                bool valid[2][2];
#pragma unroll
                for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        valid[nt][e] = tok0 + nt * 8 + 2 * t4 + e < len;
                        if (valid[nt][e]) mx = fmaxf(mx, sacc[nt][e]);
                    }
                if (a.scores_out && g < a.group) {      // what H2O eviction accumulates; off on the plain path
                    float* srow = a.scores_out + ((size_t)b * a.Hq + qh0 + g) * a.scores_ld + tok0 + 2 * t4;
#pragma unroll
                    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                        for (int e = 0; e < 2; ++e)
                            if (valid[nt][e]) srow[nt * 8 + e] = sacc[nt][e] * 0.6931471805599453f;
                }
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
                const float m_new = fmaxf(m_run, mx);
                const float corr = ex2(m_run - m_new);
                float pv[2][2], ps = 0.f;
#pragma unroll
                for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        pv[nt][e] = valid[nt][e] ? ex2(sacc[nt][e] - m_new) : 0.f;
                        ps += pv[nt][e];
                    }
                l_run = l_run * corr + ps;
                m_run = m_new;
                if (__any_sync(0xffffffffu, corr != 1.f)) {
#pragma unroll
                    for (int n = 0; n < D / 8; ++n) { o[n][0] *= corr; o[n][1] *= corr; }
                }
                const uint32_t pa0 = pack_bf16(pv[0][0], pv[0][1]), pa2 = pack_bf16(pv[1][0], pv[1][1]);
                // ---- O += P V: 16 tokens x head_dim, two 8-wide d n-tiles per ldmatrix
                {
                    const int row = 16 * warp + (lane & 7) + ((mat & 1) << 3);
#pragma unroll
                    for (int dn = 0; dn < D / 16; ++dn) {
                        uint32_t vb[4];
                        ldmatrix_x4_trans(vbase + slab_off(row, 16 * dn + ((mat >> 1) << 3)), vb);
                        mma_16816(o[2 * dn], pa0, pa2, vb[0], vb[1]);
                        mma_16816(o[2 * dn + 1], pa0, pa2, vb[2], vb[3]);
                    }
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(empty(s));
        }
        l_run += __shfl_xor_sync(0xffffffffu, l_run, 1);
        l_run += __shfl_xor_sync(0xffffffffu, l_run, 2);
    }

    __syncthreads();
    if (*ctx.abort) {
        // A wait ran out: what has been issued must land before the shared memory is used again and released.  A producer that stops cannot
        // tell which of its stages another group has left unread, nor whether a slot is someone else's by now, so each slot waits for
        // the last stage that any of them issued there; for local copies, whatever budget the caller has set for the waits.
        if (tid < NST) {
            const int i = last_in_slot<NST, PROD>(reinterpret_cast<const int*>(smem + SMEM_BAR + 256), 32, tid);
            const long long t0 = clock64();
            while (i >= 0 && !mbar_try_wait(full(tid), (i / NST) & 1) && clock64() - t0 < kDefaultWaitLimitCycles) {}
        }
        __syncthreads();
    }
    // ---- merge the warps' partials (the ring is idle now: reuse it)
    // The next kernel may launch under the merges.  Not before: its CTAs would take slots beside this kernel's and end up
    // unevenly placed (two on some SMs, none on others: 196 us instead of 107 for a 131072-token quantised step).  Where the
    // CTAs have an SM each the next one's could only wait for this one's shared memory, so it is left to start at the end
    // (131072 tokens x 2 heads, decode after decode: 84.8 us with an early start, 81.5 without).
    if (!a.alone) pdl_trigger();
    float* sm_o = reinterpret_cast<float*>(smem);                 // [warps][8 heads][128]
    float* sm_m = sm_o + COMPUTE * 8 * D;                         // [warps][8]
    float* sm_l = sm_m + COMPUTE * 8;
    if (warp < COMPUTE) {
        if constexpr (QUANT) {
            // tile (grp, j): columns are heads 2 t4 | 2 t4 + 1, rows elements 32 grp + 4 g + 2 j | + 1
#pragma unroll
            for (int n = 0; n < 8; ++n) {
                const int d0 = 32 * (n >> 1) + 4 * g + 2 * (n & 1);
                *reinterpret_cast<float2*>(&sm_o[(warp * 8 + 2 * t4) * D + d0]) = make_float2(o[n][0], o[n][2]);
                *reinterpret_cast<float2*>(&sm_o[(warp * 8 + 2 * t4 + 1) * D + d0]) = make_float2(o[n][1], o[n][3]);
            }
        } else {
#pragma unroll
            for (int n = 0; n < D / 8; ++n)
                *reinterpret_cast<float2*>(&sm_o[(warp * 8 + g) * D + n * 8 + 2 * t4]) = make_float2(o[n][0], o[n][1]);
        }
        if (t4 == 0) { sm_m[warp * 8 + g] = m_run; sm_l[warp * 8 + g] = l_run; }
    }
    __syncthreads();
    const int rows = a.B * a.Hq;
    const int used = COMPUTE == 4 ? 4 : min(COMPUTE, 4 * (p_end - p_begin));         // warps that had a slice
    float* cl_o = sm_l + COMPUTE * 8;                                      // cluster form: this split's rows [8][D], then m [8], l [8]
    float* cl_ml = cl_o + 8 * D;
    for (int idx = tid; idx < a.group * D; idx += kThreads) {
        const int h = idx / D, d = idx % D;
        float mt = kEmpty;
#pragma unroll
        for (int w = 0; w < COMPUTE; ++w)
            if (w < used) mt = fmaxf(mt, sm_m[w * 8 + h]);
        float ov = 0.f, lt = 0.f;
#pragma unroll
        for (int w = 0; w < COMPUTE; ++w)
            if (w < used) {
                const float wgt = ex2(sm_m[w * 8 + h] - mt);
                ov = fmaf(wgt, sm_o[(w * 8 + h) * D + d], ov);
                lt = fmaf(wgt, sm_l[w * 8 + h], lt);
            }
        const int row = b * a.Hq + kvh * a.group + h;
        if (a.direct) {
            a.out[(size_t)row * D + d] = lt > 0.f ? ov / lt : 0.f;
        } else if (a.cluster > 1) {
            cl_o[h * D + d] = ov;
            if (d == 0) { cl_ml[h] = mt; cl_ml[8 + h] = lt; }
        } else {
            float* part = a.part + (size_t)split * rows * (D + 2);
            part[(size_t)row * D + d] = ov;
            if (d == 0) {
                part[(size_t)rows * D + row] = mt * 0.6931471805599453f;   // back to the natural-log domain
                part[(size_t)rows * D + rows + row] = lt;
            }
        }
    }
    if (a.direct || !a.fuse) return;
    // parts of the merge through global memory below: clusters where there are any, else splits
    const int n_parts = a.cluster > 1 ? a.n_splits / a.cluster : a.n_splits;
    if (a.cluster > 1) {
        // ---- consecutive splits of a head are the CTAs of one cluster: every CTA combines its share of the columns, reading all
        // of the cluster's rows, maxima and sums at once through distributed shared memory.  With one cluster per head nothing
        // leaves the SMs but the result and nobody counts arrivals; with several, a cluster is one part of the merge below.
        cluster_sync();
        const int rank = split % a.cluster;
        for (int q = tid * a.cluster + rank; q < a.group * (D / 4); q += kThreads * a.cluster) {
            const int h = q / (D / 4);
            const uint32_t o_addr = smem_u32(cl_o + 4 * q), ml_addr = smem_u32(cl_ml + h);
            float4 v[kMaxCluster];
            float m[kMaxCluster], l[kMaxCluster];
#pragma unroll
            for (int p = 0; p < kMaxCluster; ++p)
                if (p < a.cluster) {
                    v[p] = ld_cluster_f32x4(cluster_map(o_addr, p));
                    m[p] = ld_cluster_f32(cluster_map(ml_addr, p));
                    l[p] = ld_cluster_f32(cluster_map(ml_addr + 32, p));
                }
            float mt = kEmpty;
#pragma unroll
            for (int p = 0; p < kMaxCluster; ++p)
                if (p < a.cluster) mt = fmaxf(mt, m[p]);
            float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
            float lt = 0.f;
#pragma unroll
            for (int p = 0; p < kMaxCluster; ++p)
                if (p < a.cluster) {
                    const float w = ex2(m[p] - mt);
                    acc.x = fmaf(w, v[p].x, acc.x); acc.y = fmaf(w, v[p].y, acc.y);
                    acc.z = fmaf(w, v[p].z, acc.z); acc.w = fmaf(w, v[p].w, acc.w);
                    lt = fmaf(w, l[p], lt);
                }
            const int row = b * a.Hq + kvh * a.group + h;
            // where un-normalised rows go: the part of this cluster, or the caller's partial
            float* part = n_parts > 1 ? a.part + (size_t)(split / a.cluster) * rows * (D + 2) : a.partial_out;
            float* dst = (part ? part : a.out) + (size_t)row * D + 4 * (q % (D / 4));
            if (part) {
                if (q % (D / 4) == 0) {
                    part[(size_t)rows * D + row] = mt * 0.6931471805599453f;
                    part[(size_t)rows * D + rows + row] = lt;
                }
            } else {
                const float inv = lt > 0.f ? 1.f / lt : 0.f;
                acc = make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv);
            }
            dst[0] = acc.x; dst[1] = acc.y; dst[2] = acc.z; dst[3] = acc.w;
        }
        if (n_parts > 1) __threadfence();
        cluster_sync();         // a CTA leaves only when nobody reads its rows any more
        if (n_parts == 1 || rank != 0) return;
    }

    // ---- fused merge: whoever arrives last for this (sequence, kv head) combines its parts
    __threadfence();
    __syncthreads();
    int* s_flag = reinterpret_cast<int*>(smem + SMEM_BAR + 2 * NST * 8 + 8);
    const int slot = b * a.Hkv + kvh;
    if (tid == 0) {
        const int t = atomicAdd(&a.counters[slot], 1);
        const int last = (t == n_parts - 1);
        if (last) a.counters[slot] = 0;          // nobody else touches the slot before the next launch
        *s_flag = last;
    }
    __syncthreads();
    if (!*s_flag) return;
    __threadfence();
    float* sm_w = reinterpret_cast<float*>(smem);              // [8 heads][256 splits]: m, then the weights
    float* sm_ls = sm_w + 8 * kMaxFusedSplits;                 // [8][256]: l of every split
    float* sm_mt = sm_ls + 8 * kMaxFusedSplits;                // [8] max (natural log), [8] l
    float* sm_res = sm_mt + 16;                                // [8][128] merged un-normalised rows
    const size_t pstride = (size_t)rows * (D + 2);
    const int row0 = b * a.Hq + kvh * a.group;
    for (int idx = tid; idx < a.group * n_parts; idx += kThreads) {
        const int h = idx / n_parts, s = idx % n_parts;
        const float* ml = a.part + (size_t)s * pstride + (size_t)rows * D + row0 + h;
        sm_w[h * kMaxFusedSplits + s] = __ldcg(ml);
        sm_ls[h * kMaxFusedSplits + s] = __ldcg(ml + rows);
    }
    __syncthreads();
    for (int h = warp; h < a.group; h += kThreads / 32) {
        float mt = kEmpty;
        for (int s = lane; s < n_parts; s += 32) mt = fmaxf(mt, sm_w[h * kMaxFusedSplits + s]);
#pragma unroll
        for (int sh = 16; sh > 0; sh >>= 1) mt = fmaxf(mt, __shfl_xor_sync(0xffffffffu, mt, sh));
        float lt = 0.f;
        for (int s = lane; s < n_parts; s += 32) {
            const float w = __expf(sm_w[h * kMaxFusedSplits + s] - mt);
            sm_w[h * kMaxFusedSplits + s] = w;
            lt = fmaf(w, sm_ls[h * kMaxFusedSplits + s], lt);
        }
#pragma unroll
        for (int sh = 16; sh > 0; sh >>= 1) lt += __shfl_xor_sync(0xffffffffu, lt, sh);
        if (lane == 0) { sm_mt[h] = mt; sm_mt[8 + h] = lt; }
    }
    __syncthreads();
    const PeerExchange& x = a.x;
    const bool exchange = x.world > 1;
    // Merged un-normalised rows into shared memory.  A thread owns two columns of one head and has the loads of
    // up to 16 splits in flight: the partials sit in L2, so the chain is latency, not bandwidth.
    for (int c = tid; c < a.group * (D / 2); c += kThreads) {
        const int h = c / (D / 2), d2 = c % (D / 2);
        const float* col = a.part + (size_t)(row0 + h) * D + 2 * d2;     // 8-byte aligned: D and pstride are even
        float2 acc = make_float2(0.f, 0.f);
        for (int s0 = 0; s0 < n_parts; s0 += 16) {
            float2 v[16];
#pragma unroll
            for (int j = 0; j < 16; ++j)
                if (s0 + j < n_parts) v[j] = __ldcg(reinterpret_cast<const float2*>(col + (size_t)(s0 + j) * pstride));
#pragma unroll
            for (int j = 0; j < 16; ++j)
                if (s0 + j < n_parts) {
                    const float w = sm_w[h * kMaxFusedSplits + s0 + j];
                    acc.x = fmaf(w, v[j].x, acc.x);
                    acc.y = fmaf(w, v[j].y, acc.y);
                }
        }
        *reinterpret_cast<float2*>(&sm_res[h * D + 2 * d2]) = acc;
    }
    __syncthreads();
    if (!exchange) {
        for (int idx = tid; idx < a.group * D; idx += kThreads) {
            const int h = idx / D;
            const float lt = sm_mt[8 + h];
            if (a.partial_out) a.partial_out[(size_t)row0 * D + idx] = sm_res[idx];
            else a.out[(size_t)row0 * D + idx] = lt > 0.f ? sm_res[idx] / lt : 0.f;
        }
        if (a.partial_out && tid < a.group) {
            a.partial_out[(size_t)rows * D + row0 + tid] = sm_mt[tid];
            a.partial_out[(size_t)rows * D + rows + row0 + tid] = sm_mt[8 + tid];
        }
        return;
    }

    // ---- cross-GPU exchange of this head's rows.  An item is one float of the head's part: group*D values of
    // O, then group maxima, then group sums; every 8-byte inbox element carries the step number next to the
    // value, so a reader that sees the number sees the value: neither a fence nor a flag between the peers.
    const unsigned int e = *x.seq + 1;
    const int par = e & 1;
    const int n_items = a.group * (D + 2);
    auto item_off = [&](int i) -> size_t {       // offset of item i inside a part laid out [O | m | l]
        if (i < a.group * D) return (size_t)row0 * D + i;
        i -= a.group * D;
        return i < a.group ? (size_t)rows * D + row0 + i : (size_t)rows * D + rows + row0 + (i - a.group);
    };
    auto item_val = [&](int i) -> float {
        if (i < a.group * D) return sm_res[i];
        i -= a.group * D;
        return i < a.group ? sm_mt[i] : sm_mt[8 + (i - a.group)];
    };
    const int total = (x.world - 1) * n_items;
    for (int it = tid; it < total; it += kThreads) {
        const int pi = it / n_items, i = it - pi * n_items, r = pi + (pi >= x.rank);
        reinterpret_cast<uint2*>(x.peer_inbox[r])[((size_t)par * x.world + x.rank) * pstride + item_off(i)] =
            make_uint2(__float_as_uint(item_val(i)), e);
    }
    // Poll the peers' items of this head, all peers side by side: a thread issues the loads of up to 16 missing
    // items before it examines any, so a round is one trip to L2 whatever the number of peers.
    float* sm_in = sm_res + 8 * D;                 // [world-1][n_items]
    constexpr int kChunk = 16;
    bool ok = true;
    const long long t0 = clock64();
    for (int base_it = 0; base_it < total && ok; base_it += kChunk * kThreads) {
        unsigned int pending = 0;
        unsigned int off[kChunk];                  // element offset inside the local inbox
#pragma unroll
        for (int j = 0; j < kChunk; ++j) {
            const int it = base_it + j * kThreads + tid;
            off[j] = 0;
            if (it < total) {
                const int pi = it / n_items, i = it - pi * n_items, r = pi + (pi >= x.rank);
                off[j] = (unsigned int)(((size_t)par * x.world + r) * pstride + item_off(i));
                pending |= 1u << j;
            }
        }
        const uint2* inbox = reinterpret_cast<const uint2*>(x.inbox);
        while (pending) {
            uint2 v[kChunk];
#pragma unroll
            for (int j = 0; j < kChunk; ++j)
                if (pending >> j & 1u) v[j] = ld_pair_volatile(inbox + off[j]);
#pragma unroll
            for (int j = 0; j < kChunk; ++j)
                if ((pending >> j & 1u) && v[j].y == e) {
                    sm_in[base_it + j * kThreads + tid] = __uint_as_float(v[j].x);
                    pending &= ~(1u << j);
                }
            if (pending && clock64() - t0 > x.wait_cycles) {
                ok = false;
                if (a.status && atomicCAS(a.status, 0, GRL_ERR_TIMEOUT) == 0) {
                    const int it = base_it + (__ffs(pending) - 1) * kThreads + tid, pi = it / n_items;
                    a.status[1] = (3 << 28) | (pi + (pi >= x.rank));     // a peer that did not post
                    a.status[2] = (int)e;
                    a.status[3] = x.rank;
                }
                break;
            }
        }
    }
    ok = __syncthreads_and(ok);                    // the whole CTA agrees: no row is written after a timeout
    if (ok) {
        for (int idx = tid; idx < a.group * D; idx += kThreads) {
            const int h = idx / D;
            float mt = sm_mt[h];
            for (int pi = 0; pi < x.world - 1; ++pi) mt = fmaxf(mt, sm_in[pi * n_items + a.group * D + h]);
            const float w0 = __expf(sm_mt[h] - mt);
            float ov = w0 * sm_res[idx], lt = w0 * sm_mt[8 + h];
            for (int pi = 0; pi < x.world - 1; ++pi) {
                const float* in = sm_in + pi * n_items;
                const float w = __expf(in[a.group * D + h] - mt);
                ov = fmaf(w, in[idx], ov);
                lt = fmaf(w, in[a.group * D + a.group + h], lt);
            }
            a.out[(size_t)row0 * D + idx] = lt > 0.f ? ov / lt : 0.f;
        }
    }
    // the head that finishes last advances the step counter for the next launch (every head has read it by
    // then); after a timeout the counter stays, grl_sync reports the failure and grl_exchange_reset on every
    // rank puts the ranks back in step
    if (tid == 0 && ok) {
        const int heads = a.B * a.Hkv;
        if (atomicAdd(&a.counters[kDoneSlot], 1) == heads - 1) {
            a.counters[kDoneSlot] = 0;
            *x.seq = e;
        }
    }
}

// The K (or V) pool as a 2-D bf16 tensor (rows = pages * Hkv * page tokens, head_dim columns); box = 64 columns x
// one page of one kv head.
static int make_pool_map(grl_device* dev, CUtensorMap* tm, const void* pool, uint64_t rows, int head_dim, int page_tokens) {
    TmapKey k{};
    k.ptr = pool; k.rank = 2; k.swizzle_128b = 1;
    k.dims[0] = (uint64_t)head_dim; k.dims[1] = rows;
    k.strides[0] = (uint64_t)head_dim * 2;
    k.box[0] = 64; k.box[1] = (uint32_t)page_tokens;
    return get_tensor_map(dev, k, tm);
}

}  // namespace dmma

bool decode_mma_supported(const grl_decode_params* p) {
    const grl_kv_layout& kv = p->kv;
    const int group = p->num_q_heads / kv.num_kv_heads;
    const bool geometry = (kv.page_tokens == 64 || kv.page_tokens == 32 || kv.page_tokens == 16) && group >= 1 && group <= 8 &&
                          ((uintptr_t)kv.k_pages % 16 == 0) && ((uintptr_t)kv.v_pages % 16 == 0);
    if (kv.cache_dtype == GRL_FP8_INT4)
        return geometry && kv.head_dim == 128 && kv.scales && ((uintptr_t)kv.scales % 16 == 0) && ((uintptr_t)p->q % 16 == 0);
    return kv.cache_dtype == GRL_BF16 && geometry && (kv.head_dim == 128 || kv.head_dim == 64) && ((uintptr_t)p->q % 8 == 0);
}

template <int FORM, int HD>
static int set_attributes(grl_device* dev) {
    using namespace dmma;
    constexpr int kAlone = FORM == QUANT_WIDE ? Smem<FORM, HD>::TOTAL : kAloneSmem;
    static bool attr_set[64] = {};
    if (!attr_set[dev->ordinal & 63]) {      // a function attribute belongs to the device that was current
        GRL_CUDA(cudaFuncSetAttribute(decode_mma_kernel<FORM, HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, kAlone));
        GRL_CUDA(cudaFuncSetAttribute(decode_mma_kernel<FORM, HD>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        attr_set[dev->ordinal & 63] = true;
    }
    return GRL_OK;
}

template <int FORM, int HD>
static int instance_clusters(grl_device* dev, int size) {
    using namespace dmma;
    return set_attributes<FORM, HD>(dev) != GRL_OK ? 0
        : max_active_clusters(dev, (const void*)decode_mma_kernel<FORM, HD>, Warps<FORM>::THREADS, Smem<FORM, HD>::TOTAL, size);
}

// Clusters of `size` CTAs of the kernel that serves this call that the device holds at once.
int decode_mma_clusters(grl_device* dev, const grl_decode_params* p, bool wide, int size) {
    using namespace dmma;
    DeviceGuard g(dev->ordinal);
    if (p->kv.cache_dtype == GRL_FP8_INT4) return wide ? instance_clusters<QUANT_WIDE, 128>(dev, size) : instance_clusters<QUANT_PAIR, 128>(dev, size);
    return p->kv.head_dim == 64 ? instance_clusters<BF16, 64>(dev, size) : instance_clusters<BF16, 128>(dev, size);
}

template <int FORM, int HD>
static int launch_instance(grl_device* dev, const CUtensorMap& tk, const CUtensorMap& tv, const dmma::Args& a, dim3 grid) {
    using namespace dmma;
    constexpr int kAlone = FORM == QUANT_WIDE ? Smem<FORM, HD>::TOTAL : kAloneSmem;
    const int rc = set_attributes<FORM, HD>(dev);
    if (rc) return rc;
    if (a.alone)
        GRL_CUDA(launch_pdl(decode_mma_kernel<FORM, HD>, grid, Warps<FORM>::THREADS, kAlone, dev->stream, tk, tv, a));
    else
        GRL_CUDA(launch_pdl_cluster(decode_mma_kernel<FORM, HD>, grid, Warps<FORM>::THREADS, Smem<FORM, HD>::TOTAL, dev->stream,
                                    a.cluster, tk, tv, a));
    GRL_LAUNCHED(FORM == BF16 ? "decode_mma_kernel" : "decode_mma_kernel<quantised>");
    return GRL_OK;
}

int decode_mma_launch(grl_device* dev, const grl_decode_params* p, const DecodePlan& plan, float scale) {
    using namespace dmma;
    const int n_splits = plan.n_splits;
    const grl_kv_layout& kv = p->kv;
    const uint64_t pages = kv.num_pages > 0 ? (uint64_t)kv.num_pages : (uint64_t)kv.batch * kv.max_pages;
    const uint64_t rows = pages * kv.num_kv_heads * kv.page_tokens;
    const bool quant = kv.cache_dtype == GRL_FP8_INT4;
    CUtensorMap tk, tv;
    int rc;
    if (quant) {
        // the key pool as a 2-D byte tensor (rows, 128); box = one page of one kv head; values and scales are
        // contiguous per (page, kv head) and travel as plain bulk copies
        TmapKey k{};
        k.ptr = kv.k_pages; k.rank = 2; k.swizzle_128b = 1; k.bytes = 1;
        k.dims[0] = D; k.dims[1] = rows;
        k.strides[0] = (uint64_t)D;
        k.box[0] = D; k.box[1] = (uint32_t)kv.page_tokens;
        rc = get_tensor_map(dev, k, &tk);
        tv = tk;
    } else {
        rc = make_pool_map(dev, &tk, kv.k_pages, rows, kv.head_dim, kv.page_tokens);
        if (!rc) rc = make_pool_map(dev, &tv, kv.v_pages, rows, kv.head_dim, kv.page_tokens);
    }
    if (rc) return rc;
    Args a{};
    a.v_q = static_cast<const uint8_t*>(kv.v_pages); a.scales = static_cast<const uint16_t*>(kv.scales);
    a.block_table = kv.block_table; a.seq_lens = kv.seq_lens; a.q = p->q;
    a.part = (float*)p->workspace; a.out = p->out; a.status = dev->d_status;
    a.B = kv.batch; a.Hq = p->num_q_heads; a.Hkv = kv.num_kv_heads; a.max_pages = kv.max_pages;
    a.page = kv.page_tokens; a.ppt = P / kv.page_tokens;
    a.n_splits = n_splits; a.group = p->num_q_heads / kv.num_kv_heads;
    a.scale = scale; a.direct = plan.direct ? 1 : 0; a.cluster = plan.cluster; a.alone = plan.alone ? 1 : 0;
    a.fuse = plan.fused ? 1 : 0; a.counters = dev->d_counters; a.partial_out = p->partial_out;
    a.scores_out = p->scores_out; a.scores_ld = p->scores_ld;
    a.x.world = 1;
    a.wait_limit = dev->wait_limit_cycles;
    const int bound = p->max_seq_len > 0 ? p->max_seq_len : kv.max_pages * kv.page_tokens;
    const int stages = (bound + P - 1) / P;
    a.pps_hint = (stages + n_splits - 1) / n_splits;
    if (p->exchange) {
        GRL_REQUIRE(plan.fused, "the fused cross-GPU merge needs the split-KV path");
        rc = fill_peer_exchange(dev, p->exchange, &a.x);
        if (rc) return rc;
        const int heads = kv.batch * kv.num_kv_heads;
        GRL_REQUIRE(heads <= dev->prop.multiProcessorCount,
                    "fused cross-GPU merge: B*Hkv = %d exceeds the %d SMs (waiting CTAs must leave room for the rest)",
                    heads, dev->prop.multiProcessorCount);
        GRL_REQUIRE(p->exchange->low_latency, "the exchange inside the decode kernel uses the low-latency inbox "
                                              "format ({value, step} pairs): set low_latency");
        GRL_REQUIRE(p->out, "out is NULL");
    }
    dev->status_dirty = true;
    dim3 grid(n_splits, kv.num_kv_heads, kv.batch);
    if (quant) return plan.wide ? launch_instance<QUANT_WIDE, 128>(dev, tk, tv, a, grid) : launch_instance<QUANT_PAIR, 128>(dev, tk, tv, a, grid);
    return kv.head_dim == 64 ? launch_instance<BF16, 64>(dev, tk, tv, a, grid) : launch_instance<BF16, 128>(dev, tk, tv, a, grid);
}

}  // namespace grl
