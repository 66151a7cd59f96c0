// Paged head-major KV cache kernels: fused RoPE + cast + scatter append, and gather back to
// token-major float32.  Replaces ops::kvCacheAppend / ops::kvCacheDecode
// (cpp/src/ops/kv_cache.cpp:155-419, 435-578) for the uncompressed mode, in which the reference
// stores only metadata.
#include "common.cuh"

namespace grl {

struct AppendArgs {
    void* k_pages;
    void* v_pages;
    const int32_t* block_table;
    int32_t* seq_lens;
    const float* k_new;
    const float* v_new;
    const float* q_in;
    float* q_out;
    int B, Hkv, Hq, D, P, max_pages, n_new;
    int rope_mode, pos_base, update_lens;
    const int32_t* pos_offsets;
    int32_t* status;     // device status word: GRL_ERR_INVALID when a sequence has no room for the new tokens
    uint16_t* scales;    // quantised cache only
    int skip_kv;         // rotate the queries only (the quantised append stores K and V with its own kernel)
    int heads_per_item;  // quantised append: kv heads that one warp walks for the same token and group
    RopeFreq freq;
};

// grid (chunks, B).  A work item is (token i, head slot, pair j), head slots being the Hkv key/value
// heads followed by the Hq query heads, so that a one-token decode step spreads its (Hkv+Hq)*D/2
// pairs over the whole CTA instead of walking the heads serially behind dependent loads.  With
// update_lens the grid has ONE chunk per sequence, so that the length read at entry cannot race
// with the write at exit.
template <typename T>
__global__ void __launch_bounds__(1024) kv_append_kernel(AppendArgs a) {
    const int b = blockIdx.y;
    const int half = a.D / 2;
    const int len0 = a.seq_lens[b];
    // A sequence without room for the new tokens is left untouched (no store, no length update): the block
    // table has no page for them.  The op layer checks this on the host; a direct caller of the C ABI gets
    // GRL_ERR_KERNEL from the next grl_sync.
    if (len0 < 0 || len0 + a.n_new > a.max_pages * a.P) {
        if (threadIdx.x == 0 && blockIdx.x == 0 && a.status && atomicCAS(a.status, 0, GRL_ERR_INVALID) == 0) {
            a.status[1] = 4 << 28;
            a.status[2] = b;
            a.status[3] = len0;
        }
        return;
    }
    const int pos_off = a.pos_offsets ? a.pos_offsets[b] : 0;
    T* kp = reinterpret_cast<T*>(a.k_pages);
    T* vp = reinterpret_cast<T*>(a.v_pages);
    const int slots = a.Hkv + (a.q_in ? a.Hq : 0);
    const int items = a.n_new * slots * half;
    // The angle depends on (position, pair) only: a thread whose stride keeps its pair (block size a
    // multiple of D/2, the decode step's case) evaluates the double-precision range reduction once.
    int cached_pos = -1, cached_j = -1;
    float c = 1.f, s = 0.f;
#pragma unroll 2
    for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < items; idx += gridDim.x * blockDim.x) {
        const int j = idx % half;
        const int hs = (idx / half) % slots;
        const int i = idx / (half * slots);
        const int slot_pos = len0 + i;
        const int rope_pos = a.pos_base + pos_off + slot_pos;
        int d0 = 2 * j, d1 = 2 * j + 1;
        if (a.rope_mode == GRL_ROPE_HALF) { d0 = j; d1 = j + half; }
        if (a.rope_mode != GRL_ROPE_NONE && (slot_pos != cached_pos || j != cached_j)) {
            rope_sincos(rope_pos, a.freq.inv_freq[j], &c, &s);
            cached_pos = slot_pos; cached_j = j;
        }
        if (hs < a.Hkv) {
            if (a.skip_kv) continue;
            const int page = a.block_table[(size_t)b * a.max_pages + slot_pos / a.P];
            const int slot = slot_pos % a.P;
            const size_t src = (((size_t)b * a.n_new + i) * a.Hkv + hs) * a.D;
            const size_t dst = (((size_t)page * a.Hkv + hs) * a.P + slot) * a.D;
            const float k0 = a.k_new[src + d0], k1 = a.k_new[src + d1];
            const float v0 = a.v_new[src + d0], v1 = a.v_new[src + d1];
            store_from_float<T>(kp + dst + d0, k0 * c - k1 * s);
            store_from_float<T>(kp + dst + d1, k0 * s + k1 * c);
            store_from_float<T>(vp + dst + d0, v0);
            store_from_float<T>(vp + dst + d1, v1);
        } else {
            const size_t qo = (((size_t)b * a.n_new + i) * a.Hq + (hs - a.Hkv)) * a.D;
            const float q0 = a.q_in[qo + d0], q1 = a.q_in[qo + d1];
            a.q_out[qo + d0] = q0 * c - q1 * s;
            a.q_out[qo + d1] = q0 * s + q1 * c;
        }
    }
    if (a.update_lens) {  // gridDim.x == 1 here
        __syncthreads();
        if (threadIdx.x == 0) a.seq_lens[b] = len0 + a.n_new;
    }
}

// Append, head_dim a multiple of 8 and rows on 16-byte boundaries.  Bound by HBM (float32 in, cache elements out), so a
// thread moves 8 elements of a row (two 16-byte loads, one 16-byte store of bf16), two heads of keys and values in flight.
// It owns four rotation pairs of ONE token and walks that token's heads: the double-precision angle reduction, once per
// (token, head, pair) in the element-wise kernel above and most of its time, runs once per (token, pair).  Measured (4 x 2048
// tokens x 8 kv heads x 128, bf16, RoPE; 100 MB): 61 us before, 20 us now (5.0 TB/s).
constexpr int kAppendHeads = 2;
template <typename T>
__device__ __forceinline__ void store8(T* row, int o0, int o1, const float (&y)[8]);
template <>
__device__ __forceinline__ void store8<float>(float* row, int o0, int o1, const float (&y)[8]) {
    *reinterpret_cast<float4*>(row + o0) = make_float4(y[0], y[1], y[2], y[3]);
    *reinterpret_cast<float4*>(row + o1) = make_float4(y[4], y[5], y[6], y[7]);
}
template <>
__device__ __forceinline__ void store8<__nv_bfloat16>(__nv_bfloat16* row, int o0, int o1, const float (&y)[8]) {
    uint32_t w[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const __nv_bfloat162 v = __floats2bfloat162_rn(y[2 * e], y[2 * e + 1]);
        w[e] = *reinterpret_cast<const uint32_t*>(&v);
    }
    if (o1 == o0 + 4) *reinterpret_cast<uint4*>(row + o0) = make_uint4(w[0], w[1], w[2], w[3]);
    else {
        *reinterpret_cast<uint2*>(row + o0) = make_uint2(w[0], w[1]);
        *reinterpret_cast<uint2*>(row + o1) = make_uint2(w[2], w[3]);
    }
}
// y = the eight elements x[0..3] at o0, x[4..7] at o1, rotated: neighbours (interleaved) or x[e] with x[e + 4] (half)
__device__ __forceinline__ void rotate8(const float4 lo, const float4 hi, int mode, const float (&c)[4], const float (&s)[4], float (&y)[8]) {
    const float x[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        if (mode == GRL_ROPE_INTERLEAVED) {
            y[2 * e] = x[2 * e] * c[e] - x[2 * e + 1] * s[e];
            y[2 * e + 1] = x[2 * e] * s[e] + x[2 * e + 1] * c[e];
        } else if (mode == GRL_ROPE_HALF) {
            y[e] = x[e] * c[e] - x[e + 4] * s[e];
            y[e + 4] = x[e] * s[e] + x[e + 4] * c[e];
        } else {
            y[2 * e] = x[2 * e];
            y[2 * e + 1] = x[2 * e + 1];
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(256, 3) kv_append_rows_kernel(const __grid_constant__ AppendArgs a) {
    __shared__ double freq[128];        // lanes index the frequencies apart, which the constant bank would serialise
    const int b = blockIdx.y, lanes = a.D / 8, groups = 256 / lanes;
    const int group = threadIdx.x / lanes, l = threadIdx.x % lanes;
    if (a.rope_mode != GRL_ROPE_NONE && threadIdx.x < a.D / 2) freq[threadIdx.x] = a.freq.inv_freq[threadIdx.x];
    pdl_wait();
    pdl_trigger();      // the decode that follows sets itself up meanwhile
    const int len0 = a.seq_lens[b];
    const int pos0 = a.pos_base + (a.pos_offsets ? a.pos_offsets[b] : 0) + len0;
    // A token's runs: pairs of kv heads, then pairs of query heads.  Every thread group takes an equal, contiguous share of
    // all (token, run): the CTAs that fit the SMs at once are busy to the end, and the angles change only with the token.
    const int kv_runs = a.skip_kv ? 0 : (a.Hkv + kAppendHeads - 1) / kAppendHeads;
    const int runs = kv_runs + (a.q_in ? (a.Hq + kAppendHeads - 1) / kAppendHeads : 0);
    const int o0 = a.rope_mode == GRL_ROPE_HALF ? 4 * l : 8 * l, o1 = a.rope_mode == GRL_ROPE_HALF ? o0 + a.D / 2 : o0 + 4;
    const long long total = (long long)a.n_new * runs, all = (long long)gridDim.x * groups, mine = (long long)blockIdx.x * groups + group;
    const long long lo = group < groups ? mine * total / all : 0, hi = group < groups ? (mine + 1) * total / all : 0;
    float4 k[kAppendHeads][2], v[kAppendHeads][2];
    auto fetch = [&](int i, int r) {
        const bool is_kv = r < kv_runs;
        const int h0 = (is_kv ? r : r - kv_runs) * kAppendHeads, heads = is_kv ? a.Hkv : a.Hq;
        const size_t src = (((size_t)b * a.n_new + i) * heads + h0) * a.D;
        const float* in = (is_kv ? a.k_new : a.q_in) + src;
#pragma unroll
        for (int h = 0; h < kAppendHeads; ++h)
            if (h0 + h < heads) {
                k[h][0] = __ldcs(reinterpret_cast<const float4*>(in + h * a.D + o0));
                k[h][1] = __ldcs(reinterpret_cast<const float4*>(in + h * a.D + o1));
                if (is_kv) {
                    v[h][0] = __ldcs(reinterpret_cast<const float4*>(a.v_new + src + h * a.D + o0));
                    v[h][1] = __ldcs(reinterpret_cast<const float4*>(a.v_new + src + h * a.D + o1));
                }
            }
    };
    int i = (int)(lo / runs), r = (int)(lo % runs);
    if (lo < hi) fetch(i, r);           // beside the length: in a decode step the trips to memory are the time
    if (len0 < 0 || len0 + a.n_new > a.max_pages * a.P) {      // no room: nothing is stored (see kv_append_kernel)
        if (threadIdx.x == 0 && blockIdx.x == 0 && a.status && atomicCAS(a.status, 0, GRL_ERR_INVALID) == 0) {
            a.status[1] = 4 << 28;
            a.status[2] = b;
            a.status[3] = len0;
        }
        return;
    }
    __syncthreads();                    // freq
    T* kp = reinterpret_cast<T*>(a.k_pages);
    T* vp = reinterpret_cast<T*>(a.v_pages);
    {
        float c[4] = {1.f, 1.f, 1.f, 1.f}, s[4] = {0.f, 0.f, 0.f, 0.f};
        int angles_of = -1, page = 0;
        for (long long item = lo; item < hi; ++item, ++r) {
            if (r == runs) { r = 0; ++i; }
            if (item > lo) fetch(i, r);
            const int slot = len0 + i;
            const bool is_kv = r < kv_runs;
            const int h0 = (is_kv ? r : r - kv_runs) * kAppendHeads, heads = is_kv ? a.Hkv : a.Hq;
            const size_t src = (((size_t)b * a.n_new + i) * heads + h0) * a.D;
            if (angles_of != i) {       // under the first run's loads
                page = a.block_table[(size_t)b * a.max_pages + slot / a.P];
                if (a.rope_mode != GRL_ROPE_NONE) {
#pragma unroll
                    for (int e = 0; e < 4; ++e) rope_sincos(pos0 + i, freq[4 * l + e], &c[e], &s[e]);
                }
                angles_of = i;
            }
            float y[8];
#pragma unroll
            for (int h = 0; h < kAppendHeads; ++h)
                if (h0 + h < heads) {
                    rotate8(k[h][0], k[h][1], a.rope_mode, c, s, y);
                    if (is_kv) {
                        const size_t dst = (((size_t)page * a.Hkv + h0 + h) * a.P + slot % a.P) * a.D;
                        store8<T>(kp + dst, o0, o1, y);
                        rotate8(v[h][0], v[h][1], GRL_ROPE_NONE, c, s, y);
                        store8<T>(vp + dst, o0, o1, y);
                    } else {
                        store8<float>(a.q_out + src + h * a.D, o0, o1, y);
                    }
                }
        }
    }
    if (a.update_lens) {    // gridDim.x == 1 here: every thread has read len0
        __syncthreads();
        if (threadIdx.x == 0) a.seq_lens[b] = len0 + a.n_new;
    }
}

__global__ void advance_lens_kernel(int32_t* seq_lens, int B, int n, int capacity) {
    int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b < B && seq_lens[b] >= 0 && seq_lens[b] + n <= capacity) seq_lens[b] += n;   // a full sequence was skipped
}

template <typename T>
__global__ void kv_gather_kernel(const T* __restrict__ kp, const T* __restrict__ vp,
                                 const int32_t* __restrict__ block_table, int b, int n_tokens, int Hkv, int D,
                                 int P, int max_pages, float* __restrict__ out_k, float* __restrict__ out_v) {
    const size_t total = (size_t)n_tokens * Hkv * D;
    for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (size_t)gridDim.x * blockDim.x) {
        const int d = (int)(idx % D);
        const int h = (int)((idx / D) % Hkv);
        const int t = (int)(idx / ((size_t)D * Hkv));
        const int page = block_table[(size_t)b * max_pages + t / P];
        const size_t src = (((size_t)page * Hkv + h) * P + t % P) * D + d;
        out_k[idx] = load_as_float<T>(kp + src);
        out_v[idx] = load_as_float<T>(vp + src);
    }
}

// Block swizzle of cpp/src/ops/swizzle.cpp:49-123: (B,H,S,D) <-> (B,H,S_pad/W,D_pad/W,W,W), padding zero.
// One thread per element of the swizzled tensor; W consecutive threads touch W consecutive floats on
// both sides.
__global__ void swizzle_kv_kernel(const float* __restrict__ in, float* __restrict__ out, int S, int D, int W,
                                  int s_pad, int d_pad, size_t total, int reverse) {
    const int d_blocks = d_pad / W;
    for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (size_t)gridDim.x * blockDim.x) {
        const int dw = (int)(idx % W);
        const int sw = (int)((idx / W) % W);
        const int db = (int)((idx / ((size_t)W * W)) % d_blocks);
        const size_t rest = idx / ((size_t)W * W * d_blocks);
        const int sb = (int)(rest % (s_pad / W));
        const size_t bh = rest / (s_pad / W);
        const int s = sb * W + sw, d = db * W + dw;
        const bool inside = s < S && d < D;
        const size_t plain = (bh * S + s) * D + d;
        if (reverse) {
            if (inside) out[plain] = in[idx];
        } else {
            out[idx] = inside ? in[plain] : 0.f;
        }
    }
}

// ---------------------------------------------------------------------------------------------
// Quantised storage (GRL_FP8_INT4): the reference's asymmetric quantisation, cpp/src/ops/kv_cache.cpp:272-399,
// byte for byte.  One warp owns one group of 32 elements of one (token, kv head): lane = element, the group
// maximum is a warp reduction, every lane encodes its own key byte and value nibble.
__device__ __forceinline__ uint16_t scale_to_half_bits(float scale) {       // kv_cache.cpp:297-303: bit surgery
    const uint32_t b = __float_as_uint(scale);
    return (uint16_t)(((b >> 16) & 0x8000u) | (((b >> 23) - 112u) << 10) | ((b >> 13) & 0x03FFu));
}
__device__ __forceinline__ float half_bits_to_scale(uint16_t h) {           // kv_cache.cpp:517-530
    const uint32_t sign = (h >> 15) & 1u, e = (h >> 10) & 0x1Fu, m = h & 0x03FFu;
    if (e == 0) return (float)m * 5.9604644775390625e-08f;                  // ldexp(m, -24), exact
    return __uint_as_float((sign << 31) | ((e + 112u) << 23) | (m << 13));
}
// int(log2f(a)) of the reference (kv_cache.cpp:318): the float32 logarithm, truncated toward zero.  Away from the powers of
// two that is the exponent field (plus one below 1, where truncation rounds up).  Within 64 ulps of a power of two the float32
// logarithm may round to the integer: there it is taken in double and rounded to float, which is what a correctly rounded
// log2f returns (the double logarithm for every element was most of a bulk append's time).
__device__ __forceinline__ int trunc_log2f(float a) {                       // a >= 2^-9, a normal number
    const uint32_t bits = __float_as_uint(a), m = bits & 0x7fffffu;
    if (m - 64u < 0x7fffffu - 128u) {
        const int e = (int)(bits >> 23) - 127;
        return e < 0 ? e + 1 : e;
    }
    return (int)(float)log2((double)a);
}
__device__ __forceinline__ uint8_t fp8_encode(float scaled) {               // kv_cache.cpp:306-327
    scaled = fmaxf(-448.0f, fminf(448.0f, scaled));
    const int sign = scaled < 0.f ? 1 : 0;
    const float a = fabsf(scaled);
    if (a < 1.0f / 512.0f) return 0;
    int e = trunc_log2f(a);
    e = max(0, min(15, e + 7));
    const float mantissa = __fsub_rn(__fdiv_rn(a, __uint_as_float((uint32_t)(e - 7 + 127) << 23)), 1.0f);
    // a negative fraction (magnitudes below 1, whose exponent came out one too high) wraps like the reference's
    // cast does on x86-64: to int32 with truncation, low 8 bits kept
    const uint8_t mant = (uint8_t)((uint32_t)(int)__fmul_rn(mantissa, 8.0f) & 0xFFu) & 0x07u;
    return (uint8_t)((sign << 7) | (e << 3) | mant);
}
__device__ __forceinline__ float fp8_decode(uint8_t c) {                    // kv_cache.cpp:540-552
    const uint32_t s = (c >> 7) & 1u, e = (c >> 3) & 0x0Fu, m = c & 7u;
    const float v = e == 0 ? (float)m * 0.001953125f                         // m * 2^-9
                           : __uint_as_float(((e - 7u + 127u) << 23) | (m << 20));
    return s ? -v : v;
}

// One group of 32 elements of one token and kv head, an element a lane: scales, key byte, value nibble.
__device__ __forceinline__ void quantise_group(const AppendArgs& a, float kx, float vx, int page, int h, int slot, int g, int lane) {
    const int G = a.D / 32, half = a.D / 2, d = g * 32 + lane;
    uint8_t* kp = reinterpret_cast<uint8_t*>(a.k_pages);
    uint8_t* vp = reinterpret_cast<uint8_t*>(a.v_pages);
    float kmax = fabsf(kx), vmax = fabsf(vx);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        kmax = fmaxf(kmax, __shfl_xor_sync(0xffffffffu, kmax, o));
        vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
    }
    const float kscale = kmax > 0.f ? __fdiv_rn(448.0f, kmax) : 1.0f;
    const float vscale = vmax > 0.f ? __fdiv_rn(7.0f, vmax) : 1.0f;
    const size_t row = ((size_t)page * a.Hkv + h) * a.P + slot;
    kp[row * a.D + d] = fp8_encode(__fmul_rn(kx, kscale));
    int q = (int)roundf(__fmul_rn(vx, vscale)) + 8;                       // kv_cache.cpp:363-366
    q = max(0, min(15, q));
    const int q_hi = __shfl_down_sync(0xffffffffu, q, 1);
    if ((lane & 1) == 0)
        vp[((size_t)page * a.Hkv + h) * a.P * half + quant_v_off(slot, d >> 1, a.D)] =
            (uint8_t)((q & 0x0F) | ((q_hi & 0x0F) << 4));
    if (lane == 0) a.scales[row * G + g] = scale_to_half_bits(kscale);   // the value scale is dropped (:393-398)
}

// Bulk: grid (ceil(n_new*Hkv*G / warps per CTA), B), G = D/32 groups per head.
__global__ void __launch_bounds__(256) kv_append_quant_kernel(const __grid_constant__ AppendArgs a) {
    const int b = blockIdx.y, lane = threadIdx.x & 31;
    const int G = a.D / 32;
    pdl_wait();
    pdl_trigger();      // the decode that follows sets itself up meanwhile
    const int len0 = a.seq_lens[b];
    if (len0 < 0 || len0 + a.n_new > a.max_pages * a.P) {
        if (threadIdx.x == 0 && blockIdx.x == 0 && a.status && atomicCAS(a.status, 0, GRL_ERR_INVALID) == 0) {
            a.status[1] = 4 << 28;
            a.status[2] = b;
            a.status[3] = len0;
        }
        return;
    }
    const int pos_off = a.pos_offsets ? a.pos_offsets[b] : 0;
    // an item is one group of one token for a run of heads: the angles of its elements are the same for all of them
    const int half = a.D / 2, per = a.heads_per_item, runs = (a.Hkv + per - 1) / per;
    const int items = a.n_new * runs * G;
    for (int item = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); item < items; item += gridDim.x * (blockDim.x >> 5)) {
        const int g = item % G, h0 = ((item / G) % runs) * per, i = item / (G * runs);
        const int d = g * 32 + lane;
        const int slot_pos = len0 + i;
        const int page = a.block_table[(size_t)b * a.max_pages + slot_pos / a.P];
        float c = 1.f, s = 0.f;
        int d_other = d;
        bool first = true;
        if (a.rope_mode != GRL_ROPE_NONE) {
            int j;
            if (a.rope_mode == GRL_ROPE_INTERLEAVED) { j = d >> 1; first = (d & 1) == 0; d_other = d ^ 1; }
            else { j = d % half; first = d < half; d_other = first ? d + half : d - half; }
            rope_sincos(a.pos_base + pos_off + slot_pos, a.freq.inv_freq[j], &c, &s);
        }
        for (int h = h0; h < min(h0 + per, a.Hkv); ++h) {
            const size_t src = (((size_t)b * a.n_new + i) * a.Hkv + h) * a.D;
            float kx = a.k_new[src + d];
            if (a.rope_mode != GRL_ROPE_NONE) {
                const float other = a.k_new[src + d_other];
                kx = first ? kx * c - other * s : other * s + kx * c;
            }
            const float vx = a.v_new[src + d];
            quantise_group(a, kx, vx, page, h, slot_pos % a.P, g, lane);
        }
    }
}

// A decode step, or as few tokens: one CTA a sequence, a warp a (token, kv head, group of 32), and the step's queries and its length
// with them.  Latency: what does not depend on the length is read beside it, and an angle is formed once, in shared memory, for all
// heads (forming it per key element and per query pair took most of the kernel: 1 sequence x 8 kv heads, append before decode
// 8.0 -> 4.3 us of the step).
constexpr int kStepWarps = 32;
// Dynamic shared memory that the kernel does not use: it keeps the decode's CTAs (82 KiB and more) off an append's SM while there are no
// more sequences than SMs.  Beside one, half of an SM's two decode CTAs would start under the append and the other half after it, and
// a decode that needs nearly every slot took longer than behind the kernel before this one.  Append + decode, us, that kernel / sharing an SM /
// alone on it: 9 sequences x 8 kv heads x 700 tokens 21.2 / 21.8 / 18.3, 36 x 8 x 300 16.2 / 16.6 / 13.0, 18 x 8 x 300 16.8 / 17.2 / 13.7, 64 x 2 x 500 13.9
// / 13.5 / 12.7; 8 x 8 x 700 16.5 / 13.8 / 13.8, 25 x 8 x 2000 42.4 / 34.7 / 34.5, 32 x 8 x 4096 75.0 / 61.8 / 62.0.  More sequences than SMs need two
// appends an SM: 200 x 1 x 700 21.1 / 17.1.
constexpr int kStepAloneSmem = 150 * 1024;
__global__ void __launch_bounds__(32 * kStepWarps) kv_append_quant_step_kernel(const __grid_constant__ AppendArgs a) {
    __shared__ float2 cs[kStepWarps * 16];           // (cos, sin) [token][pair]: n_new * D / 2 <= 32 * 32 / 2
    const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31;
    const int G = a.D / 32, half = a.D / 2, angles = a.n_new * half;
    const bool rope = a.rope_mode != GRL_ROPE_NONE;
    const double freq = rope && tid < angles ? a.freq.inv_freq[tid % half] : 0.0;
    const int item = tid >> 5, g = item % G, h = (item / G) % a.Hkv, i = item / (G * a.Hkv), d = g * 32 + lane;
    const bool live = item < a.n_new * a.Hkv * G;
    int j = 0, d_other = d;
    bool first = true;
    if (a.rope_mode == GRL_ROPE_INTERLEAVED) { j = d >> 1; first = (d & 1) == 0; d_other = d ^ 1; }
    else if (rope) { j = d % half; first = d < half; d_other = first ? d + half : d - half; }
    pdl_wait();
    pdl_trigger();      // the decode that follows sets itself up meanwhile
    const int len0 = a.seq_lens[b], pos_off = a.pos_offsets ? a.pos_offsets[b] : 0;
    const size_t src = (((size_t)b * a.n_new + i) * a.Hkv + h) * a.D;
    float kx = 0.f, other = 0.f, vx = 0.f;
    if (live) { kx = a.k_new[src + d]; other = a.k_new[src + d_other]; vx = a.v_new[src + d]; }
    // this thread's first query pairs
    constexpr int kAhead = 2;
    const int qitems = a.q_in ? a.n_new * a.Hq * half : 0;
    float q0[kAhead], q1[kAhead];
    auto q_place = [&](int idx, int* d0, int* d1) -> size_t {
        const int jq = idx % half;
        *d0 = a.rope_mode == GRL_ROPE_HALF ? jq : 2 * jq;
        *d1 = a.rope_mode == GRL_ROPE_HALF ? jq + half : 2 * jq + 1;
        return ((size_t)b * a.n_new * a.Hq + idx / half) * a.D;
    };
#pragma unroll
    for (int e = 0; e < kAhead; ++e) {
        const int idx = tid + e * 32 * kStepWarps;
        int d0, d1;
        q0[e] = q1[e] = 0.f;
        if (idx < qitems) { const size_t qo = q_place(idx, &d0, &d1); q0[e] = a.q_in[qo + d0]; q1[e] = a.q_in[qo + d1]; }
    }
    if (len0 < 0 || len0 + a.n_new > a.max_pages * a.P) {
        if (tid == 0 && a.status && atomicCAS(a.status, 0, GRL_ERR_INVALID) == 0) {
            a.status[1] = 4 << 28;
            a.status[2] = b;
            a.status[3] = len0;
        }
        return;
    }
    const int slot_pos = len0 + i;
    const int page = live ? a.block_table[(size_t)b * a.max_pages + slot_pos / a.P] : 0;
    if (rope && tid < angles) {
        float c, s;
        rope_sincos(a.pos_base + pos_off + len0 + tid / half, freq, &c, &s);
        cs[tid] = make_float2(c, s);
    }
    __syncthreads();
    if (live) {
        if (rope) {
            const float c = cs[i * half + j].x, s = cs[i * half + j].y;
            kx = first ? kx * c - other * s : other * s + kx * c;
        }
        quantise_group(a, kx, vx, page, h, slot_pos % a.P, g, lane);
    }
    auto rotate_q = [&](int idx, float x0, float x1) {
        int d0, d1;
        const size_t qo = q_place(idx, &d0, &d1);
        float c = 1.f, s = 0.f;
        if (rope) { const float2 v = cs[idx / (half * a.Hq) * half + idx % half]; c = v.x; s = v.y; }
        a.q_out[qo + d0] = x0 * c - x1 * s;
        a.q_out[qo + d1] = x0 * s + x1 * c;
    };
#pragma unroll
    for (int e = 0; e < kAhead; ++e)
        if (tid + e * 32 * kStepWarps < qitems) rotate_q(tid + e * 32 * kStepWarps, q0[e], q1[e]);
    for (int idx = tid + kAhead * 32 * kStepWarps; idx < qitems; idx += 32 * kStepWarps) {
        int d0, d1;
        const size_t qo = q_place(idx, &d0, &d1);
        rotate_q(idx, a.q_in[qo + d0], a.q_in[qo + d1]);
    }
    if (a.update_lens && tid == 0) a.seq_lens[b] = len0 + a.n_new;      // every warp has read len0: the barrier above
}

// Dequantise sequence b as token-major float32 (T, Hkv, D): kv_cache.cpp:500-577.  One thread per element.
__global__ void kv_gather_quant_kernel(const uint8_t* __restrict__ kp, const uint8_t* __restrict__ vp,
                                       const uint16_t* __restrict__ scales, const int32_t* __restrict__ block_table,
                                       int b, int n_tokens, int Hkv, int D, int P, int max_pages,
                                       float* __restrict__ out_k, float* __restrict__ out_v) {
    const size_t total = (size_t)n_tokens * Hkv * D;
    for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (size_t)gridDim.x * blockDim.x) {
        const int d = (int)(idx % D);
        const int h = (int)((idx / D) % Hkv);
        const int t = (int)(idx / ((size_t)D * Hkv));
        const int page = block_table[(size_t)b * max_pages + t / P];
        const size_t row = ((size_t)page * Hkv + h) * P + t % P;
        const float scale = half_bits_to_scale(scales[row * (D / 32) + d / 32]);
        const float inv = scale > 0.f ? __fdiv_rn(1.0f, scale) : 1.0f;
        out_k[idx] = __fmul_rn(fp8_decode(kp[row * D + d]), inv);
        const uint8_t packed = vp[((size_t)page * Hkv + h) * P * (D / 2) + quant_v_off(t % P, d >> 1, D)];
        const int q = (d & 1) ? (packed >> 4) & 0x0F : packed & 0x0F;
        out_v[idx] = __fmul_rn((float)(q - 8), inv);
    }
}

// C = A B, all row-major float32: the reference's gemm_mnk shader (shaders/gemm_mnk.glsl:34-80), which the MLA
// latent path dispatches (cpp/src/ops/kv_cache.cpp:216-234, :441-498): 16 x 16 tiles in shared memory, the sum
// over k in ascending order with separate multiplies and adds.
__global__ void __launch_bounds__(256) gemm_f32_kernel(const float* __restrict__ A, const float* __restrict__ B,
                                                        float* __restrict__ C, int M, int K, int N) {
    __shared__ float As[16][17], Bs[16][17];
    const int lx = threadIdx.x & 15, ly = threadIdx.x >> 4;
    const int m = blockIdx.y * 16 + ly, n = blockIdx.x * 16 + lx;
    float acc = 0.f;
    for (int k0 = 0; k0 < K; k0 += 16) {
        As[ly][lx] = (m < M && k0 + lx < K) ? A[(size_t)m * K + k0 + lx] : 0.f;
        Bs[ly][lx] = (n < N && k0 + ly < K) ? B[(size_t)(k0 + ly) * N + n] : 0.f;
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < 16; ++kk) acc = __fadd_rn(acc, __fmul_rn(As[ly][kk], Bs[kk][lx]));
        __syncthreads();
    }
    if (m < M && n < N) C[(size_t)m * N + n] = acc;
}

// rows x [K (D) | V (D)] <-> separate (rows, D) K and V: the concatenation in front of the MLA down-projection
// (kv_cache.cpp:190-203) and the split behind the up-projection (:483-494).
__global__ void mla_concat_kernel(const float* __restrict__ k, const float* __restrict__ v, float* __restrict__ out,
                                  size_t rows, int D) {
    const size_t total = rows * 2 * D;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const size_t r = i / (2 * D);
        const int c = (int)(i % (2 * D));
        out[i] = c < D ? k[r * D + c] : v[r * D + c - D];
    }
}
__global__ void mla_split_kernel(const float* __restrict__ in, float* __restrict__ k, float* __restrict__ v,
                                 size_t rows, int D) {
    const size_t total = rows * 2 * D;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const size_t r = i / (2 * D);
        const int c = (int)(i % (2 * D));
        if (c < D) k[r * D + c] = in[i];
        else v[r * D + c - D] = in[i];
    }
}

// kv_append_rows_kernel: rows of whole 8-element pieces, everything on 16-byte boundaries
static bool append_rows_fit(const AppendArgs& a) {
    const uintptr_t all = (uintptr_t)a.k_new | (uintptr_t)a.v_new | (uintptr_t)a.q_in | (uintptr_t)a.q_out | (uintptr_t)a.k_pages | (uintptr_t)a.v_pages;
    return a.D % 8 == 0 && all % 16 == 0;
}
// One (token, run of heads) a thread group while that leaves SMs idle, the CTAs that are resident at once beyond.
static dim3 append_rows_grid(grl_device* dev, const AppendArgs& a) {
    const int runs = (a.skip_kv ? 0 : (a.Hkv + kAppendHeads - 1) / kAppendHeads) + (a.q_in ? (a.Hq + kAppendHeads - 1) / kAppendHeads : 0);
    const int groups = 256 / (a.D / 8);
    const long long ctas = ((long long)a.n_new * runs + groups - 1) / groups, resident = (3LL * dev->prop.multiProcessorCount + a.B - 1) / a.B;
    return dim3((unsigned)(ctas < resident ? ctas : resident), a.B);
}

static int check_layout(const grl_kv_layout& kv) {
    GRL_REQUIRE(kv.k_pages && kv.v_pages && kv.block_table && kv.seq_lens, "NULL cache pointer");
    GRL_REQUIRE(kv.batch > 0 && kv.num_kv_heads > 0 && kv.page_tokens > 0 && kv.max_pages > 0, "bad cache shape");
    GRL_REQUIRE(kv.head_dim > 0 && kv.head_dim % 2 == 0 && kv.head_dim <= 256, "head_dim must be even and <= 256");
    GRL_REQUIRE(kv.cache_dtype == GRL_BF16 || kv.cache_dtype == GRL_F32 || kv.cache_dtype == GRL_FP8_INT4,
                "unknown cache dtype");
    if (kv.cache_dtype == GRL_FP8_INT4) {
        GRL_REQUIRE(kv.scales, "the quantised cache needs its scales buffer");
        GRL_REQUIRE(kv.head_dim % 32 == 0, "the quantised cache needs head_dim to be a multiple of 32 (scale groups)");
        GRL_REQUIRE(kv.page_tokens % 2 == 0, "the quantised cache stores value bytes by token pairs: page_tokens must be even");
    }
    return GRL_OK;
}

}  // namespace grl

using namespace grl;

extern "C" {

int grl_kv_append(grl_device* dev, const grl_append_params* p) {
    GRL_REQUIRE(dev && p, "NULL argument");
    int rc = check_layout(p->kv);
    if (rc) return rc;
    GRL_REQUIRE(p->k_new && p->v_new, "k_new / v_new is NULL");
    GRL_REQUIRE(p->n_new > 0, "n_new must be positive");
    GRL_REQUIRE(!p->q_in || (p->q_out && p->num_q_heads > 0), "q_in given without q_out / num_q_heads");
    GRL_REQUIRE(p->rope_mode >= GRL_ROPE_NONE && p->rope_mode <= GRL_ROPE_HALF, "unknown rope mode");
    DeviceGuard g(dev->ordinal);
    const grl_kv_layout& kv = p->kv;
    AppendArgs a{};
    a.k_pages = kv.k_pages; a.v_pages = kv.v_pages; a.block_table = kv.block_table; a.seq_lens = kv.seq_lens;
    a.k_new = p->k_new; a.v_new = p->v_new; a.q_in = p->q_in; a.q_out = p->q_out;
    a.B = kv.batch; a.Hkv = kv.num_kv_heads; a.Hq = p->num_q_heads; a.D = kv.head_dim; a.P = kv.page_tokens;
    a.max_pages = kv.max_pages; a.n_new = p->n_new;
    a.rope_mode = p->rope_mode; a.pos_base = p->pos_base; a.pos_offsets = p->pos_offsets;
    a.status = dev->d_status;
    a.scales = static_cast<uint16_t*>(kv.scales);
    dev->status_dirty = true;
    if (p->rope_mode != GRL_ROPE_NONE) a.freq = cached_rope_freq(dev, kv.head_dim, p->rope_theta, p->rope_scaling);
    if (kv.cache_dtype == GRL_FP8_INT4) {
        const long long warps = (long long)p->n_new * kv.num_kv_heads * (kv.head_dim / 32);
        if (warps <= kStepWarps) {      // a decode step: one wide CTA per sequence does keys, values, queries and the length
            a.update_lens = p->update_lens ? 1 : 0;
            const int smem = kv.batch <= dev->prop.multiProcessorCount ? kStepAloneSmem : 0;
            static bool attr_set[64] = {};
            if (!attr_set[dev->ordinal & 63]) {
                GRL_CUDA(cudaFuncSetAttribute(kv_append_quant_step_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kStepAloneSmem));
                attr_set[dev->ordinal & 63] = true;
            }
            GRL_CUDA(launch_pdl(kv_append_quant_step_kernel, dim3(kv.batch), 32 * kStepWarps, smem, dev->stream, a));
            GRL_LAUNCHED("kv_append_quant_step_kernel");
            return GRL_OK;
        }
        // Bulk: K and V by a warp per (token, kv head, group of 32), then the queries, if any, by the float32 cache's kernels.
        // Eight heads a warp once there are enough tokens to fill the SMs (64 warps each) all the same
        a.heads_per_item = warps * kv.batch / 8 >= 64LL * dev->prop.multiProcessorCount ? 8 : 1;
        int ctas = (int)((warps / a.heads_per_item + 7) / 8);
        if (ctas > 1024) ctas = 1024;
        GRL_CUDA(launch_pdl(kv_append_quant_kernel, dim3(ctas, kv.batch), 256, 0, dev->stream, a));
        GRL_LAUNCHED("kv_append_quant_kernel");
        if (p->q_in) {
            a.skip_kv = 1;
            if (append_rows_fit(a)) {
                GRL_CUDA(launch_pdl(kv_append_rows_kernel<float>, append_rows_grid(dev, a), 256, 0, dev->stream, a));
            } else {
                const long long qitems = (long long)p->n_new * (kv.num_kv_heads + p->num_q_heads) * (kv.head_dim / 2);
                const int qchunks = (int)((qitems + 4095) / 4096);
                kv_append_kernel<float><<<dim3(qchunks < 128 ? qchunks : 128, kv.batch), 256, 0, dev->stream>>>(a);
            }
            GRL_LAUNCHED("kv_append_kernel");
        }
        if (p->update_lens) {
            advance_lens_kernel<<<(kv.batch + 127) / 128, 128, 0, dev->stream>>>(kv.seq_lens, kv.batch, p->n_new,
                                                                                 kv.max_pages * kv.page_tokens);
            GRL_LAUNCHED("advance_lens_kernel");
        }
        return GRL_OK;
    }
    bool fused_update;
    if (append_rows_fit(a)) {
        dim3 grid = append_rows_grid(dev, a);
        // a decode step (or a few tokens): one CTA per sequence also advances the length, which saves a launch
        if (p->update_lens && grid.x <= 4) grid.x = 1;
        fused_update = p->update_lens && grid.x == 1;
        a.update_lens = fused_update ? 1 : 0;
        GRL_CUDA(launch_pdl(kv.cache_dtype == GRL_BF16 ? kv_append_rows_kernel<__nv_bfloat16> : kv_append_rows_kernel<float>, grid, 256, 0,
                            dev->stream, a));
    } else {
        const long long items = (long long)p->n_new * (kv.num_kv_heads + (p->q_in ? p->num_q_heads : 0)) * (kv.head_dim / 2);
        // one CTA per sequence while a CTA has at most 16 items per thread (a decode step), more for bulk appends
        int chunks = (int)((items + 4095) / 4096);
        if (chunks > 128) chunks = 128;
        fused_update = p->update_lens && chunks == 1;
        a.update_lens = fused_update ? 1 : 0;
        dim3 grid(chunks, kv.batch);
        // one chunk (the decode step): a wide CTA, so that every thread has only a few dependent load chains
        const int threads = chunks == 1 ? (items > 512 ? 1024 : 512) : 256;
        if (kv.cache_dtype == GRL_BF16) kv_append_kernel<__nv_bfloat16><<<grid, threads, 0, dev->stream>>>(a);
        else kv_append_kernel<float><<<grid, threads, 0, dev->stream>>>(a);
    }
    GRL_LAUNCHED("kv_append_kernel");
    if (p->update_lens && !fused_update) {
        advance_lens_kernel<<<(kv.batch + 127) / 128, 128, 0, dev->stream>>>(kv.seq_lens, kv.batch, p->n_new,
                                                                                 kv.max_pages * kv.page_tokens);
        GRL_LAUNCHED("advance_lens_kernel");
    }
    return GRL_OK;
}

int grl_gemm_f32(grl_device* dev, const float* a, const float* b, float* c, int m, int k, int n) {
    GRL_REQUIRE(dev && a && b && c, "NULL argument");
    GRL_REQUIRE(m > 0 && k > 0 && n > 0, "bad shape (%d,%d,%d)", m, k, n);
    DeviceGuard g(dev->ordinal);
    gemm_f32_kernel<<<dim3((n + 15) / 16, (m + 15) / 16), 256, 0, dev->stream>>>(a, b, c, m, k, n);
    GRL_LAUNCHED("gemm_f32_kernel");
    return GRL_OK;
}

int grl_mla_concat(grl_device* dev, const float* k, const float* v, float* out, size_t rows, int head_dim) {
    GRL_REQUIRE(dev && k && v && out && rows > 0 && head_dim > 0, "bad argument");
    DeviceGuard g(dev->ordinal);
    const size_t blocks = (rows * 2 * head_dim + 255) / 256;
    mla_concat_kernel<<<(unsigned)(blocks < 4096 ? blocks : 4096), 256, 0, dev->stream>>>(k, v, out, rows, head_dim);
    GRL_LAUNCHED("mla_concat_kernel");
    return GRL_OK;
}

int grl_mla_split(grl_device* dev, const float* in, float* k, float* v, size_t rows, int head_dim) {
    GRL_REQUIRE(dev && k && v && in && rows > 0 && head_dim > 0, "bad argument");
    DeviceGuard g(dev->ordinal);
    const size_t blocks = (rows * 2 * head_dim + 255) / 256;
    mla_split_kernel<<<(unsigned)(blocks < 4096 ? blocks : 4096), 256, 0, dev->stream>>>(in, k, v, rows, head_dim);
    GRL_LAUNCHED("mla_split_kernel");
    return GRL_OK;
}

int grl_swizzle_kv(grl_device* dev, const float* in, float* out, int batch, int heads, int seq_len, int head_dim,
                   int wave, int reverse) {
    GRL_REQUIRE(dev && in && out, "NULL argument");
    GRL_REQUIRE(batch > 0 && heads > 0 && seq_len > 0 && head_dim > 0 && wave > 0, "bad shape");
    DeviceGuard g(dev->ordinal);
    const int s_pad = (seq_len + wave - 1) / wave * wave, d_pad = (head_dim + wave - 1) / wave * wave;
    const size_t total = (size_t)batch * heads * s_pad * d_pad;
    const size_t blocks = (total + 255) / 256;
    swizzle_kv_kernel<<<(unsigned)(blocks < 65535 * 16 ? blocks : 65535 * 16), 256, 0, dev->stream>>>(
        in, out, seq_len, head_dim, wave, s_pad, d_pad, total, reverse ? 1 : 0);
    GRL_LAUNCHED("swizzle_kv_kernel");
    return GRL_OK;
}

int grl_kv_gather(grl_device* dev, const grl_kv_layout* kv, int b, int n_tokens, float* out_k, float* out_v) {
    GRL_REQUIRE(dev && kv, "NULL argument");
    int rc = check_layout(*kv);
    if (rc) return rc;
    GRL_REQUIRE(b >= 0 && b < kv->batch, "sequence index out of range");
    GRL_REQUIRE(n_tokens >= 0 && n_tokens <= kv->max_pages * kv->page_tokens, "n_tokens out of range");
    if (n_tokens == 0) return GRL_OK;
    GRL_REQUIRE(out_k && out_v, "NULL output");
    DeviceGuard g(dev->ordinal);
    const size_t total = (size_t)n_tokens * kv->num_kv_heads * kv->head_dim;
    int blocks = (int)((total + 255) / 256 < 4096 ? (total + 255) / 256 : 4096);
    if (kv->cache_dtype == GRL_FP8_INT4)
        kv_gather_quant_kernel<<<blocks, 256, 0, dev->stream>>>(
            (const uint8_t*)kv->k_pages, (const uint8_t*)kv->v_pages, (const uint16_t*)kv->scales, kv->block_table, b,
            n_tokens, kv->num_kv_heads, kv->head_dim, kv->page_tokens, kv->max_pages, out_k, out_v);
    else if (kv->cache_dtype == GRL_BF16)
        kv_gather_kernel<__nv_bfloat16><<<blocks, 256, 0, dev->stream>>>(
            (const __nv_bfloat16*)kv->k_pages, (const __nv_bfloat16*)kv->v_pages, kv->block_table, b, n_tokens,
            kv->num_kv_heads, kv->head_dim, kv->page_tokens, kv->max_pages, out_k, out_v);
    else
        kv_gather_kernel<float><<<blocks, 256, 0, dev->stream>>>(
            (const float*)kv->k_pages, (const float*)kv->v_pages, kv->block_table, b, n_tokens, kv->num_kv_heads,
            kv->head_dim, kv->page_tokens, kv->max_pages, out_k, out_v);
    GRL_LAUNCHED("kv_gather_kernel");
    return GRL_OK;
}

}  // extern "C"
