// fp32 SIMT flash-attention forward (exact path, max-abs <= 1e-4 against the fp32 oracle).
//
// Replaces the three-pass dispatch of ops::flashAttention2 (cpp/src/ops/attention.cpp:112-152)
// and the per-(q,k)-thread shaders flash-attention2.glsl / flash-attention2-rope.glsl with ONE
// launch: a CTA owns FM query rows of one (batch, head), streams K/V tiles through
// shared memory, keeps running max / sum / accumulator in registers (online softmax) and
// writes O once.  Covers every mask convention of the reference, causal and ragged lengths
// as predicates (no S x S tensor), both RoPE pairings applied while the Q/K tiles are loaded.
//
// Two shapes of CTA, 256 threads each.  FM = 64: one group of threads, 64-key tiles; bound by the FP32 pipe (packed
// multiply-adds, 16-byte shared-memory loads).  FM = 16: four groups of 64 threads take every fourth 32-key tile each, with
// a softmax state of their own, and merge at the end: a call too small to give every SM a 64-row tile is bound by the chain of
// its tiles (load, products, softmax, products), which is four times shorter this way and on four times as many SMs.
// Tiles that need no rotation are copied asynchronously, Q with the first K and V: a small CTA has few tiles, so its round trips
// to memory are much of its time.
// Measured as a host call (float32 in and out, 4 heads x 256 x 64): 138 us with 64-row CTAs alone, 130 us with both shapes and
// 110 us with the asynchronous tiles and the inputs streamed to the transfer block; 8 heads x 512 x 64: 404 and 182 us, 2 x 8
// heads x 512 x 128: 1188 and 510 us.
#include "common.cuh"

namespace grl {

constexpr float kExcluded = -1e30f;

struct FlashF32Args {
    const void* q;
    const void* k;
    const void* v;
    void* o;
    int B, H, S, D;
    float scale;
    int causal;
    const int32_t* seq_lens;
    const float* mask;
    int mask_kind;
    int rope_mode;
    const float2* rope;  // (S, D/2) cos/sin or NULL
    int vec;             // Q, K, V on 16-byte boundaries
    int wide;            // 64-row CTAs whatever the size
};

template <typename TIn>
__device__ __forceinline__ float4 load4(const TIn* p, bool vec);
template <>
__device__ __forceinline__ float4 load4<float>(const float* p, bool vec) {
    return vec ? __ldg(reinterpret_cast<const float4*>(p)) : make_float4(p[0], p[1], p[2], p[3]);
}
template <>
__device__ __forceinline__ float4 load4<__nv_bfloat16>(const __nv_bfloat16* p, bool vec) {
    if (!vec) return make_float4(load_as_float(p), load_as_float(p + 1), load_as_float(p + 2), load_as_float(p + 3));
    const uint2 w = __ldg(reinterpret_cast<const uint2*>(p));
    return make_float4(__uint_as_float(w.x << 16), __uint_as_float(w.x & 0xffff0000u), __uint_as_float(w.y << 16), __uint_as_float(w.y & 0xffff0000u));
}

// ROWS rows of D elements into [ROWS][D + 4], rotated if asked, by NT threads; rows at or past n_valid are zero.
template <typename TIn, int D, int ROWS, int NT>
__device__ __forceinline__ void load_tile(float* dst, const TIn* src, int row0, int n_valid, int rope_mode, const float2* rope, bool vec,
                                          int tid) {
    constexpr int LD = D + 4;
    if (rope_mode != GRL_ROPE_HALF) {
#pragma unroll 4
        for (int q = tid; q < ROWS * D / 4; q += NT) {
            const int r = q / (D / 4), d = (q % (D / 4)) * 4;
            float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
            if (r < n_valid) {
                x = load4<TIn>(src + (size_t)(row0 + r) * D + d, vec);
                if (rope_mode == GRL_ROPE_INTERLEAVED) {
                    const float4 t = __ldg(reinterpret_cast<const float4*>(rope + (size_t)(row0 + r) * (D / 2) + d / 2));
                    x = make_float4(x.x * t.x - x.y * t.y, x.x * t.y + x.y * t.x, x.z * t.z - x.w * t.w, x.z * t.w + x.w * t.z);
                }
            }
            *reinterpret_cast<float4*>(dst + r * LD + d) = x;
        }
    } else {
        constexpr int HALF = D / 2;
#pragma unroll 2
        for (int q = tid; q < ROWS * HALF / 4; q += NT) {
            const int r = q / (HALF / 4), d = (q % (HALF / 4)) * 4;
            float4 x = make_float4(0.f, 0.f, 0.f, 0.f), y = x;
            if (r < n_valid) {
                const TIn* p = src + (size_t)(row0 + r) * D + d;
                const float4 a = load4<TIn>(p, vec), b = load4<TIn>(p + HALF, vec);
                const float4* t = reinterpret_cast<const float4*>(rope + (size_t)(row0 + r) * HALF + d);
                const float4 t0 = __ldg(t), t1 = __ldg(t + 1);
                x = make_float4(a.x * t0.x - b.x * t0.y, a.y * t0.z - b.y * t0.w, a.z * t1.x - b.z * t1.y, a.w * t1.z - b.w * t1.w);
                y = make_float4(a.x * t0.y + b.x * t0.x, a.y * t0.w + b.y * t0.z, a.z * t1.y + b.z * t1.x, a.w * t1.w + b.w * t1.z);
            }
            *reinterpret_cast<float4*>(dst + r * LD + d) = x;
            *reinterpret_cast<float4*>(dst + r * LD + d + HALF) = y;
        }
    }
}

// The same by asynchronous copies, for float32 tiles that need no rotation: all of a tile's loads are in flight at once and none
// waits in a register.  tile_wait() before the barrier that hands the tile over.
template <int D, int ROWS, int NT>
__device__ __forceinline__ void load_tile_async(float* dst, const float* src, int row0, int n_valid, int tid) {
    constexpr int LD = D + 4;
#pragma unroll
    for (int q = tid; q < ROWS * D / 4; q += NT) {
        const int r = q / (D / 4), d = (q % (D / 4)) * 4;
        const float* from = src + (size_t)(row0 + min(r, n_valid - 1)) * D + d;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst + r * LD + d)), "l"(from),
                     "r"(r < n_valid ? 16 : 0) : "memory");
    }
}
__device__ __forceinline__ void tile_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

template <int D, int FM>
struct FlashF32Shape {
    static constexpr int G = 64 / FM;                  // groups of threads
    static constexpr int GT = 256 / G;                 // threads of a group: 16 across keys / columns x FM/4 row quads
    static constexpr int FN = FM == 64 ? 64 : 32;      // keys per tile
    static constexpr int CK = FN / 16;                 // keys per thread: tx + 16 c
    static constexpr int LD = D + 4, LP = FM + 4;      // P is stored [key][row]
    static constexpr int Q = FM * LD, KV = 2 * FN * LD + FN * LP;        // floats: once, and per group
    static constexpr int MERGE = G > 1 ? G * FM * (D + 2) : 0;           // reuses the groups' tiles
    static constexpr int TOTAL = Q + (G * KV > MERGE ? G * KV : MERGE);
    static_assert(FM % 4 == 0 && GT == 4 * FM, "thread layout");
};

template <typename TIn, typename TOut, int D, int FM>
__global__ void __launch_bounds__(256) flash_fwd_f32_kernel(FlashF32Args a) {
    using SH = FlashF32Shape<D, FM>;
    constexpr int LD = SH::LD, LP = SH::LP, FN = SH::FN, CK = SH::CK, G = SH::G, GT = SH::GT;
    constexpr int DPT = D / 16;  // output columns per thread
    constexpr int DV = DPT < 4 ? DPT : 4, ND = DPT / DV;     // columns tx*DV + e + 16*DV*n
    extern __shared__ __align__(16) float smem[];
    const int tid = threadIdx.x % GT, group = threadIdx.x / GT;
    const int tx = tid & 15, ty = tid >> 4;
    float* Qs = smem;
    float* Ks = smem + SH::Q + group * SH::KV;
    float* Vs = Ks + FN * LD;
    float* Ps = Vs + FN * LD;
    auto sync_group = [&]() {
        if (G == 1) __syncthreads();
        else asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "n"(GT) : "memory");
    };

    const int n_qt = gridDim.x;
    const int qt = a.causal ? (n_qt - 1 - blockIdx.x) : blockIdx.x;  // heavy tiles first
    const int bh = blockIdx.y, b = bh / a.H, h = bh % a.H;
    const int S = a.S;
    const int q0 = qt * FM;
    const int len = a.seq_lens ? min(a.seq_lens[b], S) : S;
    const size_t base = (size_t)bh * S * D;
    TOut* O = reinterpret_cast<TOut*>(a.o) + base;

    if (q0 >= len) {  // padded query rows are defined as zero
        for (int idx = threadIdx.x; idx < FM * D; idx += 256) {
            int r = idx / D;
            if (q0 + r < S) store_from_float<TOut>(O + (size_t)(q0 + r) * D + idx % D, 0.f);
        }
        return;
    }
    const TIn* Q = reinterpret_cast<const TIn*>(a.q) + base;
    const TIn* K = reinterpret_cast<const TIn*>(a.k) + base;
    const TIn* V = reinterpret_cast<const TIn*>(a.v) + base;

    const bool async = sizeof(TIn) == 4 && a.vec;
    if (async && a.rope_mode == GRL_ROPE_NONE) load_tile_async<D, FM, 256>(Qs, reinterpret_cast<const float*>(Q), q0, min(FM, S - q0), threadIdx.x);
    else load_tile<TIn, D, FM, 256>(Qs, Q, q0, min(FM, S - q0), a.rope_mode, a.rope, a.vec, threadIdx.x);
    auto load_kv = [&](int kt) {
        const int k0 = kt * FN, rows = min(FN, S - k0);
        if (async) load_tile_async<D, FN, GT>(Vs, reinterpret_cast<const float*>(V), k0, rows, tid);
        if (async && a.rope_mode == GRL_ROPE_NONE) load_tile_async<D, FN, GT>(Ks, reinterpret_cast<const float*>(K), k0, rows, tid);
        else load_tile<TIn, D, FN, GT>(Ks, K, k0, rows, a.rope_mode, a.rope, a.vec, tid);
        if (!async) load_tile<TIn, D, FN, GT>(Vs, V, k0, rows, GRL_ROPE_NONE, nullptr, a.vec, tid);
    };

    float m[4], l[4];
    float2 acc[4][DPT / 2];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        m[r] = kExcluded;
        l[r] = 0.f;
#pragma unroll
        for (int e = 0; e < DPT / 2; ++e) acc[r][e] = make_float2(0.f, 0.f);
    }

    int k_end = len;
    if (a.causal) k_end = min(k_end, q0 + FM);
    const int n_kt = (k_end + FN - 1) / FN;
    if (group < n_kt) load_kv(group);
    tile_wait();
    __syncthreads();      // Q is the whole CTA's

    for (int kt = group; kt < n_kt; kt += G) {
        const int k0 = kt * FN;
        if (kt != group) {
            sync_group();     // previous tile's Ks/Vs/Ps fully consumed
            load_kv(kt);
            tile_wait();
            sync_group();
        }

        float2 s2[4][CK];       // even and odd elements of d
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c = 0; c < CK; ++c) s2[r][c] = make_float2(0.f, 0.f);
#pragma unroll 4
        for (int d = 0; d < D; d += 4) {
            float4 qv[4], kv[CK];
#pragma unroll
            for (int r = 0; r < 4; ++r) qv[r] = *reinterpret_cast<const float4*>(&Qs[(ty * 4 + r) * LD + d]);
#pragma unroll
            for (int c = 0; c < CK; ++c) kv[c] = *reinterpret_cast<const float4*>(&Ks[(tx + 16 * c) * LD + d]);
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < CK; ++c) {
                    s2[r][c] = __ffma2_rn(make_float2(qv[r].x, qv[r].y), make_float2(kv[c].x, kv[c].y), s2[r][c]);
                    s2[r][c] = __ffma2_rn(make_float2(qv[r].z, qv[r].w), make_float2(kv[c].z, kv[c].w), s2[r][c]);
                }
        }

        float p[4][CK];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int qi = q0 + ty * 4 + r;
            float mx = kExcluded;
            bool valid[CK];
#pragma unroll
            for (int c = 0; c < CK; ++c) {
                const int kj = k0 + tx + 16 * c;
                bool ok = (kj < len) && (qi < S) && (!a.causal || kj <= qi);
                float sc = (s2[r][c].x + s2[r][c].y) * a.scale;
                if (ok && a.mask_kind != GRL_MASK_NONE) {
                    float mv;
                    if (a.mask_kind == GRL_MASK_KEY) mv = a.mask[(size_t)b * S + kj];
                    else if (a.mask_kind == GRL_MASK_BSS) mv = a.mask[((size_t)b * S + qi) * S + kj];
                    else mv = a.mask[(((size_t)b * a.H + h) * S + qi) * S + kj];
                    if (!(mv > 0.f)) sc = -1e9f;  // replaced, not added (tests/test_attention.py:30)
                }
                valid[c] = ok;
                p[r][c] = sc;
                if (ok) mx = fmaxf(mx, sc);
            }
#pragma unroll
            for (int off = 1; off < 16; off <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
            const float m_new = fmaxf(m[r], mx);
            float rs = 0.f;
#pragma unroll
            for (int c = 0; c < CK; ++c) {
                p[r][c] = valid[c] ? expf(p[r][c] - m_new) : 0.f;
                rs += p[r][c];
            }
#pragma unroll
            for (int off = 1; off < 16; off <<= 1) rs += __shfl_xor_sync(0xffffffffu, rs, off);
            const float corr = expf(m[r] - m_new);  // both finite (kExcluded is finite)
            l[r] = l[r] * corr + rs;
            m[r] = m_new;
#pragma unroll
            for (int e = 0; e < DPT / 2; ++e) acc[r][e] = __fmul2_rn(acc[r][e], make_float2(corr, corr));
        }
#pragma unroll
        for (int c = 0; c < CK; ++c)
            *reinterpret_cast<float4*>(&Ps[(tx + 16 * c) * LP + ty * 4]) = make_float4(p[0][c], p[1][c], p[2][c], p[3][c]);
        sync_group();

#pragma unroll 4
        for (int kk = 0; kk < FN; ++kk) {
            const float4 pr = *reinterpret_cast<const float4*>(&Ps[kk * LP + ty * 4]);
            const float pv[4] = {pr.x, pr.y, pr.z, pr.w};
#pragma unroll
            for (int n = 0; n < ND; ++n) {
                float2 vv[DV / 2];
                if constexpr (DV == 4) {
                    const float4 v4 = *reinterpret_cast<const float4*>(&Vs[kk * LD + tx * 4 + 64 * n]);
                    vv[0] = make_float2(v4.x, v4.y);
                    vv[1] = make_float2(v4.z, v4.w);
                } else {
                    vv[0] = *reinterpret_cast<const float2*>(&Vs[kk * LD + tx * 2]);
                }
#pragma unroll
                for (int r = 0; r < 4; ++r)
#pragma unroll
                    for (int e = 0; e < DV / 2; ++e)
                        acc[r][n * (DV / 2) + e] = __ffma2_rn(make_float2(pv[r], pv[r]), vv[e], acc[r][n * (DV / 2) + e]);
            }
        }
    }

    if constexpr (G > 1) {
        // merge the groups: [G][FM][D] accumulators, [G][FM] maxima and sums over the tiles
        __syncthreads();
        float* sm_acc = smem + SH::Q;
        float* sm_ml = sm_acc + G * FM * D;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int row = group * FM + ty * 4 + r;
#pragma unroll
            for (int n = 0; n < ND; ++n)
#pragma unroll
                for (int e = 0; e < DV / 2; ++e)
                    *reinterpret_cast<float2*>(&sm_acc[row * D + tx * DV + 16 * DV * n + 2 * e]) = acc[r][n * (DV / 2) + e];
            if (tx == 0) { sm_ml[2 * row] = m[r]; sm_ml[2 * row + 1] = l[r]; }
        }
        __syncthreads();
        for (int q = threadIdx.x; q < FM * D; q += 256) {
            const int r = q / D, d = q % D, qi = q0 + r;
            if (qi >= S) break;
            float mt = kExcluded, lt = 0.f, o = 0.f;
#pragma unroll
            for (int g = 0; g < G; ++g) mt = fmaxf(mt, sm_ml[2 * (g * FM + r)]);
#pragma unroll
            for (int g = 0; g < G; ++g) {
                const float w = expf(sm_ml[2 * (g * FM + r)] - mt);
                lt = fmaf(w, sm_ml[2 * (g * FM + r) + 1], lt);
                o = fmaf(w, sm_acc[(g * FM + r) * D + d], o);
            }
            store_from_float<TOut>(O + (size_t)qi * D + d, qi >= len || !(lt > 0.f) ? 0.f : o / lt);
        }
        return;
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int qi = q0 + ty * 4 + r;
        if (qi >= S) continue;
        const bool zero = (qi >= len) || !(l[r] > 0.f);
        const float inv = zero ? 0.f : 1.f / l[r];
#pragma unroll
        for (int n = 0; n < ND; ++n)
#pragma unroll
            for (int e = 0; e < DV / 2; ++e) {
                TOut* dst = O + (size_t)qi * D + tx * DV + 16 * DV * n + 2 * e;
                store_from_float<TOut>(dst, acc[r][n * (DV / 2) + e].x * inv);
                store_from_float<TOut>(dst + 1, acc[r][n * (DV / 2) + e].y * inv);
            }
    }
}

template <typename TIn, typename TOut, int D, int FM>
static int launch_f32(grl_device* dev, const FlashF32Args& a) {
    constexpr size_t smem = sizeof(float) * (size_t)FlashF32Shape<D, FM>::TOTAL;
    auto kern = flash_fwd_f32_kernel<TIn, TOut, D, FM>;
    GRL_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    dim3 grid((a.S + FM - 1) / FM, a.B * a.H);
    kern<<<grid, 256, smem, dev->stream>>>(a);
    GRL_LAUNCHED("flash_fwd_f32_kernel");
    return GRL_OK;
}
// 16-row CTAs while 64-row ones would not give every SM one
template <typename TIn, typename TOut, int D>
static int launch_rows(grl_device* dev, const FlashF32Args& a) {
    const long long ctas = (long long)((a.S + 63) / 64) * a.B * a.H;
    return !a.wide && ctas < dev->prop.multiProcessorCount ? launch_f32<TIn, TOut, D, 16>(dev, a) : launch_f32<TIn, TOut, D, 64>(dev, a);
}

template <typename TIn, typename TOut>
static int dispatch_d(grl_device* dev, const FlashF32Args& a) {
    switch (a.D) {
        case 32: return launch_rows<TIn, TOut, 32>(dev, a);
        case 64: return launch_rows<TIn, TOut, 64>(dev, a);
        case 128: return launch_rows<TIn, TOut, 128>(dev, a);
        default:
            return set_error(GRL_ERR_UNSUPPORTED, "head_dim %d not supported (32, 64 or 128)", a.D);
    }
}

int flash_fwd_simt(grl_device* dev, const grl_flash_params* p, float scale, const float2* rope, bool wide) {
    GRL_REQUIRE((int64_t)p->batch * p->heads <= 65535, "batch*heads above 65535 (grid y dimension of the fp32 kernel)");
    FlashF32Args a{p->q, p->k, p->v, p->o, p->batch, p->heads, p->seq_len, p->head_dim, scale,
                   p->causal, p->seq_lens, p->mask, p->mask ? p->mask_kind : GRL_MASK_NONE,
                   p->rope_mode, rope,
                   (((uintptr_t)p->q | (uintptr_t)p->k | (uintptr_t)p->v) % 16) == 0, wide ? 1 : 0};
    if (p->in_dtype == GRL_F32 && p->out_dtype == GRL_F32) return dispatch_d<float, float>(dev, a);
    if (p->in_dtype == GRL_BF16 && p->out_dtype == GRL_F32) return dispatch_d<__nv_bfloat16, float>(dev, a);
    if (p->in_dtype == GRL_BF16 && p->out_dtype == GRL_BF16)
        return dispatch_d<__nv_bfloat16, __nv_bfloat16>(dev, a);
    if (p->in_dtype == GRL_F32 && p->out_dtype == GRL_BF16) return dispatch_d<float, __nv_bfloat16>(dev, a);
    return set_error(GRL_ERR_INVALID, "unknown dtype");
}

}  // namespace grl
