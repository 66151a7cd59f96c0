// The unfused attention pieces and the attention backward pass, for callers of the legacy three-step path.
//
// Replaces shaders/attention-scores.glsl (Q.K^T * scale into a (B,H,S,S) tensor), activation-softmax.glsl
// (three passes: row maximum, sum of exponentials, normalise), attention-output.glsl / attention-output-gpt.glsl
// (weights . V, the GPT form summing only over k <= q) and attention-backward.glsl (grad_V = A^T gO; grad_A = gO V^T;
// softmax backward; grad_Q, grad_K).  The fused kernels are the fast path; these exist so that code written against
// the separate shaders keeps working, and so that training code has a backward.  Every product is a batched float32
// product of sgemm.cuh with the sum over the inner index in ascending order, as the shaders' loops run.
#include <type_traits>

#include "common.cuh"
#include "sgemm.cuh"

namespace grl {

using sgemm::Operand;
using sgemm::Output;
using sgemm::operand;

// Row-wise softmax of (rows, features): max from -1e10 as activation-softmax.glsl:34-84 starts it, exp(x - max) / sum.
__global__ void __launch_bounds__(256) softmax_rows_kernel(const float* __restrict__ in, float* __restrict__ out,
                                                            size_t rows, int features) {
    __shared__ float red[8];
    const size_t row = blockIdx.x;
    if (row >= rows) return;
    const float* x = in + row * features;
    float* y = out + row * features;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float mx = -1e10f;
    for (int f = tid; f < features; f += 256) mx = fmaxf(mx, x[f]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0) red[warp] = mx;
    __syncthreads();
    mx = red[0];
    for (int w = 1; w < 8; ++w) mx = fmaxf(mx, red[w]);
    __syncthreads();
    float sum = 0.f;
    for (int f = tid; f < features; f += 256) sum += expf(x[f] - mx);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0) red[warp] = sum;
    __syncthreads();
    sum = 0.f;
    for (int w = 0; w < 8; ++w) sum += red[w];
    for (int f = tid; f < features; f += 256) y[f] = expf(x[f] - mx) / sum;
}

// grad_scores[i][j] = attn[i][j] * (grad_attn[i][j] - sum_k attn[i][k] grad_attn[i][k]), in place over grad_attn
// (attention-backward.glsl pass 2, the softmax backward; the scale goes into the two products that follow).
__global__ void __launch_bounds__(256) softmax_backward_rows_kernel(const float* __restrict__ attn, float* grad, size_t rows,
                                                                     int features) {
    __shared__ float red[8];
    const size_t row = blockIdx.x;
    if (row >= rows) return;
    const float* a = attn + row * features;
    float* g = grad + row * features;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float dot = 0.f;
    for (int f = tid; f < features; f += 256) dot = fmaf(a[f], g[f], dot);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
    if (lane == 0) red[warp] = dot;
    __syncthreads();
    dot = 0.f;
    for (int w = 0; w < 8; ++w) dot += red[w];
    for (int f = tid; f < features; f += 256) g[f] = a[f] * (g[f] - dot);
}

// ---- the backward pass in three launches.  The softmax backward, gS = attn * (gA - dot) with
// dot[i] = sum_j attn[i][j] gA[i][j], is not a pass of its own: the gA product leaves, next to gA, the partial row sums
// of its tiles, and the two products that read gS form it while they stage their tiles.  The partial sums of row i wait
// in grad_v[i][0 .. tiles), which is written last.
// Measured (B4 x 12 heads x 512 tokens x 64, 6.4 GFLOP): 1244 us with 16 x 16 tiles and five launches before, 189 us now
// (34 TFLOP/s; the products alone would take 89 us at the FP32 pipe's rate).
constexpr int kMaxDotRows = 8192;       // row sums of one head that fit in shared memory beside the tiles

// The attn tile of a CTA is fetched into shared memory under its products (cp.async): read in the epilogue it was
// eight dependent trips to L2 or DRAM per thread, two thirds of this kernel's time (75 us; 22 us of FMA work).
template <typename SH> struct GradAttn {
    static constexpr int LDS = SH::BN + 4;
    static constexpr size_t SMEM = (2 * SH::TILE + SH::BM * LDS) * sizeof(float);
    static constexpr int MIN_CTAS = SH::THREADS == 256 ? 2 : 6;
};
template <typename SH>
__global__ void __launch_bounds__(SH::THREADS, GradAttn<SH>::MIN_CTAS) grad_attn_kernel(Operand GO, Operand V, Output G, const float* attn,
                                                                                        float* parts, int S, int D, int H) {
    extern __shared__ __align__(16) float dyn[];
    constexpr int LDS = GradAttn<SH>::LDS;
    float* tile = dyn + 2 * SH::TILE;   // [BM][LDS] of attn; zeros outside the tensor
    const int z = blockIdx.z, b = z / H, h = z % H;
    const int m0 = blockIdx.y * SH::BM, n0 = blockIdx.x * SH::BN;
    const float* ahead = attn + (size_t)z * S * S;
    const bool vec = ((uintptr_t)attn % 16 == 0) && S % 4 == 0;
    for (int q = threadIdx.x; q < SH::BM * SH::BN / 4; q += SH::THREADS) {
        const int r = q / (SH::BN / 4), c = (q % (SH::BN / 4)) * 4;
        float* dst = tile + r * LDS + c;
        if (vec && m0 + r < S && n0 + c < S)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
                         "l"(ahead + (size_t)(m0 + r) * S + n0 + c) : "memory");
        else
            *reinterpret_cast<float4*>(dst) = m0 + r < S ? sgemm::load4(ahead + (size_t)(m0 + r) * S, n0 + c, S, false) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    float2 acc[8][4];
    sgemm::mainloop<SH, true, true, false, false>(acc, dyn, GO.base + b * GO.sb + h * GO.sh, GO, V.base + b * V.sb + h * V.sh, V, m0, n0, S,
                                                  S, D, nullptr, nullptr);
    sgemm::store_tile<SH>(acc, G.base + b * G.sb + h * G.sh, G.ld, m0, n0, S, S, 1.f, nullptr);
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    const sgemm::Place<SH> at(threadIdx.x);
    float* red = dyn;                   // [WARPS_N][BM]
    const int lane = threadIdx.x & 31, wn = (threadIdx.x >> 5) % SH::WARPS_N;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        float dot = 0.f;
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
            const float4 a = *reinterpret_cast<const float4*>(tile + at.row(i) * LDS + at.col(4 * hh));
            dot = fmaf(a.x, acc[i][2 * hh].x, dot); dot = fmaf(a.y, acc[i][2 * hh].y, dot);
            dot = fmaf(a.z, acc[i][2 * hh + 1].x, dot); dot = fmaf(a.w, acc[i][2 * hh + 1].y, dot);
        }
#pragma unroll
        for (int o = SH::LANES_N / 2; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
        if (lane % SH::LANES_N == 0) red[wn * SH::BM + at.row(i)] = dot;
    }
    __syncthreads();
    for (int r = threadIdx.x; r < SH::BM; r += SH::THREADS) {
        if (m0 + r >= S) break;
        float dot = red[r];
        for (int w = 1; w < SH::WARPS_N; ++w) dot += red[w * SH::BM + r];
        parts[((size_t)z * S + m0 + r) * D + blockIdx.x] = dot;
    }
}

// blockIdx.z < batch * H: grad_Q[i][d] = scale sum_j gS[i][j] K[j][d]; the other half: grad_K[j][d] = scale sum_i gS[i][j] Q[i][d].
// SPLIT: the K range over four thread groups (see sgemm::split_tile).
template <typename SH, bool SPLIT> struct GradQK {
    static constexpr int THREADS = SPLIT ? sgemm::Split<SH>::THREADS : SH::THREADS;
    static constexpr int MIN_CTAS = SPLIT ? sgemm::Split<SH>::MIN_CTAS : SH::MIN_CTAS;
    static constexpr int TILES = SPLIT ? sgemm::Split<SH>::SMEM / 4 : 2 * SH::TILE;      // floats
};
template <typename SH, bool SPLIT>
__global__ void __launch_bounds__(GradQK<SH, SPLIT>::THREADS, GradQK<SH, SPLIT>::MIN_CTAS)
grad_qk_kernel(const float* __restrict__ attn, const float* __restrict__ ga, const float* __restrict__ q, const float* __restrict__ k,
               const float* __restrict__ parts, int n_parts, float* gq, float* gk, int S, int D, int n_bh, int vec_s, int vec_d, float scale) {
    extern __shared__ __align__(16) float dyn[];      // two tile stages, then the row sums of this head
    float* dots = dyn + GradQK<SH, SPLIT>::TILES;
    const bool is_q = (int)blockIdx.z < n_bh;
    const int z = is_q ? blockIdx.z : blockIdx.z - n_bh;
    const int m0 = blockIdx.y * SH::BM, n0 = blockIdx.x * SH::BN;
    const int d0 = is_q ? m0 : 0, d1 = is_q ? min(S, m0 + SH::BM) : S;          // rows whose sums this CTA needs
    for (int i = d0 + threadIdx.x; i < d1; i += GradQK<SH, SPLIT>::THREADS) {
        const float* p = parts + ((size_t)z * S + i) * D;
        float dot = 0.f;
        for (int j = 0; j < n_parts; ++j) dot += __ldg(p + j);
        dots[i - d0] = dot;
    }
    __syncthreads();
    pdl_trigger();      // the row sums are read: the grad_V product, which overwrites them, may take the idle SMs
    const size_t so = (size_t)z * S * S, to = (size_t)z * S * D;
    const Operand A{ga + so, 0, 0, S, vec_s}, B{(is_q ? k : q) + to, 0, 0, D, vec_d};
    if constexpr (SPLIT) {
        float* c = (is_q ? gq : gk) + to;
        if (is_q) sgemm::split_tile<SH, true, false, true>(dyn, A.base, A, B.base, B, c, D, nullptr, m0, n0, S, D, S, scale, attn + so, dots - m0);
        else sgemm::split_tile<SH, false, false, true>(dyn, A.base, A, B.base, B, c, D, nullptr, m0, n0, S, D, S, scale, attn + so, dots);
        return;
    }
    float2 acc[8][4];
    if (is_q) sgemm::mainloop<SH, true, false, false, true>(acc, dyn, A.base, A, B.base, B, m0, n0, S, D, S, attn + so, dots - m0);
    else sgemm::mainloop<SH, false, false, false, true>(acc, dyn, A.base, A, B.base, B, m0, n0, S, D, S, attn + so, dots);
    sgemm::store_tile<SH>(acc, (is_q ? gq : gk) + to, D, m0, n0, S, D, scale, nullptr);
}

template <typename SH>
static int launch_grad_attn(grl_device* dev, const Operand& go, const Operand& v, const Output& g, const float* attn, float* parts, int S,
                            int D, int batch, int H) {
    dim3 grid((S + SH::BN - 1) / SH::BN, (S + SH::BM - 1) / SH::BM, batch * H);
    GRL_CUDA(cudaFuncSetAttribute(grad_attn_kernel<SH>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GradAttn<SH>::SMEM));
    grad_attn_kernel<SH><<<grid, SH::THREADS, GradAttn<SH>::SMEM, dev->stream>>>(go, v, g, attn, parts, S, D, H);
    GRL_LAUNCHED("grad_attn_kernel");
    return GRL_OK;
}

template <typename SH, bool SPLIT>
static int launch_grad_qk(grl_device* dev, const float* attn, const float* ga, const float* q, const float* k, const float* parts,
                          int n_parts, float* gq, float* gk, int S, int D, int n_bh, float scale) {
    const size_t smem = (GradQK<SH, SPLIT>::TILES + (size_t)S) * sizeof(float);
    GRL_CUDA(cudaFuncSetAttribute(grad_qk_kernel<SH, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (GradQK<SH, SPLIT>::TILES + kMaxDotRows) * 4));
    const int vec_s = S % 4 == 0 && (uintptr_t)attn % 16 == 0 && (uintptr_t)ga % 16 == 0;
    const int vec_d = D % 4 == 0 && (uintptr_t)q % 16 == 0 && (uintptr_t)k % 16 == 0;
    dim3 grid((D + SH::BN - 1) / SH::BN, (S + SH::BM - 1) / SH::BM, 2 * n_bh);
    grad_qk_kernel<SH, SPLIT><<<grid, GradQK<SH, SPLIT>::THREADS, smem, dev->stream>>>(attn, ga, q, k, parts, n_parts, gq, gk, S, D, n_bh, vec_s, vec_d, scale);
    GRL_LAUNCHED("grad_qk_kernel");
    return GRL_OK;
}

}  // namespace grl

using namespace grl;

extern "C" {

int grl_attention_scores(grl_device* dev, const float* q, const float* k, float* scores, int batch, int seq_len, int heads,
                         int head_dim, float scale) {
    GRL_REQUIRE(dev && q && k && scores, "NULL argument");
    GRL_REQUIRE(batch > 0 && seq_len > 0 && heads > 0 && head_dim > 0, "bad shape");
    DeviceGuard g(dev->ordinal);
    const long long S = seq_len, H = heads, D = head_dim;
    if (scale == 0.f) scale = 1.f / sqrtf((float)head_dim);
    // Q, K: (B,S,H,D); scores (B,H,S,S)
    return sgemm::launch<true, true>(dev, operand(q, S * H * D, D, H * D), operand(k, S * H * D, D, H * D),
                                     Output{scores, H * S * S, S * S, S}, nullptr, seq_len, seq_len, head_dim, batch, heads, scale,
                                     "attention_scores");
}

int grl_softmax(grl_device* dev, const float* in, float* out, size_t rows, int features) {
    GRL_REQUIRE(dev && in && out, "NULL argument");
    GRL_REQUIRE(rows > 0 && features > 0, "bad shape");
    GRL_REQUIRE(rows <= 0x7fffffffull, "too many rows");
    DeviceGuard g(dev->ordinal);
    softmax_rows_kernel<<<(unsigned)rows, 256, 0, dev->stream>>>(in, out, rows, features);
    GRL_LAUNCHED("softmax_rows_kernel");
    return GRL_OK;
}

int grl_attention_output(grl_device* dev, const float* weights, const float* v, float* out, int batch, int seq_len,
                         int heads, int head_dim, int causal) {
    GRL_REQUIRE(dev && weights && v && out, "NULL argument");
    GRL_REQUIRE(batch > 0 && seq_len > 0 && heads > 0 && head_dim > 0, "bad shape");
    DeviceGuard g(dev->ordinal);
    const long long S = seq_len, H = heads, D = head_dim;
    // weights (B,H,S,S); V, out (B,S,H,D)
    const Operand A = operand(weights, H * S * S, S * S, S), B = operand(v, S * H * D, D, H * D);
    const Output C{out, S * H * D, D, H * D};
    if (causal)
        return sgemm::launch<true, false, true>(dev, A, B, C, nullptr, seq_len, head_dim, seq_len, batch, heads, 1.f, "attention_output");
    return sgemm::launch<true, false>(dev, A, B, C, nullptr, seq_len, head_dim, seq_len, batch, heads, 1.f, "attention_output");
}

int grl_attention_backward(grl_device* dev, const float* grad_out, const float* q, const float* k, const float* v,
                           const float* attn, float* grad_q, float* grad_k, float* grad_v, float* scratch, int batch,
                           int heads, int seq_len, int head_dim, float scale) {
    GRL_REQUIRE(dev && grad_out && q && k && v && attn && grad_q && grad_k && grad_v && scratch, "NULL argument");
    GRL_REQUIRE(batch > 0 && seq_len > 0 && heads > 0 && head_dim > 0, "bad shape");
    DeviceGuard g(dev->ordinal);
    const long long S = seq_len, H = heads, D = head_dim;
    if (scale == 0.f) scale = 1.f / sqrtf((float)head_dim);
    // all of Q, K, V, grad_out and the three gradients: (B,H,S,D); attn, scratch: (B,H,S,S)
    const long long qb = H * S * D, qh = S * D, ab = H * S * S, ah = S * S;
    const size_t rows = (size_t)batch * heads * seq_len;
    GRL_REQUIRE(rows <= 0x7fffffffull, "too many rows");
    const Operand go_rows = operand(grad_out, qb, qh, D), v_rows = operand(v, qb, qh, D);
    const Output g_attn{scratch, ab, ah, S};
    // gA[i][j] = sum_d gO[i][d] V[j][d] -> scratch, with the row sums of attn * gA on the side when grad_v has room for
    // them (a column per tile) and both products that read them can hold a head's sums in shared memory
    const int sms = dev->prop.multiProcessorCount, n_bh = batch * heads;
    const bool wide = sgemm::tile_rows(seq_len, seq_len, n_bh, 128, sms) == 128;
    const int n_parts = (seq_len + (wide ? 127 : 63)) / (wide ? 128 : 64);
    int rc;
    if (n_parts <= head_dim && seq_len <= kMaxDotRows && 2LL * n_bh <= 65535) {
        rc = wide ? launch_grad_attn<sgemm::Shape<128, 128>>(dev, go_rows, v_rows, g_attn, attn, grad_v, seq_len, head_dim, batch, heads)
                  : launch_grad_attn<sgemm::Shape<64, 64>>(dev, go_rows, v_rows, g_attn, attn, grad_v, seq_len, head_dim, batch, heads);
        if (rc) return rc;
        auto qk = [&](auto shape, auto split) {
            return launch_grad_qk<decltype(shape), decltype(split)::value>(dev, attn, scratch, q, k, grad_v, n_parts, grad_q, grad_k, seq_len, head_dim, n_bh, scale);
        };
        const int tile = sgemm::tile_rows(seq_len, head_dim, 3 * n_bh, 64, sms);    // the grad_V product runs beside these two
        const bool split = sgemm::split_pays(seq_len);
        if (head_dim <= 32) rc = split ? qk(sgemm::Shape<64, 32>(), std::true_type()) : qk(sgemm::Shape<64, 32>(), std::false_type());
        else if (tile == 128) rc = qk(sgemm::Shape<128, 64>(), std::false_type());
        else rc = split ? qk(sgemm::Shape<64, 64>(), std::true_type()) : qk(sgemm::Shape<64, 64>(), std::false_type());
        if (rc) return rc;
        // grad_V[j][d] = sum_i attn[i][j] gO[i][d]
        return sgemm::launch<false, false, false, true>(dev, operand(attn, ab, ah, S), go_rows, Output{grad_v, qb, qh, D}, nullptr, seq_len,
                                                        head_dim, seq_len, batch, heads, 1.f, "grad_v", tile);
    } else {
        rc = sgemm::launch<true, true>(dev, go_rows, v_rows, g_attn, nullptr, seq_len, seq_len, head_dim, batch, heads, 1.f, "grad_attn");
        if (rc) return rc;
        softmax_backward_rows_kernel<<<(unsigned)rows, 256, 0, dev->stream>>>(attn, scratch, rows, seq_len);
        GRL_LAUNCHED("softmax_backward_rows_kernel");
        rc = sgemm::launch<true, false>(dev, operand(scratch, ab, ah, S), operand(k, qb, qh, D), Output{grad_q, qb, qh, D}, nullptr, seq_len,
                                        head_dim, seq_len, batch, heads, scale, "grad_q");
        if (!rc)
            rc = sgemm::launch<false, false>(dev, operand(scratch, ab, ah, S), operand(q, qb, qh, D), Output{grad_k, qb, qh, D}, nullptr,
                                             seq_len, head_dim, seq_len, batch, heads, scale, "grad_k");
        if (rc) return rc;
    }
    return sgemm::launch<false, false>(dev, operand(attn, ab, ah, S), go_rows, Output{grad_v, qb, qh, D}, nullptr, seq_len, head_dim,
                                       seq_len, batch, heads, 1.f, "grad_v");
}

}  // extern "C"
