// The shared-memory ring of the tensor-core decode: how many stages it has, which warps fill them and which read them.
// Constants only, so that the order of its waits can be checked without a GPU.
#pragma once

#ifdef __CUDACC__
#define GRL_RING_FN __host__ __device__
#else
#define GRL_RING_FN
#endif

namespace grl {
namespace dmma {

// FORM of an instance: over the bf16 cache, over the quantised cache, and that with one CTA an SM.
enum Form { BF16 = 0, QUANT_PAIR = 1, QUANT_WIDE = 2 };
// Compute warps, in groups of four that take the ring's stages in turn (16 tokens of one a warp), and the producer warps behind
// them (stages in turn, too).  A producer's serial chain of waits and copies is some 1300 cycles a stage beside busy compute
// warps, so the quantised stages, which are small, have several (131072 tokens x 8 heads, decode alone: 15 compute warps and one
// producer 79 us, 14 and 2 64, 12 and 4 64; with the shorter conversion 12 and 1 61, 12 and 4 59; four compute warps and 1 / 2
// producers, two CTAs an SM, 66 / 65).
template <int FORM> struct Warps {
    static constexpr int COMPUTE = FORM == QUANT_WIDE ? 12 : 4, PROD = FORM == QUANT_WIDE ? 4 : FORM == QUANT_PAIR ? 2 : 1;
    static constexpr int THREADS = 32 * (COMPUTE + PROD), CTAS = FORM == QUANT_WIDE ? 1 : 2;
    static constexpr int GROUPS = COMPUTE / 4;
};
// Stages: 96 KiB in flight per CTA over the bf16 cache, 195 KiB over the quantised one with one CTA an SM.
//
// Stage i lies in slot i mod NST, is filled by producer i mod PROD and read by group i mod GROUPS.  A wait names the parity of its
// phase, and returns at once where the phase BEFORE that one has not ended; copies land in any order, so that nothing but a wait of
// the same warps tells them that it has.  Hence:
//  - full: a slot belongs to one group, NST % GROUPS == 0.  That group has waited for stage i - NST in it before it looks for stage i.
//    (With 14 stages and three groups it had not: a copy later than those issued after it would have let a group read stage i too early.)
//  - empty: the producer of stage i must know that stage i - 2 NST was read.  It issued stage i - PROD * GROUPS, for which it waited for
//    stage i - PROD * GROUPS - NST; the same group read that one, not before i - 2 NST where PROD * GROUPS <= NST.
template <int FORM, int HD> struct Stages {
    static constexpr int NST = FORM == QUANT_WIDE ? 15 : FORM == QUANT_PAIR ? 6 : 3 * 128 / HD;
    static_assert(NST % Warps<FORM>::GROUPS == 0 && Warps<FORM>::PROD * Warps<FORM>::GROUPS <= NST, "phases of a slot in order");
};

// The last stage that was issued into slot s, or -1.  issued[stride * p] is one past the last stage that producer p has issued.  After a
// wait that ran out, these stages are the only ones whose copies may still be in flight, and each is the phase its barrier is in.
template <int NST, int PROD> GRL_RING_FN int last_in_slot(const int* issued, int stride, int s) {
    int last = -1;
    for (int p = 0; p < PROD; ++p)
        for (int j = issued[stride * p] - 1, n = 0; j > last && n < NST; j -= PROD, ++n)
            if (j % NST == s) last = j;
    return last;
}

}  // namespace dmma
}  // namespace grl
