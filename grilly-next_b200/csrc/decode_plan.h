// How a split-KV decode is laid out on the GPU: split count, form of the kernel, cluster size and the workspace the call needs.
// Host arithmetic only.  grl_decode_pick_splits, the workspace check of grl_gqa_decode and the launch all read it here, so that they
// cannot disagree about where the partial rows of a head go.
#pragma once
#include <cstddef>

namespace grl {

constexpr int kMaxCluster = 16;            // CTAs of a thread-block cluster that merge through its shared memory
constexpr int kMaxFusedSplits = 256;       // splits (or clusters) of a head that its last CTA to arrive can merge

struct DecodeShape {
    int heads = 0;            // (sequence, kv head) pairs
    int stages = 0;           // of the longest length: 64 tokens each, pages for the generic kernel
    int sms = 0;
    int counter_slots = 0;    // heads whose arrivals can be counted
    bool mma = false;         // the tensor-core kernel, else the generic one
    bool quant = false;
    bool exchange = false;    // the rows are merged with the peers' in the same launch
    int world = 1;            // ranks of that exchange
    bool partial = false;     // the rows leave un-normalised
};

struct DecodePlan {
    int n_splits = 1;
    bool direct = false;      // one split, whose CTA writes the result itself
    bool fused = false;       // the kernel merges its splits; else a merge kernel follows
    bool wide = false;        // quantised: one CTA an SM, twelve compute warps (QUANT_WIDE)
    int cluster = 1;          // CTAs of a head that merge through distributed shared memory
    bool alone = false;       // CTAs that must not share an SM
    int parts = 0;            // splits whose rows the workspace has to hold
};

// The quantised cache's one-CTA-an-SM form: where the CTAs are no more than the SMs and each streams at least 12 stages.
// us, decode alone, pair / wide: 1 x 8 x 131072 tokens 65 / 59, x 65536 43 / 34, x 16384 24 / 18.7, 1 x 2 x
// 131072 52 / 27, 64 x 2 x 2048 20.7 / 18.9; shorter splits or more CTAs: 1 x 8 x 4096 11.5 / 13.2, 64 x 8 x 500 21 / 29, 32 x 8 x 4096 60 / 65.
constexpr int kWideStages = 12;

// Splits merge in clusters while they are short, the largest equal share of them whose clusters fit the device at once.
// Long splits (more than 40 stages) are bound by the stream, and a cluster's CTAs sit two on an SM where one each would
// stream faster: 131072 tokens x 8 heads in 18 splits 97 us apart, 111 us in clusters of 9; 4096 tokens in 16 splits 13.8 us
// in clusters of 16, 16.1 us apart.
constexpr int kClusterStages = 40;

// Quantised, (sequence, head) pairs just past one CTA an SM: most SMs hold one CTA, whose four compute warps take as long as the two
// that others hold (19 to 36 sequences x 8 heads x 4096 tokens are all 61 us).  In thirds they are two rounds of half-length clusters
// instead, while two rounds hold them; a cluster is the whole head, so nothing is left in the workspace and nobody counts arrivals.
// us, append + decode, whole / thirds: 19 x 8 x 8192 110.1 / 86.3, x 4096 61.1 / 54.1, x 2600 42.0 / 39.5, 20 x 8 x 4096 ragged 56.3 / 46.1,
// 22 x 8 x 6000 84.0 / 70.7, 38 x 4 x 3000 45.3 / 42.5, 75 x 2 x 30000 366 / 258; shorter: 19 x 8 x 2000 34.2 / 34.5.  Fifths of the first
// two: 87, 57.5.  The rounds (93 clusters of three each) may not be full: they start while the append still holds SMs, and what is placed late
// is a third round.  4096 tokens, 178 / 180 / 182 / 184 heads: 55.9 / 58.5 / 62.3 / 69.0 for 59.6 whole; hence a twentieth of slack.
// fits(wide, c): clusters of c CTAs of that form that the device holds at once.
template <typename Fits>
bool decode_thirds(const DecodeShape& d, Fits&& fits) {
    return d.mma && d.quant && !d.exchange && d.heads > d.sms && d.heads <= 2 * d.sms && d.heads <= d.counter_slots && d.stages >= 40 &&
           d.heads + d.heads / 20 <= 2 * fits(false, 3);
}

template <typename Fits>
int decode_splits(const DecodeShape& d, Fits&& fits) {
    // The generic kernel (128-thread CTAs, no shared-memory ring) wants several CTAs per SM to hide its loads and,
    // over a quantised cache, its dequantising arithmetic: aim at eight per SM.
    int s = d.mma ? d.sms / d.heads : (8 * d.sms + d.heads - 1) / d.heads;
    if (d.mma && !d.exchange) {
        // Two CTAs an SM (twice the bytes in flight, or twice the warps that dequantise) while the splits of a head are one
        // cluster: a power of two up to 16, which packs into the GPCs (16 sequences x 8 heads x 4096 tokens: 63 us unsplit, 51 us
        // in 2 splits; 4 x 8 x 2048: 15.0 us in 8 splits, 19.1 in 9).  Few heads: one CTA an SM over the bf16 cache (131072 tokens
        // x 8 heads, append + decode: 97 us with 18 splits, 97 with 36; decode alone 93 and 94) and over the quantised one where each
        // CTA then has 12 stages or more (kWideStages); below that two over the quantised one, in whole
        // clusters of 16 of at least 8 stages a split while splits are short enough to merge in clusters.
        // More (sequence, head) pairs than SMs: unsplit (us, unsplit / 2 splits, decode alone: 19 x 8 x 8192 tokens 114 / 142, 25 x 8 x
        // 4096 67 / 82, 32 x 8 x 4096 81 / 92, 37 x 8 x 2048 52 / 62; quantised, before its present form, 25 x 8 x 4096 66 / 73, 32 x 8 x 4096
        // 66 / 78; lengths from 4096 to 8192 24 x 8 106 / 114), but just past one CTA an SM over the quantised cache in three
        // (decode_thirds); two splits of ragged lengths over the bf16 cache (20 x 8, 4096 to 8192 tokens: 95 / 90) are not distinguished.
        const bool one = d.quant && d.heads <= d.sms && (long long)d.stages * d.heads >= (long long)kWideStages * d.sms;
        const int most = (one ? 1 : 2) * d.sms / d.heads, wide = (d.quant && !one ? 2 : 1) * d.sms / d.heads;
        if (d.heads > d.sms) s = decode_thirds(d, fits) ? 3 : 1;
        else if (most < 32) {
            s = 1;
            while (2 * s <= most) s *= 2;
            // Splits too long for clusters (kClusterStages) need no power of two: as many as there are SMs for.  us, append + decode over the
            // quantised cache, power of two / all: 10 heads, 8 / 14 splits of 41 stages 27.8 / 23.4, of 100 50.2 / 35.7, of 256 107 / 69; 40
            // heads, 2 / 3 splits 28.9 / 22.2, 51.4 / 39.6, 108 / 77.9; 24 heads, 4 / 6 29.3 / 26.7, 52.1 / 40.9; 16 heads, 8 / 9 29.5 / 28.7, 52.8 / 49.
            if ((s == 16 && d.stages > 32 * wide) || (one && d.stages > kClusterStages * s)) s = wide;
        } else {
            s = wide;
            if (d.stages <= 32 * s) {
                if (s > d.stages / 8) s = d.stages / 8;
                s = s < 32 ? 16 : s / 16 * 16;
            }
        }
    }
    if (s > d.stages / 2) s = d.stages / 2;          // every split keeps at least 2 stages
    if (s > kMaxFusedSplits) s = kMaxFusedSplits;
    return s < 1 ? 1 : s;
}

// The smallest count that decode_splits gives at this length or a longer one.  It falls only where the quantised cache goes over to
// one CTA an SM; before and after, it rises with the length.
template <typename Fits>
int decode_splits_at_longest(DecodeShape d, Fits&& fits) {
    const int here = decode_splits(d, fits);
    if (!d.mma || !d.quant || d.exchange || d.heads > d.sms) return here;
    const int turn = (kWideStages * d.sms + d.heads - 1) / d.heads;
    if (d.stages < turn) d.stages = turn;
    const int there = decode_splits(d, fits);
    return there < here ? there : here;
}

// asked: the caller's split count, or 0.  part_bytes: workspace bytes of one split; has, held: the caller's workspace.
template <typename Fits>
DecodePlan decode_plan(const DecodeShape& d, int asked, size_t part_bytes, bool has, size_t held, Fits&& fits) {
    DecodePlan p;
    p.n_splits = asked > 0 ? asked : decode_splits(d, fits);
    // A workspace sized at a longer max_seq_len: over the quantised cache fewer splits are chosen there than for some
    // shorter lengths.  Where it holds that choice but not this one, the call takes that one; where that choice is to write the
    // result directly, a call without a workspace does so (75 to 148 heads; it loses nothing, append + decode, unsplit / 2 splits: 16 x 8 x
    // 700 tokens 15.5 / 16.5 us, 20 x 5 x 700 13.8 / 14.0, 10 x 8 x 1000 15.7 / 17.8).  A workspace that holds not even one split is refused.
    if (asked <= 0 && (has ? held : 0) < p.n_splits * part_bytes) {
        const int fewer = decode_splits_at_longest(d, fits);
        if (has ? held >= fewer * part_bytes : fewer == 1 && !d.partial && !d.exchange) p.n_splits = fewer;
    }
    p.direct = p.n_splits == 1 && !d.partial && !d.exchange;
    // the tensor-core kernel merges its own splits when its counters can hold the heads
    p.fused = d.mma && !p.direct && p.n_splits <= kMaxFusedSplits && d.heads <= d.counter_slots;
    const int stages = (d.stages + p.n_splits - 1) / p.n_splits;          // of a split
    const long long ctas = (long long)d.heads * p.n_splits;
    p.wide = d.mma && d.quant && ctas <= d.sms && stages >= kWideStages;
    const bool thirds = p.fused && p.n_splits == 3 && decode_thirds(d, fits);
    if (thirds) p.cluster = 3;
    else if (p.fused && d.world <= 1 && stages <= kClusterStages)
        for (int c = kMaxCluster; c > 1 && p.cluster == 1; --c)
            if (p.n_splits % c == 0 && ctas / c <= fits(p.wide, c)) p.cluster = c;
    // Splits that merge through global memory, at most one CTA for every SM: two of them must not share an SM, which they do when
    // they are placed while the SMs still hold CTAs of the kernel before (a decode that merges, or the append).  So they ask for
    // more than half of an SM's shared memory.  Decode after decode / append + decode, us, 131072 tokens, bf16:
    //   8 heads, 144 CTAs: 102.5 / 97.2 where pairs could form, 93.2 / 97.1 now;  7 heads, 147 CTAs: 92.4 / 94.5 and 84.1 / 87.0;
    //   4 heads, 148 CTAs: 74.0 / 78.0 and 67.9 / 71.3.  A plain launch: 93.5 / 96.6, 84.4 / 87.3, 67.7 / 70.8 from a graph, but
    //   append + decode from a stream 99.4, 90.2 and 73.8 for 97.4, 87.2 and 71.6.
    p.alone = p.fused && p.cluster == 1 && ctas <= d.sms;
    // the kernel's own thirds merge inside clusters: they ask for the workspace of an unsplit launch, which they do not use
    p.parts = p.direct ? 0 : thirds && asked <= 0 ? (d.partial ? 1 : 0) : p.n_splits;
    return p;
}

}  // namespace grl
