// Launch-shape choices for B200 (148 SMs, 227 KB shared memory and 512 tensor-memory columns per
// SM, 64 K registers).  Stands in for the reference's get_*_config functions
// (csrc/jit_kernels/heuristics/common.hpp:8-398, sm90_arch.hpp:8-15), which pick tiles, stages
// and grids for H100.  Tile shapes are fixed by the kernels here (64-token chunks, 32-row state
// tiles); what remains to choose is how many CTAs share an SM and how large a persistent grid is.
#pragma once
#include <algorithm>
#include <cstdlib>
#include <limits>

namespace gdn {

struct RecurrentConfig {
    int stages;        // ring stages of 32 x DK state tiles
    int ctas_per_sm;   // limited by registers (128 threads x <=128 registers at DK <= 128)
    int smem_bytes;
    long long grid;    // persistent CTAs
};

// `ring`: the multi-token instance (two tile stages, the token ring, every tile a work unit);
// otherwise the decode instance (four tile stages).
inline RecurrentConfig recurrent_config(int dk, long long num_tiles, int sms, bool ring = false) {
    RecurrentConfig c;
    c.stages = ring ? 2 : 4;
    c.ctas_per_sm = ring ? (dk <= 64 ? 4 : (dk <= 256 ? 3 : 1)) : (dk <= 128 ? 4 : 2);
    const int tok_slot = 8 * (4 * dk + 64);  // k, q, v slice of 8 tokens (two ring slots; one more in every stage)
    const int stage = (32 * dk * 2 + (ring ? tok_slot : 4 * dk + 64) + 127) / 128 * 128;
    c.smem_bytes = c.stages * stage + 128 + (ring ? 2 * tok_slot : 0);
    c.grid = std::min<long long>(num_tiles, static_cast<long long>(sms) * c.ctas_per_sm);
    return c;
}

// Token-block kernel, head dims 192 and 256: groups of 16 state rows per CTA, 1 (two CTAs fit an SM) or 2 (one does; they share the
// preparation of the blocks).  A row's sums are the same in either.  A block of 16 tokens takes about 2.8 thousand cycles where a CTA
// with one group has the SM to itself, 4.3 where two share it, and 4.1 with two groups.  In us, one group : two: d=256, 8 v-heads, T=1500
// B=2 211 : 200, T=1000 B=4 283 : 270, B=3 (a last wave of few tiles) 229 : 270, T=500 B=8 (a last wave of half the tiles) 261 : 283; d=192
// T=700 B=2 91 : 84, B=4 144 : 163, B=6 178 : 164; 16 packed sequences of 500 510 : 501.  (At d=128, where two groups share less, one is as
// fast or faster: B=8 T=512, 8 v-heads 120 : 121, B=4, 32 v-heads 213 : 239, measured with a solve that took 350 cycles more.)
inline int block_groups(long long tiles, int sms) {
    const long long pairs = 2ll * sms, rest = tiles % pairs;
    const double one = 4.3 * static_cast<double>(tiles / pairs) + (rest == 0 ? 0.0 : rest <= sms ? 2.8 : 4.3);
    const double two = 4.1 * static_cast<double>((tiles + pairs - 1) / pairs);
    return two < one ? 2 : 1;
}

// One-token batches: the (sequence, v-head) units of `unit_tiles` tiles go round the `slots` CTAs; those of the last round, where it is not
// full, are cut into as many parts as leave no CTA with two of them.  (Cut finer than that, a part's own copies and norms cost more than
// the finer grain gives: every tile by itself, d=128, 32 v-heads, B=8 6.9 -> 7.6 us, B=24 13.2 -> 17.4.)  Whole : cut, us, 32 v-heads,
// d=128, the states in place B=1 5.3 : 3.5, B=5 6.0 : 5.0, B=8 7.0 : 5.5, B=19 11.9 : 10.7, B=24 12.6 : 12.3, B=27 14.0 : 13.8; in a pool B=24 13.2 : 12.6,
// B=40 18.3 : 17.8, B=56 22.9 : 22.2; fp32 B=5 7.6 : 6.3, B=14 14.7 : 12.8, B=28 23.7 : 22.5, B=46 35.5 : 34.9.  The instance that cuts is itself a
// little slower: bf16 in place it gains nothing from the third round on (B=64 25.1 : 25.6), the others from the fifth on (B=80 30.4 :
// 31.1); with two tiles per unit not from the second (d=64, B=24 6.43 : 6.46, B=46 10.3 : 10.5).
struct DecodeSplit {
    long long whole;  // units that stay whole
    int parts;        // 1: nothing is cut
};
// `later`: states in a pool or in fp32
inline DecodeSplit decode_split(long long num_tiles, int unit_tiles, long long slots, bool later) {
    const long long units = num_tiles / unit_tiles, rest = units % slots;
    DecodeSplit d{units - rest, 1};
    if (units / slots > (unit_tiles < 4 ? 0 : later ? 3 : 1)) return d;
    for (int f = 2; f <= unit_tiles && rest > 0 && rest * f <= slots; ++f)
        if (unit_tiles % f == 0) d.parts = f;
    return d;
}

struct PrefillConfig {
    int uw_ctas_per_sm;     // WY/UT kernel: 4 (52 KB shared memory, 128 tensor-memory columns, 128 registers)
    int fused_threads;      // state/output kernel: 16 warps, one CTA per SM (all 512 tensor-memory columns)
};

inline PrefillConfig prefill_config() { return PrefillConfig{4, 512}; }

// Segmented state propagation for few long sequences.  The state kernel is a serial chain
// per (sequence, v-head); with fewer chains than SMs most of the GPU idles.  The chain obeys
// S' = S M_c + N_c per chunk, so a sequence is cut into segments: one launch finds every
// segment's composite (M, N) (one CTA per chain and segment runs both), a small kernel chains them into the
// segments' start states, and a launch of the state kernel produces the output of all
// segments at once.  Two passes and a quarter instead of one, many segments wide.
// The plan must not depend on the device (the scratch size is computed without one), so it is
// made for the 148 SMs of a B200.  `max_units`: (slot, v-head) pairs whose segment states the scratch has room for; a plan
// with more is not made, the best one that fits is.
struct SegmentPlan {
    int num_segments;  // padded mode: segments per sequence; 1: not segmented
    int seg_chunks;    // chunks per segment
    int slots;         // (sequence, segment) pairs the launches cover: batch x num_segments in padded mode,
                       // an upper bound in packed mode (the lengths are only known on the device)
    int first_apart = 0;  // 1: the first segments are walked outright beside the transitions of the others (FusedParams::mode 1)
};
namespace plan_detail {
constexpr long long kSms = 148;
constexpr long long kNoLimit = std::numeric_limits<long long>::max();
// Cost model fitted to measurements (B=1..2, T=4096..131072, 4..32 v-heads), in units of "one
// chunk of the state kernel" (1.25 us): a CTA costs its chunks plus about 3 for start-up and pipeline
// fill, a chunk of the transition kernel 1.2 (1.5 us for both of its runs).  Every boundary between two segments of a chain
// costs kBoundary on top: its composite and start state move 0.4 MB, and it is one more product of a kernel that runs 9 chains
// at a time.  (Fitted when this plan decided for shorter sequences too, at 2 to 72 chains of 75 to 400 chunks.)  Plans whose launches need more
// than one wave measured worse than the model and are not made.  Sequences of up to kShortChunks chunks have the plan further down; for them
// this one only says from what scratch on a call is taken (gdn_prefill.cu, segment_plan_in).
constexpr int kFixed = 3;
constexpr double kPasses = 2.2, kBoundary = 0.15, kMargin = 0.85;
// Shortest segments, from measurements of 16 chains of 66 to 125 chunks, which the plan further down decides by now.  Above kShortChunks
// they bind little (padded: at most 32 segments, so only below 800 chunks).  Packed sequences of unequal lengths each end in a shorter
// one, hence the larger figure there.
constexpr int kMinSegment = 25, kMinSegmentPacked = 32;
inline long long waves(long long ctas) { return (ctas + kSms - 1) / kSms; }
}  // namespace plan_detail

inline SegmentPlan prefill_segments(long long chains, int chunks_per_seq, bool packed, long long max_units = plan_detail::kNoLimit) {
    using namespace plan_detail;
    SegmentPlan plan{1, chunks_per_seq, 0};
    if (packed || chains <= 0) return plan;
    double best = kMargin * static_cast<double>(waves(chains) * (chunks_per_seq + kFixed));
    for (int P = 2; P <= 32 && chunks_per_seq / P >= kMinSegment; ++P) {
        if (waves(chains * P) > 1 || chains * P > max_units) break;
        const int len = (chunks_per_seq + P - 1) / P;
        const double cost = kPasses * (len + kFixed) + kBoundary * static_cast<double>(chains * (P - 1));
        if (cost < best) {
            best = cost;
            plan.num_segments = P;
            plan.seg_chunks = len;
        }
    }
    return plan;
}

// Packed mode: the host sees the number of sequences and the total number of chunks, not the
// lengths.  Segments have one length L for all sequences; sequence s gets max(1, ceil(chunks_s / L))
// of them, at most total / L + num_seqs altogether: that many slots are launched and the surplus
// CTAs leave at once.  The unsegmented run is costed as if all sequences were equally long (its
// best case), so unequal lengths only make the segmented plan better than assumed.
constexpr int kMaxSegmentedSeqs = 64;
inline SegmentPlan prefill_segments_packed(int num_seqs, int num_v_heads, long long total_chunks,
                                           long long max_units = plan_detail::kNoLimit) {
    using namespace plan_detail;
    SegmentPlan plan{1, static_cast<int>(std::min<long long>(total_chunks, 1 << 30)), 0};
    if (num_seqs <= 0 || num_seqs > kMaxSegmentedSeqs || num_v_heads <= 0 || total_chunks <= 0 || total_chunks > (1 << 30)) return plan;
    const long long chains = static_cast<long long>(num_seqs) * num_v_heads;
    const long long even = (total_chunks + num_seqs - 1) / num_seqs;
    double best = kMargin * static_cast<double>(waves(chains) * (even + kFixed));
    for (int P = 2; P <= 128 && total_chunks / P >= kMinSegmentPacked; ++P) {
        const int len = static_cast<int>((total_chunks + P - 1) / P);
        const long long slots = total_chunks / len + num_seqs;  // launched (and given scratch): the upper bound
        // CTAs of surplus slots leave at once and free their SM, so the waves are counted for the slots that
        // hold work when the sequences are about equally long: every sequence end but the last may add one
        // short segment
        const long long work = (total_chunks + len - 1) / len + num_seqs - 1;
        if (waves(work * num_v_heads) > 1) break;
        if (slots * num_v_heads > max_units) continue;
        const double cost = kPasses * (len + kFixed) + kBoundary * static_cast<double>((work - num_seqs) * num_v_heads);
        if (cost < best) {
            best = cost;
            plan.num_segments = P;
            plan.seg_chunks = len;
            plan.slots = static_cast<int>(slots);
        }
    }
    return plan;
}

// Plan of sequences of up to kShortChunks chunks, of `chunks` chunks each (packed: on average, with `total` in all).  The first segments are walked
// outright beside the transitions of the others (FusedParams::mode 1), so P segments of c chains take c (P - 1) CTAs in either launch.
// In chunks of the state kernel, fitted to 60 shapes of 2 to 48 chains and 16 to 500 chunks with 3 to 36 segments (its choices are within 3 %
// of the best measured): both launches a chunk and more (what they read grows with the chains), one step of the start states for
// every segment from the third on, longer where many chains share their kernel, and 10.5 for four launches instead of one.  d=128, whole : so,
// us: 4 chains of 32 chunks 44.8 : 41.4, of 64 76.8 : 53.1, of 100 115 : 62.6, of 256 277 : 89.1; 16 of 64 88 : 75, of 256 322 : 170; 32 of 100 155 : 140,
// of 256 384 : 289; 48 of 256 433 : 376.  Against the plan above, whose segments have 25 chunks and more and whose first ones are found like the
// others: 1 sequence of 7919 tokens on 32 v-heads 177 : 161, 2 of 7344 on 8 125 : 101, 1 of 22109 on 4 121 : 103, packed 4 of 4000 on 4 165 : 82.
// 49 chains (7 sequences on 7 v-heads) stay whole: 172 chunks 339 us, cut so 355, 250 491 : 492, 625 1196 : 1144, in three by the plan above 350, 541, 1274.
// Longer sequences are bound by what the launches move, and a launch more costs them 1 % (4 chains of 1024 chunks in 32 segments 195 : 198): they
// keep the plans above.
constexpr int kShortChunks = 640, kManyChains = 48;
inline SegmentPlan prefill_segments_short(long long seqs, int num_v_heads, long long chunks, long long total, bool packed,
                                          long long max_units = plan_detail::kNoLimit) {
    using namespace plan_detail;
    SegmentPlan plan{1, static_cast<int>(chunks), packed ? 0 : static_cast<int>(seqs)};
    const long long chains = seqs * num_v_heads;
    if (chains <= 0 || chains > kManyChains) return plan;
    const double c = static_cast<double>(chains);
    double best = 0.985 * static_cast<double>(chunks + kFixed);
    for (int P = 3; P <= 64 && chunks / P >= 5; ++P) {
        const long long len = (chunks + P - 1) / P;
        // packed: every sequence end but the last may add a short segment; slots for any split of the chunks over the sequences are
        // launched and given scratch
        const long long work = packed ? (total + len - 1) / len + seqs - 1 : seqs * P, slots = packed ? total / len + seqs : seqs * P;
        if ((work - seqs) * num_v_heads > kSms) break;
        if (slots * num_v_heads > max_units) continue;
        const double cost = (2.0 + 0.01 * c) * static_cast<double>(len + kFixed) + (1.1 + 0.009 * c * c) * (P - 2) + 10.5;
        if (cost < best) {
            best = cost;
            plan.num_segments = P;
            plan.seg_chunks = static_cast<int>(len);
            plan.slots = static_cast<int>(slots);
            plan.first_apart = 1;
        }
    }
    return plan;
}

// Grid of the persistent WY/UT kernel: every CTA slot of the GPU, or one CTA per unit if fewer.
inline int uw_grid(long long units, int sms) {
    return static_cast<int>(std::min<long long>(units, static_cast<long long>(sms) * prefill_config().uw_ctas_per_sm));
}

// Grid of the persistent chunk-parallel kernel of the whole-layer path (units = chunks x k-heads,
// two CTAs of 256 threads per SM).
inline int zp_grid(long long units, int sms) {
    return static_cast<int>(std::min<long long>(units, static_cast<long long>(sms) * 2));
}

// Tokens per thread of the causal convolution.  A CTA streams a block of tokens; what counts is how long the fullest SM is
// busy.  Fitted to sweeps of the block (B x T from 100 to 32768 tokens, 2048 and 8192 channels): a CTA costs its tokens plus
// about 9 for its start (weights, the first loads, width - 1 tokens of halo), n CTAs side by side take n + 2 parts where
// one takes 3, and five fit.  With 32 tokens always, short inputs left most of the GPU idle and long ones its last wave.
inline int conv_tok_block(long long tokens, long long blocks_per_token_block, int sms) {
    constexpr int kStart = 9, kPerSm = 5;
    int best = 32;
    long long best_cost = -1;
    for (int t = 4; t <= 64; ++t) {
        const long long ctas = (tokens + t - 1) / t * blocks_per_token_block;
        const long long n = (ctas + sms - 1) / sms, rest = n % kPerSm;
        const long long cost = (n / kPerSm * (kPerSm + 2) + (rest ? rest + 2 : 0)) * (t + kStart);
        if (best_cost < 0 || cost <= best_cost) {
            best = t;
            best_cost = cost;
        }
    }
    return best;
}

}  // namespace gdn
