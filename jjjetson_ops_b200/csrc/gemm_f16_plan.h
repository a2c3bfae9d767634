// How the fp16-operand GEMM divides a launch: single CTAs, clusters whose CTAs split K, or pairs of CTAs.  Plain C++, so that the
// rule can be tested without a GPU.
#pragma once

#include <cstdint>

namespace jq {

constexpr int HF_MAX_SPLITS = 8;  // CTAs per tile along K: the largest portable cluster

// What the device runs at a time, as the driver says (0: this form does not run there): clusters of `i` CTAs that split K (1: single
// CTAs), and pairs of CTAs.  Clusters do not fill the SMs: a B200 (148 SMs) holds 74 of two CTAs, 45 of three, 33, 22 and 15 of
// four, six and eight.
struct GemmF16Widths {
    int splits[HF_MAX_SPLITS + 1];
    int pairs;
};

struct GemmF16Plan {
    bool pair;                 // pairs of CTAs share 256 x 256
    int k_splits;              // otherwise CTAs per 128 x 128 tile, of
    int chunks_per_split;      // this many 128-value chunks of K each (the last: what is left)
};

// The cheapest form by what a launch takes, in hundredths of a us: per wave of CTAs a fixed part and 68 for each 128-value stage
// (79 where pairs of CTAs share 256 x 256: they convert as much per stage as single CTAs and multiply twice as much).  The fixed
// part fills the pipeline and writes the tile, and adds up the parts where K is split.  A fit over 110 shapes (K 256 to 11008, N 64
// to 32000, M 64 to 2048, the multiply alone, every form): the form it names takes 0.3 % more than the quickest one on average.  Against 116
// shapes in a chain of launches, of the form it names: pairs 6 % off on average and 12 % at most (K = 8192, N = 28672, M = 2048 is 760 by
// the estimate and takes 860 to 890, at the card's power limit), the others 11 %, mostly launches of a few us that take 1 to 1.5 less.  Both sides of the lines, the multiply alone, us:
//   K = N = 4096, M = 512 (128 tiles): one 26.2, pairs 31.1 (64 on 74 places)
//   K = N = 4096, M = 128 (32 tiles): four parts 12.4, three 15.5, six 21.2, because 32 clusters of six take two waves
//   K = 8192, N = 1101, M = 167: six parts 15.6, eight 24.6
//   K = 2304, N = 24089, M = 1386: pairs 192, one 251
inline GemmF16Plan plan_gemm_f16(int n_chunks, int64_t tiles, int64_t pair_tiles, const GemmF16Widths &width) {
    constexpr int64_t STAGE = 68, PAIR_STAGE = 79, PAIR_WAVE = 800, PAIR_ONCE = -126;
    constexpr int64_t WAVE[HF_MAX_SPLITS + 1] = {0, 429, 834, 741, 668, 0, 718, 0, 805};  // by CTAs per tile; 0: not used
    GemmF16Plan plan{false, 1, n_chunks};
    int64_t best = -1;
    for (int s = 1; s <= HF_MAX_SPLITS; ++s) {
        const int chunks = ((n_chunks + s - 1) / s + 1) / 2 * 2;  // whole pairs of chunks: a weight copy brings two
        if (WAVE[s] == 0 || width.splits[s] <= 0 || (n_chunks + chunks - 1) / chunks != s) continue;
        const int64_t cost = (tiles + width.splits[s] - 1) / width.splits[s] * (chunks * STAGE + WAVE[s]);
        if (best < 0 || cost < best) {
            best = cost;
            plan.k_splits = s;
            plan.chunks_per_split = chunks;
        }
    }
    if (width.pairs > 0) {
        const int64_t cost = (pair_tiles + width.pairs - 1) / width.pairs * (n_chunks * PAIR_STAGE + PAIR_WAVE) + PAIR_ONCE;
        if (best < 0 || cost < best) plan = {true, 1, n_chunks};
    }
    return plan;
}

}  // namespace jq
