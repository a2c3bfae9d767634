// How the fp16-operand GEMM divides a launch: single CTAs, clusters whose CTAs split K, or pairs of CTAs.  Plain C++, so that the
// rule can be tested without a GPU.
#pragma once

#include <cstdint>

namespace jq {

constexpr int HF_MAX_SPLITS = 8;  // CTAs per tile along K: the largest portable cluster
constexpr int HF_MAX_NARROW_SPLITS = HF_MAX_SPLITS / 2;  // pairs per tile along K

// What the device runs at a time, as the driver says (0: this form does not run there): clusters of `i` CTAs that split K (1: single
// CTAs), and pairs of CTAs.  Clusters do not fill the SMs: a B200 (148 SMs) holds 74 of two CTAs, 45 of three, 33, 22 and 15 of
// four, six and eight.
struct GemmF16Widths {
    int splits[HF_MAX_SPLITS + 1];
    int pairs;
    int narrow[HF_MAX_NARROW_SPLITS + 1];
};

struct GemmF16Plan {
    bool pair;                 // pairs of CTAs share 256 x 256
    bool narrow;
    int k_splits;              // otherwise CTAs per 128 x 128 tile, of
    int chunks_per_split;      // this many 128-value chunks of K each (the last: what is left)
};

// The cheapest form by what a launch takes, in hundredths of a us: per wave of CTAs a fixed part and 74 for each 128-value stage
// (101 where pairs of CTAs share 256 x 256: they convert as much per stage as single CTAs and multiply twice as much).  The fixed
// part fills the pipeline and writes the tile, and adds up the parts where K is split.  A fit over 1677 shapes (K 256 to 11008, N 64
// to 32000, M 64 to 2048, whole linears, every form): within 3 % on average, and the form it names takes 0.05 % more than the
// quickest one on average, 6 % at most (K = 1536, N = 3072, M = 384: two parts 15.8, one 14.9 us).  Both sides of the lines, whole linear, us:
//   K = 2048, 16 tiles (N = 2048, M = 128): one 17.2, two 15.0, four 11.3; eight 20.0, because 16 clusters take two waves
//   K = 11008, 16 tiles: six 22.8, eight 36.2; K = 4096, 15 tiles or less: eight
//   K = 1024, N = 2048, M = 512 (64 tiles): one 11.8, two 14.1
//   K = 256, N = 32000, M = 300: single CTAs 32.1, pairs 35.5 (multiply alone)
// `n_chunks` is K / 128 (even), `tiles` the 128 x 128 tiles of all matrices, `pair_tiles` the 256 x 256 ones.
inline GemmF16Plan plan_gemm_f16(int n_chunks, int64_t tiles, int64_t pair_tiles, const GemmF16Widths &width,
                                 int64_t narrow_tiles = 0) {
    (void)narrow_tiles;
    constexpr int64_t STAGE = 74, PAIR_STAGE = 101, PAIR_WAVE = 780, PAIR_ONCE = -200;
    constexpr int64_t WAVE[HF_MAX_SPLITS + 1] = {0, 420, 860, 730, 710, 0, 740, 0, 880};  // by CTAs per tile; 0: not used
    GemmF16Plan plan{false, false, 1, n_chunks};
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
        if (best < 0 || cost < best) plan = {true, false, 1, n_chunks};
    }
    return plan;
}

}  // namespace jq
