"""Which form of a kernel a shape is given: the GEMM's own rule compiled for the host, and the small-batch kernel's restated.  Tests
that are there for a form say which one they mean, so that a change of a rule cannot quietly take their coverage away."""
import functools
import os
import subprocess
import tempfile

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = """
#include <cstdio>
#include "gemm_f16_plan.h"
int main() {
    jq::GemmF16Widths w{};
    int n_chunks;
    long long tiles, pair_tiles;
    // widths of 1 to 8 CTAs per tile and of pairs, then the shape
    for (;;) {
        for (int s = 1; s <= jq::HF_MAX_SPLITS; ++s)
            if (std::scanf("%d", &w.splits[s]) != 1) return 0;
        if (std::scanf("%d %d %lld %lld", &w.pairs, &n_chunks, &tiles, &pair_tiles) != 4) return 1;
        const jq::GemmF16Plan p = jq::plan_gemm_f16(n_chunks, tiles, pair_tiles, w);
        std::printf("%d %d %d\\n", (int)p.pair, p.k_splits, p.chunks_per_split);
    }
}
"""
B200_SMS = 148
B200_WIDTHS = (148, 74, 45, 33, 26, 22, 15, 15, 74)  # what the occupancy query answers: clusters of 1 to 8 CTAs, pairs


@functools.lru_cache(maxsize=None)
def _plan_program():
    exe = os.path.join(tempfile.mkdtemp(prefix="jq_plan_"), "plan")
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", os.path.join(ROOT, "jjjetson_ops_b200", "csrc"), "-x", "c++", "-", "-o", exe],
                   input=SOURCE, text=True, check=True)
    return exe


def plans(widths, shapes):
    """(pair, k_splits, chunks_per_split) for each (chunks of 128, tiles, 256 x 256 tiles)."""
    text = "".join("%s %d %d %d\n" % (" ".join(map(str, widths)), *s) for s in shapes)
    r = subprocess.run([_plan_program()], input=text, capture_output=True, text=True, check=True)
    return [tuple(map(int, line.split())) for line in r.stdout.splitlines()]


def gemm_f16_form(K, rows, M):
    """"pair" or the number of parts of K, for weight matrices of these rows on a B200."""
    tiles = sum(-(-n // 128) for n in rows) * -(-M // 128)
    pair_tiles = sum(-(-n // 256) for n in rows) * -(-M // 256)
    pair, parts, _ = plans(B200_WIDTHS, [(K // 128, tiles, pair_tiles)])[0]
    return "pair" if pair else parts


def small_batch_form(K, rows, M):
    """How K is shared out on a B200, which fixes the order of the additions: (odd K, column tiles of a group of at most 32, rows and
    whether the CTA is alone on its SM, for CTAs of 32 or 64 rows): 64 rows are four warps along K, 32 are eight, alone sixteen."""
    odd = K // 128 % 2 != 0
    groups = -(-M // 32)
    ct = -(-(-(-M // groups)) // 8)
    wide = sum(-(-n // 64) for n in rows) * groups
    wr = 2 if not (odd and K > 2048) and ct >= 3 and wide >= B200_SMS else 1
    return odd, ct, 32 * wr, wr == 1 and sum(-(-n // 32) for n in rows) * groups <= B200_SMS


def small_batch_tile(K, rows, M):
    """(rows, column tiles, consumer warps, CTAs per SM) of a launch on a B200, as launch_mmq_stream chooses them."""
    odd, ct, narrow_rows, alone = small_batch_form(K, rows, M)
    groups = -(-M // 32)
    tiles = {r: sum(-(-n // r) for n in rows) for r in (32, 64, 96, 128)}
    if alone:
        return 32, ct, 16, 1
    along_k = 4 if narrow_rows == 64 else 8
    one_wave = next((r for r in (64, 96, 128) if tiles[r] * groups <= B200_SMS and r * along_k <= 768), None)
    if odd or (along_k == 4 and one_wave == 64):
        return narrow_rows, ct, 8, 2
    if one_wave and (along_k == 4 or one_wave != 64 or K >= 4096 or (ct < 4 and tiles[32] * groups > 1.1 * B200_SMS)):
        return one_wave, ct, one_wave // 32 * along_k, 1
    if along_k == 4 and groups == 2:
        for r, most in ((96, 8), (128, 6)):
            if tiles[r] <= B200_SMS:
                return (r, -(-M // 8), r // 8, 1) if -(-M // 8) <= most else (64, ct, 8, 2)
    return narrow_rows, ct, 8, 3 if along_k == 8 and tiles[32] * groups > 4 * B200_SMS else 2
