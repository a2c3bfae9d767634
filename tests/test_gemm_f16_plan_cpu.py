"""The rule that divides a launch of the fp16-operand GEMM, compiled for the host."""
import os
import subprocess

import pytest

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
B200 = (148, 74, 45, 33, 26, 22, 15, 15, 74)


@pytest.fixture(scope="module")
def plans(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("plan") / "plan")
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", os.path.join(ROOT, "jjjetson_ops_b200", "csrc"), "-x", "c++", "-", "-o", exe],
                   input=SOURCE, text=True, check=True)

    def run(widths, shapes):
        text = "".join("%s %d %d %d\n" % (" ".join(map(str, widths)), *s) for s in shapes)
        r = subprocess.run([exe], input=text, capture_output=True, text=True, check=True)
        return [tuple(map(int, line.split())) for line in r.stdout.splitlines()]

    return run


SHAPES = [(n, t, (t + 3) // 4 + extra) for n in (2, 4, 6, 8, 12, 16, 32, 42, 64, 86) for t in (1, 7, 15, 16, 17, 33, 34, 74, 75, 148, 149, 300, 2000)
          for extra in (0, t // 2)]


def test_plans_cover_k_exactly(plans):
    for (n, _, _), (pair, splits, chunks) in zip(SHAPES, plans(B200, SHAPES)):
        assert chunks % 2 == 0 and (splits - 1) * chunks < n <= splits * chunks
        assert not pair or splits == 1


def test_a_split_fits_the_clusters_the_device_runs(plans):
    """A split takes one wave of clusters where a split with fewer parts would: 16 clusters of eight do not run at a time."""
    for (n, tiles, _), (pair, splits, _) in zip(SHAPES, plans(B200, SHAPES)):
        if not pair and splits > 1 and tiles <= B200[1]:
            assert tiles <= B200[splits - 1], (n, tiles, splits)


@pytest.mark.parametrize("widths,allowed", [
    ((9, 4, 2, 2, 1, 1, 1, 0, 4), {1, 2, 3, 4, 6}),  # nine SMs: no cluster of eight
    ((1, 0, 0, 0, 0, 0, 0, 0, 0), {1}),              # one SM
    ((148, 0, 0, 0, 0, 0, 0, 0, 0), {1}),            # a driver that does not answer
])
def test_forms_that_do_not_run_are_not_named(plans, widths, allowed):
    for (n, _, _), (pair, splits, chunks) in zip(SHAPES, plans(widths, SHAPES)):
        assert splits in allowed and (splits > 1 or chunks == n) and (not pair or widths[-1] > 0)
