"""The rule that divides a launch of the fp16-operand GEMM, compiled for the host."""
import pytest

from launch_forms import B200_WIDTHS as B200, plans

SHAPES = [(n, t, (t + 3) // 4 + extra) for n in (2, 4, 6, 8, 12, 16, 32, 42, 64, 86) for t in (1, 7, 15, 16, 17, 33, 34, 74, 75, 148, 149, 300, 2000)
          for extra in (0, t // 2)]


def test_plans_cover_k_exactly():
    for (n, _, _), (pair, splits, chunks) in zip(SHAPES, plans(B200, SHAPES)):
        assert chunks % 2 == 0 and (splits - 1) * chunks < n <= splits * chunks
        assert not pair or splits == 1


def test_a_split_fits_the_clusters_the_device_runs():
    """A split takes one wave of clusters where a split with fewer parts would: 16 clusters of eight do not run at a time."""
    for (n, tiles, _), (pair, splits, _) in zip(SHAPES, plans(B200, SHAPES)):
        if not pair and splits > 1 and tiles <= B200[1]:
            assert tiles <= B200[splits - 1], (n, tiles, splits)


@pytest.mark.parametrize("widths,allowed", [
    ((9, 4, 2, 2, 1, 1, 1, 0, 4), {1, 2, 3, 4, 6}),  # nine SMs: no cluster of eight
    ((1, 0, 0, 0, 0, 0, 0, 0, 0), {1}),              # one SM
    ((148, 0, 0, 0, 0, 0, 0, 0, 0), {1}),            # a driver that does not answer
])
def test_forms_that_do_not_run_are_not_named(widths, allowed):
    for (n, _, _), (pair, splits, chunks) in zip(SHAPES, plans(widths, SHAPES)):
        assert splits in allowed and (splits > 1 or chunks == n) and (not pair or widths[-1] > 0)
