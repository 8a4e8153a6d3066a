"""The rule that sizes the boxes of node moments around the particles."""
import pytest
import torch

from funlbm_b200.lbm import LBMD3


def _sphere(r, n):
    g = torch.Generator().manual_seed(1)
    v = torch.randn(n, 3, generator=g, dtype=torch.float64)
    return r * v / v.norm(dim=1, keepdim=True)


@pytest.mark.parametrize("r,markers,count,used", [
    (6, 11776, 32, True),        # many small bodies
    (40, 20106, 1, True),
    (40, 5000, 1, False),        # markers far apart: fewer slots than nodes
    (60, 47000, 11, False),      # small bodies beside a large one
    (130, 1 << 20, 1, False),    # a box of more than 2^24 nodes
])
def test_box_cells(r, markers, count, used):
    cells = LBMD3._box_cells(_sphere(r, markers), count)
    assert (cells > 0) == used
    if used:                     # holds the body with two nodes on either side and rounding
        assert cells >= (2 * r + 5) ** 3


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), float("-inf")])
def test_box_cells_of_markers_that_are_not_finite(bad):
    lag = _sphere(6, 11776)
    lag[77, 1] = bad
    assert LBMD3._box_cells(lag, 32) == 0
