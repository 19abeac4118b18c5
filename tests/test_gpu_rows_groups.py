"""The row engine where a transform's rows are split over four groups of warps: k_rows with two rows of five
layers of an axis of 302 points, with two rows of four and one row of five layers of an axis of 514 points
(there the last group has fewer rows than the others), and k_cols with sixteen columns.  Against the float64
oracle, at the bound of the engine's other tests (1e-5 after three steps)."""

import pytest

from test_gpu_rows import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nl,scheme,members", [
    (300, 299, 5, "ssprk3", 1), (512, 40, 4, "heun", 4), (512, 40, 5, "tsit5", 1), (380, 299, 5, "ssprk3", 1),
])
def test_four_row_groups(nx, ny, nl, scheme, members):
    check(nx, ny, nl, scheme, members)
