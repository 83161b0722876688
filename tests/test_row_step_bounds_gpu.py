"""Row steps of few screens on either side of the bounds between the one-launch step
and the tiled product, against the float64 recursion."""

import pytest

import test_row_step_gpu as steps

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,m,counts,anchored", [
    (40, 8, [2] * 5, False), (40, 8, [2] * 6, False),       # 45 and 54 staged rows
    (40, 7, [1] * 6, False), (520, 4, [1] * 11, False), (520, 4, [1] * 12, False),
    (33, 8, [2] * 8, True), (33, 8, [2] * 9, True),         # 72 and 81
    (40, 2, [3] * 16, False), (40, 4, [2] * 16, True)])
def test_either_side_of_the_bounds(W, m, counts, anchored):
    steps.test_rows_match_float64_recursion(W, m, counts, [0] * len(counts), anchored)
