"""Scratch that the products ask for, by the library's own size functions: no
more than the path that runs can use, and bounded for batches of any length."""
import pytest

from btorch_b200 import _lib as L

LIST_ROWS = 4096  # rows of one pass of the weight gradient over row lists


@pytest.mark.parametrize("n_in", [1, 70, 8192])
@pytest.mark.parametrize("rows", [0, 1, 128, LIST_ROWS - 1, LIST_ROWS])
def test_weight_gradient_reserves_the_transpose_that_it_uses(rows, n_in):
    words = L.lib().bt_grad_weight_work_words
    assert words(rows, n_in, 1) - words(rows, n_in, 0) == n_in * (-(-rows // 4) * 4)


@pytest.mark.parametrize("n_in", [1, 70, 8192])
@pytest.mark.parametrize("rows", [LIST_ROWS + 1, 10**5, 10**6])
def test_weight_gradient_of_long_batches_reserves_no_transpose(rows, n_in):
    words = L.lib().bt_grad_weight_work_words
    assert words(rows, n_in, 1) == words(rows, n_in, 0) == words(LIST_ROWS, n_in, 0)
