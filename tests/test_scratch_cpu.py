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


@pytest.mark.parametrize("n_in", [1, 70, 8192, 140000, 1 << 22])
@pytest.mark.parametrize("batch", [1, 3, 5, 128, 511, 4000, 10**5])
def test_forward_product_scratch(batch, n_in):
    """Two arrays of x's size up to 256 MB each, then no more than one of the whole batch (rows padded to 4)."""
    if batch * n_in >= 1 << 31:
        pytest.skip("refused by the product")
    words = L.lib().bt_spmv_push_work_words(batch, n_in, 0)
    assert words >= 8 + min(batch * n_in, 1 << 20)
    assert words <= 8 + 4 + max(2**27 + 8 * n_in, batch * n_in + 8 * n_in)
    if batch * n_in <= 2**26 and batch <= 2**22:  # one pass: every sample's list and transposed row
        assert words >= 8 + 2 * batch * n_in


def test_forward_product_scratch_holds_the_packed_weights():
    words = L.lib().bt_spmv_push_work_words
    assert words(1, 100, 10**6 + 4) >= 100 + 10**6 + 4
