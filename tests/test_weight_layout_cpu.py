"""A connection's weights with strides of their own (a magnitude bound to a view):
the product's launches get them as one run, with the gradient through the copy."""
import numpy as np
import pytest
import torch

from btorch_b200 import _lib as L
from btorch_b200.models import SparseConn, _ops


@pytest.mark.parametrize("kind", ["strided", "expanded", "plain"])
@pytest.mark.parametrize("direction", ["gather", "scatter"])
def test_products_get_contiguous_weights(monkeypatch, kind, direction):
    rng = np.random.default_rng(0)
    post, src = np.nonzero(rng.random((9, 13)) < 0.4)
    m = SparseConn.from_canonical(post, src, np.ones(post.size, np.float32), (13, 9), enforce_dale=False)
    base = torch.arange(1.0, 2 * post.size + 1)
    w = {"strided": base[::2], "expanded": base[:1].expand(post.size), "plain": base[: post.size].clone()}[kind]
    m.magnitude = torch.nn.Parameter(w)
    seen = []

    def product(direction, layout, x, w_canon, w_csr):
        seen.append(w_canon)
        return torch.zeros(x.shape[0], layout.n_out)

    monkeypatch.setattr(_ops, "_spmv", product)
    monkeypatch.setattr(L, "require_cuda", lambda *a, **k: None)
    x = torch.ones(2, 13)
    with torch.no_grad():
        _ops.sparse_mm(x, m.magnitude, m.layout("cpu"), direction)
    _ops.sparse_mm(x, m.magnitude, m.layout("cpu"), direction)
    for got in seen:
        assert got.is_contiguous() and torch.equal(got, w)
    if kind == "plain":
        assert all(got.data_ptr() == m.magnitude.data_ptr() for got in seen)
