"""The weight gradient over row lists (bt_spmv_grad_weight_rows) at its edges:
row counts around a mask word, a list vector and a row segment, posts around a
CTA, silent and always-active sources, graded values, dense inputs, and the
accumulating call."""
import numpy as np
import pytest
import torch

from btorch_b200 import _lib as L
from btorch_b200.models import SparseConn

pytestmark = pytest.mark.gpu
DEV = "cuda"


def grad_weight(lay, x, g, n_in, dense, into=None):
    rows = x.shape[0]
    gw = torch.full((lay.nnz,), 3.0, device=DEV) if into is None else into
    work = torch.empty(L.lib().bt_grad_weight_work_words(rows, n_in, dense), device=DEV, dtype=torch.int32)
    L.check(L.lib().bt_spmv_grad_weight_rows(rows, n_in, lay.n_out, lay.csc_ptr.data_ptr(), lay.csc_src.data_ptr(),
                                             x.data_ptr(), g.data_ptr(), gw.data_ptr(), int(into is not None), dense,
                                             work.data_ptr(), L.stream_of(torch.device(DEV))),
            "bt_spmv_grad_weight_rows")
    return gw


@pytest.mark.parametrize("rows", [1, 6, 7, 8, 15, 16, 31, 33, 64, 130, 4096, 4097, 8200])
@pytest.mark.parametrize("kind", ["spikes", "graded", "dense"])
@pytest.mark.parametrize("n_out,n_in", [(1, 70), (8, 70), (61, 70), (19, 900)])
def test_grad_weight_rows(rows, kind, n_out, n_in):
    rng = np.random.default_rng(rows * 7 + n_out)
    mask = rng.random((n_out, n_in)) < 0.4
    post, src = np.nonzero(mask)
    m = SparseConn.from_canonical(post, src, np.ones(post.size, np.float32), (n_in, n_out), enforce_dale=False).to(DEV)
    lay = m.layout(DEV)
    x = (rng.random((rows, n_in)) < 0.05).astype(np.float32)
    x[:, 3], x[:, 4] = 1.0, 0.0
    if kind != "spikes":
        x *= rng.standard_normal((rows, n_in)).astype(np.float32)
    if kind == "dense":
        x = rng.standard_normal((rows, n_in)).astype(np.float32)
    g = rng.standard_normal((rows, n_out)).astype(np.float32)
    xd, gd = torch.tensor(x, device=DEV), torch.tensor(g, device=DEV)
    x64, g64 = x.astype(np.float64), g.astype(np.float64)
    want = (x64.T @ g64)[src, post]
    size = (np.abs(x64).T @ np.abs(g64))[src, post]
    # a sum of t terms in any order is within t * 2^-24 of the sum of magnitudes (first order); t <= rows
    terms = (x != 0).sum(0)[src] + 2
    for dense in (0, 1):
        got = grad_weight(lay, xd, gd, n_in, dense)
        assert (np.abs(got.cpu().numpy() - want) <= terms * 2.0**-24 * size).all()
        again = grad_weight(lay, xd, gd, n_in, dense, into=got.clone()).cpu().numpy()
        assert (np.abs(again - 2 * want) <= (2 * terms + 1) * 2.0**-24 * 2 * size).all()
        torch.testing.assert_close(grad_weight(lay, xd, gd, n_in, dense), got, rtol=0, atol=0)


def test_grad_weight_rows_skips_zero_inputs():
    """A zero input adds nothing, whatever the gradient of its row; no rows give zeros."""
    n = 40
    post, src = np.nonzero(np.ones((n, n)))
    m = SparseConn.from_canonical(post, src, np.ones(post.size, np.float32), (n, n), enforce_dale=False).to(DEV)
    lay = m.layout(DEV)
    for fill in (0.05, 0.9):
        x = (torch.rand((20, n), device=DEV) < fill).float() * 2.0
        x[5] = 0.0
        g = torch.ones((20, n), device=DEV)
        g[5] = float("inf")
        for dense in (0, 1):
            got = grad_weight(lay, x, g, n, dense)
            want = 2.0 * (x != 0).sum(0).float()[torch.tensor(src, device=DEV)]
            torch.testing.assert_close(got, want, rtol=0, atol=0)
    empty = torch.empty((0, n), device=DEV)
    assert (grad_weight(lay, empty, empty, n, 1) == 0).all()
