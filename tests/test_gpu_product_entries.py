"""The C entries of the sparse product that the modules no longer call themselves
(the push, the lane-split and the transposed input gradient, the masked weight
gradient), for callers of the library, against the float64 product: odd batches, one sample, mask words
and their edges, empty rows and columns, silent and always-active sources."""
import numpy as np
import pytest
import torch

from btorch_b200 import _lib as L
from btorch_b200.models import SparseConn
from btorch_b200.models._ops import pack_csr_weights

pytestmark = pytest.mark.gpu
DEV = "cuda"


def problem(n_in, n_out, batch, activity):
    rng = np.random.default_rng(n_in * 7 + batch)
    mask = rng.random((n_out, n_in)) < min(0.5, 20 / n_in)
    mask[::5] = False  # posts without in-edges
    mask[:, ::7] = False  # sources without out-edges
    post, src = np.nonzero(mask)
    w = rng.standard_normal(post.size).astype(np.float32)
    m = SparseConn.from_canonical(post, src, w, (n_in, n_out), enforce_dale=False).to(DEV)
    x = (rng.standard_normal((batch, n_in)) * (rng.random((batch, n_in)) < activity)).astype(np.float32)
    x[:, n_in // 2] = 0.0
    x[:, n_in // 3] = 1.0
    g = rng.standard_normal((batch, n_out)).astype(np.float32)
    dense = np.zeros((n_in, n_out))
    dense[src, post] = w
    return m.layout(DEV), m.magnitude.detach(), x, g, dense, post, src


def stream():
    return L.stream_of(torch.device(DEV))


SHAPES = [(1, 5, 1), (300, 77, 3), (70, 900, 33), (1100, 1500, 64), (129, 40, 131)]


@pytest.mark.parametrize("n_in,n_out,batch", SHAPES)
@pytest.mark.parametrize("activity", [0.0, 0.05, 1.0])
def test_scatter_entry(n_in, n_out, batch, activity):
    lay, w, x, _, dense, post, _ = problem(n_in, n_out, batch, activity)
    out = torch.full((batch, n_out), 7.0, device=DEV)
    work = torch.empty(batch * n_in + 2, device=DEV, dtype=torch.int32)
    packed, xd = pack_csr_weights(lay, w), torch.tensor(x, device=DEV)
    L.check(L.lib().bt_spmv_scatter(batch, n_in, n_out, lay.csr_ptr.data_ptr(), lay.csr_dst.data_ptr(), packed.data_ptr(),
                                    xd.data_ptr(), out.data_ptr(), work.data_ptr(), stream()), "bt_spmv_scatter")
    x64 = x.astype(np.float64)
    # a sum of t terms in any order is within t * 2^-24 of the sum of magnitudes (first order)
    terms = np.bincount(post, minlength=n_out) + 8
    assert (np.abs(out.cpu().numpy() - x64 @ dense) <= terms * 2.0**-24 * (np.abs(x64) @ np.abs(dense))).all()


@pytest.mark.parametrize("n_in,n_out,batch", SHAPES)
@pytest.mark.parametrize("activity", [0.0, 0.05, 1.0])
def test_weight_gradient_entry(n_in, n_out, batch, activity):
    lay, _, x, g, _, post, src = problem(n_in, n_out, batch, activity)
    gw = torch.full((max(1, lay.nnz),), 7.0, device=DEV)
    masks = torch.empty(n_in * ((batch + 31) // 32), device=DEV, dtype=torch.int32)
    xd, gd = torch.tensor(x, device=DEV), torch.tensor(g, device=DEV)
    L.check(L.lib().bt_spmv_grad_weight(batch, n_in, n_out, lay.csc_ptr.data_ptr(), lay.csc_src.data_ptr(), xd.data_ptr(),
                                        gd.data_ptr(), gw.data_ptr(), masks.data_ptr(), stream()), "bt_spmv_grad_weight")
    x64, g64 = x.astype(np.float64), g.astype(np.float64)
    want, size = (x64.T @ g64)[src, post], (np.abs(x64).T @ np.abs(g64))[src, post]
    got = gw[: lay.nnz].cpu().numpy()
    assert (np.abs(got - want) <= (batch + 2) * 2.0**-24 * size).all()
    assert (got[size == 0.0] == 0.0).all()  # silent sources: exact zeros


@pytest.mark.parametrize("n_in,n_out,batch", SHAPES)
@pytest.mark.parametrize("entry", ["bt_spmv_grad_input", "bt_spmv_grad_input_t", "bt_spmv_grad_input_pad"])
def test_input_gradient_entries(entry, n_in, n_out, batch):
    lay, w, _, g, dense, _, src = problem(n_in, n_out, batch, 1.0)
    gx = torch.full((batch, n_in), 7.0, device=DEV)
    packed, gd = pack_csr_weights(lay, w), torch.tensor(g, device=DEV)
    args = [batch, n_in, n_out, lay.csr_ptr.data_ptr(), lay.csr_dst.data_ptr(), packed.data_ptr(), gd.data_ptr(),
            gx.data_ptr()]
    if entry != "bt_spmv_grad_input":
        work = torch.empty((batch + 3) // 4 * 4 * n_out, device=DEV)
        args.append(work.data_ptr())
    L.check(getattr(L.lib(), entry)(*args, stream()), entry)
    g64 = g.astype(np.float64)
    terms = np.bincount(src, minlength=n_in) + 8
    assert (np.abs(gx.cpu().numpy() - g64 @ dense.T) <= terms * 2.0**-24 * (np.abs(g64) @ np.abs(dense.T))).all()
