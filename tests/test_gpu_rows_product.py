"""The backward's product through the transposed gradient (bt_spmv_grad_input_pad)
at its edges: batches around the vector width and the sample block, row counts
around the warps-per-row rule, empty rows and rows longer than a warp."""
import numpy as np
import pytest
import torch

from btorch_b200 import _lib as L
from btorch_b200.models import SparseConn
from btorch_b200.models._ops import pack_csr_weights

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("rows", [33, 1600, 3100, 6100])
@pytest.mark.parametrize("batch", [1, 2, 3, 4, 5, 17, 31, 64, 127, 130])
def test_grad_input_padded(rows, batch):
    rng = np.random.default_rng(rows + batch)
    n_out = 75
    deg = rng.integers(0, 3, rows)
    deg[::7] = 0
    deg[5] = 70  # more than two warps' edges
    src = np.repeat(np.arange(rows), deg)
    post = np.concatenate([rng.choice(n_out, d, replace=False) for d in deg if d]).astype(np.int64)
    order = np.lexsort((src, post))
    post, src = post[order], src[order]
    w = rng.standard_normal(src.size).astype(np.float32)
    m = SparseConn.from_canonical(post, src, w, (rows, n_out), enforce_dale=False).to(DEV)
    lay = m.layout(DEV)
    w_csr = pack_csr_weights(lay, m.magnitude.detach())
    g = torch.tensor(rng.standard_normal((batch, n_out)).astype(np.float32), device=DEV)
    work = torch.empty((batch + 3) // 4 * 4 * n_out, device=DEV)
    outs = []
    for _ in range(2):
        gx = torch.full((batch, rows), 7.0, device=DEV)
        L.check(L.lib().bt_spmv_grad_input_pad(batch, rows, n_out, lay.csr_ptr.data_ptr(), lay.csr_dst.data_ptr(),
                                               w_csr.data_ptr(), g.data_ptr(), gx.data_ptr(), work.data_ptr(),
                                               L.stream_of(torch.device(DEV))), "bt_spmv_grad_input_pad")
        outs.append(gx.cpu().numpy())
    np.testing.assert_array_equal(outs[0], outs[1])
    dense = np.zeros((rows, n_out))
    dense[src, post] = w
    g64 = g.cpu().numpy().astype(np.float64)
    # any order of a sum of d terms is within d * 2^-24 of the sum of magnitudes (first order); 80 >= d + 8
    bound = 80 * 2.0**-24 * (np.abs(g64) @ np.abs(dense).T) + 1e-30
    assert (np.abs(outs[0] - g64 @ dense.T) <= bound).all()
