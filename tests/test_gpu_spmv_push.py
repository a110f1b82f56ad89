"""The device-chosen forward product (bt_spmv_push) on both of its paths and
around its edges: batches around the vector width, compaction blocks, empty
rows, packed and unpacked weights, zero inputs against infinite weights."""
import numpy as np
import pytest
import torch

from btorch_b200.models import SparseConn
from btorch_b200.models import _ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("n_in,n_out", [(1, 40), (300, 77), (70, 900), (1100, 1500)])
@pytest.mark.parametrize("batch", [1, 3, 4, 9, 33, 128, 131])
@pytest.mark.parametrize("activity", [0.0, 0.01, 0.045, 0.3, 1.0])
def test_push_both_paths(n_in, n_out, batch, activity):
    rng = np.random.default_rng(n_in * 3 + batch)
    mask = rng.random((n_out, n_in)) < min(0.6, 30 / n_in)
    mask[:: 5] = False
    post, src = np.nonzero(mask)
    w = rng.standard_normal(post.size).astype(np.float32)
    m = SparseConn.from_canonical(post, src, w, (n_in, n_out), enforce_dale=False).to(DEV)
    lay = m.layout(DEV)
    x = (rng.standard_normal((batch, n_in)) * (rng.random((batch, n_in)) < activity)).astype(np.float32)
    xd, wd = torch.tensor(x, device=DEV), m.magnitude.detach()
    dense = np.zeros((n_in, n_out))
    dense[src, post] = w
    want, size = x.astype(np.float64) @ dense, np.abs(x.astype(np.float64)) @ np.abs(dense)
    # any order of a sum of t terms is within t * 2^-24 of the sum of magnitudes (first order)
    bound = (mask.sum(1).max() + 8) * 2.0**-24 * size
    for packed in (None, _ops.pack_csr_weights(lay, wd)):
        got = _ops._spmv("scatter", lay, xd, wd, packed).cpu().numpy()
        assert (np.abs(got - want) <= bound).all()


def test_push_skips_zero_inputs():
    """A zero input adds nothing, whatever the weight, on either path."""
    n = 64
    post, src = np.nonzero(np.ones((n, n)))
    w = np.ones(post.size, np.float32)
    w[src == 5] = np.inf
    m = SparseConn.from_canonical(post, src, w, (n, n), enforce_dale=False).to(DEV)
    for fill in (0.02, 0.8):
        x = (torch.rand((40, n), device=DEV) < fill).float()
        x[:, 5] = 0.0
        got = _ops._spmv("scatter", m.layout(DEV), x, m.magnitude.detach(), None)
        torch.testing.assert_close(got, x.sum(1, keepdim=True).expand(-1, n), rtol=0, atol=0)


@pytest.mark.parametrize("batch", [1, 5, 300])
@pytest.mark.parametrize("n_out", [40, 9500])
def test_ordered_gather_samples_over_the_grid(batch, n_out):
    """Every (sample, output) is the ascending fmaf chain whatever the grid: equal to one sample at a time."""
    rng = np.random.default_rng(batch)
    post, src = np.nonzero(rng.random((n_out, 30)) < 0.3)
    w = rng.standard_normal(post.size).astype(np.float32)
    m = SparseConn.from_canonical(post, src, w, (30, n_out), enforce_dale=False).to(DEV)
    x = torch.tensor((rng.standard_normal((batch, 30)) * (rng.random((batch, 30)) < 0.5)).astype(np.float32), device=DEV)
    lay, wd = m.layout(DEV), m.magnitude.detach()
    whole = _ops._spmv("gather", lay, x, wd, None)
    rows = torch.cat([_ops._spmv("gather", lay, x[b:b + 1].contiguous(), wd, None) for b in range(batch)])
    assert torch.equal(whole, rows)


@pytest.mark.parametrize("activity", [0.02, 1.0])
def test_push_batches_beyond_the_grid(activity):
    """More samples than sample blocks fit the grid's y: dyadic weights, exact in any order."""
    batch, n_in, n_out = (1 << 23) + 5, 3, 2
    m = SparseConn.from_canonical(np.array([0, 0, 1, 1]), np.array([0, 2, 1, 2]),
                                  np.array([0.5, -2.0, 1.0, 0.25], np.float32), (n_in, n_out), enforce_dale=False).to(DEV)
    x = (torch.rand((batch, n_in), device=DEV) < activity).float()
    got = _ops._spmv("scatter", m.layout(DEV), x, m.magnitude.detach(), None)
    dense = torch.tensor([[0.5, 0.0], [0.0, 1.0], [-2.0, 0.25]], device=DEV)
    want = x[:, :1] * dense[0] + x[:, 1:2] * dense[1] + x[:, 2:] * dense[2]
    assert torch.equal(got, want)
