"""Device memory of SparseConn calls over many samples: scratch stays bounded."""
import numpy as np
import pytest
import torch

from btorch_b200.models import SparseConn

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("rows", [4096, 4097, 20000])
def test_module_backward_scratch(rows):
    """SparseConn over [T, B, n]: the weight gradient of many rows, right, and its scratch below half of x beyond
    one pass (the lists of 4096 rows; with the transposed copy, one and a half times x within it)."""
    n = 512
    rng = np.random.default_rng(rows)
    post, src = np.nonzero(rng.random((n, n)) < 0.02)
    m = SparseConn.from_canonical(post, src, np.ones(post.size, np.float32), (n, n), enforce_dale=False).to(DEV)
    x = (torch.rand((rows, n), device=DEV) < 0.02).float()
    g = (torch.rand((rows, n), device=DEV) < 0.1).float()
    out = m(x)
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    base = torch.cuda.memory_allocated()
    out.backward(g)
    peak = torch.cuda.max_memory_allocated() - base
    want = (x.double().T @ g.double())[torch.tensor(src, device=DEV), torch.tensor(post, device=DEV)]
    assert torch.equal(m.magnitude.grad.double(), want)  # counts: exact
    assert peak <= (1.6 if rows <= 4096 else 0.6) * 4096 * n * 4 + 4 * 2**20


@pytest.mark.parametrize("activity", [0.01, 0.5])  # pushed, gathered
@pytest.mark.parametrize("packed", [False, True])
def test_forward_in_passes(activity, packed):
    """More samples than one pass takes: equal to the same samples a few at a time (dyadic weights, exact in any
    order), and scratch of no more than x's own size."""
    n_in, n_out, batch = 70000, 64, 2001
    rng = np.random.default_rng(3)
    key = np.unique(rng.integers(0, n_in * n_out, 30000))
    post, src = key // n_in, key % n_in
    w = (rng.integers(1, 9, key.size) * 2.0**-4).astype(np.float32)
    m = SparseConn.from_canonical(post, src, w, (n_in, n_out), enforce_dale=False,
                                  sparse_config={"direction": "scatter"}).to(DEV)
    x = torch.rand((batch, n_in), device=DEV)
    x = x.lt_(activity)
    with torch.no_grad():
        if packed:
            m.prepare_sparse()
        want = torch.cat([m(x[b:b + 200]) for b in range(0, batch, 200)])
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        base = torch.cuda.memory_allocated()
        got = m(x)
        peak = torch.cuda.max_memory_allocated() - base
    assert torch.equal(got, want)
    assert want.sum() > 0 and peak <= 1.05 * x.numel() * 4
