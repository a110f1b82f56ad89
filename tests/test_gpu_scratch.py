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
