"""Products and gradients of a connection whose magnitude is a strided or expanded view."""
import numpy as np
import pytest
import torch

from btorch_b200.models import SparseConn

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("kind", ["strided", "expanded"])
@pytest.mark.parametrize("direction", ["gather", "scatter"])
@pytest.mark.parametrize("activity", [0.02, 0.8])
def test_views_as_weights(kind, direction, activity):
    rng = np.random.default_rng(1)
    n = 150
    post, src = np.nonzero(rng.random((n, n)) < 0.2)
    m = SparseConn.from_canonical(post, src, np.ones(post.size, np.float32), (n, n), enforce_dale=False,
                                  sparse_config={"direction": direction}).to(DEV)
    base = torch.tensor(rng.integers(1, 9, 2 * post.size) * 2.0**-3, dtype=torch.float32, device=DEV)
    w = base[::2] if kind == "strided" else base[:1].expand(post.size)
    m.magnitude = torch.nn.Parameter(w)
    dense = torch.zeros((n, n), device=DEV)
    dense[src, post] = w
    x = (torch.rand((40, n), device=DEV) < activity).float().requires_grad_(True)
    g = (torch.rand((40, n), device=DEV) < 0.5).float()
    out = m(x)
    gx, gw = torch.autograd.grad(out, (x, m.magnitude), g)
    assert torch.equal(out, x.detach() @ dense) and torch.equal(gx, g @ dense.T)  # dyadic: exact in any order
    assert torch.equal(gw, (x.detach().T @ g)[src, post])
    with torch.no_grad():
        assert torch.equal(m(x), x @ dense)
