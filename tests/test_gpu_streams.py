"""One connection used on two streams that do not wait for one another: the
first call on a stream finds nothing that another stream's queue still has to
write.  Streams are kept busy first, so that a call's device work runs long
after the host has queued the other stream's."""
import numpy as np
import pytest
import torch

from btorch_b200.models import SparseConn, _ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


def conn(seed, n=700, grad=False):
    rng = np.random.default_rng(seed)
    post, src = np.nonzero(rng.random((n, n)) < 0.05)
    w = (rng.integers(1, 9, post.size) * 2.0**-4).astype(np.float32)
    m = SparseConn.from_canonical(post, src, w, (n, n), enforce_dale=False, sparse_config={"direction": "scatter"}).to(DEV)
    m.magnitude.requires_grad_(grad)
    dense = np.zeros((n, n), np.float32)
    dense[src, post] = w
    return m, torch.tensor(dense, device=DEV)


def keep_busy(stream):
    with torch.cuda.stream(stream):
        a = torch.rand((4096, 4096), device=DEV)
        for _ in range(20):
            a = a @ a
            a = a / a.amax()


@pytest.mark.parametrize("seed", range(3))
def test_forward_on_two_streams(seed):
    m, dense = conn(seed)
    x = (torch.rand((16, 700), device=DEV) < 0.1).float()
    want = x @ dense  # dyadic weights, small counts: exact in any order
    torch.cuda.synchronize()
    first, second = torch.cuda.Stream(), torch.cuda.Stream()
    keep_busy(first)
    outs = []
    with torch.no_grad():
        for s in (first, second):
            with torch.cuda.stream(s):
                outs.append(m(x))
                outs.append(_ops.pack_edges(m.layout(DEV), m.magnitude.detach()))
    torch.cuda.synchronize()
    lay = m.layout(DEV)
    rec = outs[1].view(-1, 2)[: lay.nnz, 1]
    assert torch.equal(rec, m.magnitude.detach()[lay.csr_perm.long()].view(torch.int32))
    assert torch.equal(outs[0], want) and torch.equal(outs[2], want) and torch.equal(outs[1], outs[3])
