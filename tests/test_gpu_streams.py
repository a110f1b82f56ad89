"""One connection used on two streams that do not wait for one another: the
first call on a stream finds nothing that another stream's queue still has to
write.  Streams are kept busy first, so that a call's device work runs long
after the host has queued the other stream's."""
import numpy as np
import pytest
import torch

from btorch_b200 import _lib as L
from btorch_b200.models import LIF, ExponentialPSC, RecurrentNN, SparseConn, _ops, environ
from btorch_b200.models.autotune import EngineChoice
from btorch_b200.models.functional import init_net_state

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


@pytest.mark.parametrize("seed", range(3))
def test_backward_on_two_streams(seed):
    """The weights packed for the transposed gather by the first stream's backward."""
    m, dense = conn(seed, grad=True)
    x = [(torch.rand((16, 700), device=DEV) < 0.1).float().requires_grad_(True) for _ in range(2)]
    g = (torch.rand((16, 700), device=DEV) < 0.3).float()
    want = g @ dense.T
    torch.cuda.synchronize()
    first, second = torch.cuda.Stream(), torch.cuda.Stream()
    outs = []
    for xs, s in zip(x, (first, second)):
        with torch.cuda.stream(s):
            outs.append(m(xs))
    torch.cuda.synchronize()
    keep_busy(first)
    grads = []
    for xs, out, s in zip(x, outs, (first, second)):
        with torch.cuda.stream(s):
            grads += torch.autograd.grad(out, xs, g)
    torch.cuda.synchronize()
    assert torch.equal(grads[0], want) and torch.equal(grads[1], want)


def net(n, batch, tau=20.0, **cfg):
    rng = np.random.default_rng(n)
    mask = rng.random((n, n)) < 0.05
    w = np.where(mask, rng.integers(1, 5, (n, n)) * 2.0**-6, 0.0).astype(np.float32)
    rnn = RecurrentNN(LIF(n, tau=tau, tau_ref=2.0, hard_reset=True),
                      ExponentialPSC(n, 5.0, SparseConn(w, sparse_config=cfg)), update_state_names=("neuron.v",)).to(DEV)
    init_net_state(rnn, batch_size=batch, dtype=torch.float32, device=DEV)
    return rnn


@pytest.mark.parametrize("mode", ["cluster", "tile", "scatter"])
def test_runs_on_two_streams(mode):
    """Packed in-edges, tile offsets and per-neuron parameters that are converted for the kernels."""
    n, T = 640, 20
    choice = {"cluster": EngineChoice(L.BT_MODE_CLUSTER), "tile": EngineChoice(L.BT_MODE_TILE),
              "scatter": EngineChoice(L.BT_MODE_SCATTER, scatter_lanes=32, neuron_spt=1)}[mode]
    x = (torch.rand((T, 1, n), device=DEV) < 0.4).float() * 4.0

    def make():
        return net(n, 1, tau=torch.linspace(10.0, 30.0, n, dtype=torch.float64), direction="auto", tile=True)

    with torch.no_grad(), environ.context(dt=1.0):
        want, _ = make()(x, engine_choice=choice)
        assert want.sum() > 0
        rnn = make()
        v = rnn.neuron.v.clone()
        torch.cuda.synchronize()
        first, second = torch.cuda.Stream(), torch.cuda.Stream()
        keep_busy(first)
        got = []
        rnn.engine_status_check = "deferred"
        for s in (first, second):
            with torch.cuda.stream(s):
                # the state is this stream's own
                rnn.neuron.v, rnn.neuron.refractory = v.clone(), torch.zeros_like(v)
                rnn.synapse.psc = torch.zeros_like(v)
                got.append(rnn(x, engine_choice=choice)[0])
        torch.cuda.synchronize()
    assert torch.equal(got[0], want) and torch.equal(got[1], want)


def test_a_copied_connection_starts_without_kept_arrays():
    import copy

    m, dense = conn(5, grad=True)
    x = (torch.rand((16, 700), device=DEV) < 0.1).float().requires_grad_(True)
    g = torch.ones((16, 700), device=DEV)
    torch.autograd.grad(m(x), x, g)  # keeps the packed weights
    twin = copy.deepcopy(m)
    with torch.no_grad():
        twin.magnitude.mul_(2.0)
    assert torch.equal(torch.autograd.grad(twin(x), x, g)[0], 2.0 * (g @ dense.T))
    assert torch.equal(torch.autograd.grad(m(x), x, g)[0], g @ dense.T)
    rnn = net(640, 1, direction="auto")
    z = torch.ones((3, 1, 640), device=DEV) * 3.0
    with torch.no_grad(), environ.context(dt=1.0):
        rnn(z, engine_choice=EngineChoice(L.BT_MODE_CLUSTER))
    assert copy.deepcopy(rnn.synapse.linear)._cluster_packed is None
