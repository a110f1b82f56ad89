"""State and input arrays that do not start on 16 bytes, for neuron counts that
are a multiple of 4: the engine and the BPTT chunk take their word-wise kernels and
give the same results, and the tuner tries their samples per thread."""
import numpy as np
import pytest
import torch

from btorch_b200 import _lib as L
from btorch_b200.models import ALIF, LIF, ExponentialPSC, RecurrentNN, Sigmoid, SparseConn, autotune, environ
from btorch_b200.models.autotune import EngineChoice
from btorch_b200.models.engine import match
from btorch_b200.models.functional import init_net_state

pytestmark = pytest.mark.gpu
DEV = "cuda"


def shifted(t):
    """The same values one word past a 16-byte boundary."""
    buf = torch.empty(t.numel() + 4, device=DEV, dtype=t.dtype)
    at = 1 + (-buf.data_ptr() // 4) % 4
    out = buf[at: at + t.numel()].view(t.shape)
    out.copy_(t)
    assert out.data_ptr() % 16 == 4 and out.is_contiguous()
    return out


def net(n, batch, alif, shift, direction="scatter", **kw):
    rng = np.random.default_rng(n)
    w = np.where(rng.random((n, n)) < 0.2, rng.integers(1, 5, (n, n)) * 2.0**-6, 0.0).astype(np.float32)
    neuron = ALIF(n, g_leak=0.05, E_leak=0.0, E_k=-1.0, dg_k=0.0625, tau_adapt=200.0, tau_ref=2.0, hard_reset=True,
                  surrogate_function=Sigmoid(alpha=2.0)) if alif else \
        LIF(n, tau_ref=2.0, hard_reset=True, surrogate_function=Sigmoid(alpha=2.0))
    rnn = RecurrentNN(neuron, ExponentialPSC(n, 5.0, SparseConn(w, sparse_config={"direction": direction, **kw})),
                      update_state_names=("neuron.v", "synapse.psc")).to(DEV)
    init_net_state(rnn, batch_size=batch, dtype=torch.float32, device=DEV)
    if shift:
        neuron.v, neuron.refractory, rnn.synapse.psc = map(shifted, (neuron.v, neuron.refractory, rnn.synapse.psc))
        if alif:
            neuron.g_k = shifted(neuron.g_k)
    return rnn


@pytest.mark.parametrize("n,batch", [(4, 1), (64, 3), (516, 33)])
@pytest.mark.parametrize("alif", [False, True])
@pytest.mark.parametrize("spt", [1, 4])
def test_engine_on_unaligned_arrays(n, batch, alif, spt):
    x = (torch.rand((20, batch, n), device=DEV) < 0.4).float() * 2.0
    outs = []
    for shift in (False, True):
        rnn = net(n, batch, alif, shift)
        xs = shifted(x) if shift else x
        with torch.no_grad(), environ.context(dt=1.0):
            z, st = rnn(xs, engine_choice=EngineChoice(L.BT_MODE_SCATTER, scatter_lanes=32, neuron_spt=spt))
        outs.append([z, st["neuron.v"], st["synapse.psc"], rnn.neuron.v, rnn.synapse.psc])
    assert outs[0][0].sum() > 0
    for a, b in zip(*outs):
        assert torch.equal(a, b)


@pytest.mark.parametrize("n,batch", [(4, 1), (64, 5), (100, 33)])
@pytest.mark.parametrize("alif,direction", [(False, "scatter"), (True, "gather")])
def test_bptt_chunk_on_unaligned_arrays(n, batch, alif, direction):
    """The backward of a chunk reads the input in place: with x one word off, its word-wise kernel runs."""
    outs = []
    for shift in (False, True):
        rnn = net(n, batch, alif, shift, direction)
        gen = torch.Generator(device=DEV).manual_seed(1)
        x = (torch.rand((10, batch, n), generator=gen, device=DEV) < 0.5).float() * 0.75
        x = (shifted(x) if shift else x).requires_grad_(True)
        with environ.context(dt=1.0):
            z, st = rnn(x)
            assert rnn.last_path == "fused-bptt"
            (z.sum() + st["neuron.v"].square().sum()).backward()
        outs.append([z.detach(), st["neuron.v"].detach(), x.grad, rnn.synapse.linear.magnitude.grad])
    assert outs[0][0].sum() > 0
    for a, b in zip(outs[0][:2], outs[1][:2]):
        assert torch.equal(a, b)
    for a, b in zip(outs[0][2:], outs[1][2:]):  # the same sums in the same order
        assert float((a - b).norm()) <= 1e-6 * float(a.norm())


def test_tuner_tries_samples_per_thread_on_unaligned_state():
    x = torch.zeros((4, 8, 64), device=DEV)
    for shift, want in ((False, {1}), (True, {1, 2, 4})):
        rnn = net(64, 8, False, shift)
        plan, _ = match(rnn)
        assert autotune.aligned(plan, rnn, x) is not shift
        got = autotune.candidates(plan.conn, 8, 1, 1, 64, torch.device(DEV), autotune.aligned(plan, rnn, x))
        assert {c.neuron_spt for c in got if c.mode == L.BT_MODE_SCATTER} == want
    assert not autotune.aligned(match(net(64, 8, False, False))[0], rnn, shifted(x))
    rnn.cudagraph = True
    assert autotune.aligned(match(rnn)[0], rnn, shifted(x))


def test_tuning_on_unaligned_state_tries_them():
    rnn = net(64, 8, False, True, autotune=True)
    x = (torch.rand((max(autotune.TUNE_MIN_STEPS, autotune.TRIAL_WARM + autotune.TRIAL_STEPS), 8, 64), device=DEV) < 0.4).float()
    with torch.no_grad(), environ.context(dt=1.0):
        rnn(x)
    (_, timings), = autotune.tuned(rnn).values()
    assert {c.neuron_spt for c in timings} == {1, 2, 4}
