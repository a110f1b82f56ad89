"""The native BPTT chunk (engine forward + bt_bptt_backward) against the
single-step kernels on the same model: neuron counts and batches around the
vector width and the tile, LIF / ALIF, hard / soft reset, with and without
refractoriness, an input layer, state stacks, per-neuron parameters and
recomputed chunks.  Weights are dyadic, so both forwards give the same spikes
and states bit for bit; gradients are sums in another order of at most a few
hundred terms per step over 12 steps of a contracting recursion."""
import numpy as np
import pytest
import torch

from btorch_b200.models import ALIF, LIF, DenseConn, ExponentialPSC, RecurrentNN, Sigmoid, SparseConn, bptt, environ
from btorch_b200.models.functional import init_net_state

pytestmark = pytest.mark.gpu
DEV = "cuda"


def run(monkeypatch, native, n, B, kind, hard, ref, c_in, chunk, direction, stacks, per_neuron):
    rng = np.random.default_rng(n * 131 + B)
    dense = ((rng.random((n, n)) < min(0.5, 20 / n)) * rng.integers(1, 8, (n, n)) * 2.0**-6).astype(np.float32)
    dense[int(0.8 * n):] *= -1.0
    conn = SparseConn(dense, enforce_dale=False, sparse_config={"direction": direction})
    kw = dict(tau_ref=2.0 if ref else None, hard_reset=hard, surrogate_function=Sigmoid(alpha=2.0))
    if kind == "alif":
        neuron = ALIF(n, g_leak=0.05, E_leak=0.0, E_k=-1.0, tau_adapt=50.0, dg_k=0.0625, **kw)
    else:
        neuron = LIF(n, tau=torch.linspace(10.0, 30.0, n) if per_neuron else 20.0, **kw)
    inp = None
    if c_in:
        w_in = np.round(rng.normal(0, 0.3, (c_in, n)) * 64) / 64
        inp = DenseConn(c_in, n, weight=torch.tensor(w_in.astype(np.float32)),
                        bias=torch.full((n,), 0.125))
    net = RecurrentNN(neuron, ExponentialPSC(n, tau_syn=5.0, linear=conn), neuron_inp_module=inp,
                      update_state_names=("neuron.v", "synapse.psc") if stacks else (), grad_checkpoint=chunk > 0,
                      chunk_size=chunk or None, unroll=1).to(DEV)
    init_net_state(net, batch_size=B, dtype=torch.float32, device=DEV)
    x = torch.tensor((rng.random((12, B, c_in or n)) < 0.4).astype(np.float32), device=DEV)
    if not c_in:
        x = (x * 0.25).requires_grad_(True)
    if not native:
        monkeypatch.setattr(bptt, "native_steps", lambda *a: False)
    with environ.context(dt=1.0):
        z, st = net(x)
        assert net.last_path == "fused-bptt"
        probe = torch.linspace(0.5, 1.5, n, device=DEV)
        loss = (z * probe).sum() + net.neuron.v.square().sum() + (net.synapse.psc * probe).sum()
        if stacks:
            loss = loss + (st["neuron.v"] * probe).sum() + st["synapse.psc"].square().sum()
        loss.backward()
    monkeypatch.undo()
    out = {"z": z.detach(), "v": net.neuron.v.detach(), "psc": net.synapse.psc.detach(), "gw": conn.magnitude.grad}
    out.update({f"stack {k}": t.detach() for k, t in st.items()})
    if c_in:
        out["g_in"], out["g_b"] = inp.weight.grad, inp.bias.grad
    else:
        out["g_x"] = x.grad
    return out


@pytest.mark.parametrize("n,B", [(32, 4), (33, 3), (64, 1), (65, 33), (100, 5), (200, 40)])
@pytest.mark.parametrize("kind,hard,ref,c_in,chunk,direction,stacks,per_neuron", [
    ("lif", True, True, 7, 5, "scatter", False, False),
    ("lif", False, False, 0, 0, "scatter", True, True),
    ("alif", True, True, 0, 5, "scatter", True, False),
    ("alif", False, True, 7, 0, "gather", True, False),
    ("lif", True, False, 7, 5, "gather", False, True),
])
def test_native_equals_single_steps(monkeypatch, n, B, kind, hard, ref, c_in, chunk, direction, stacks, per_neuron):
    a, b = (run(monkeypatch, native, n, B, kind, hard, ref, c_in, chunk, direction, stacks, per_neuron)
            for native in (True, False))
    assert a["z"].sum() > 0
    for key in a:
        if key.startswith("g"):
            err = float((a[key] - b[key]).double().norm() / b[key].double().norm().clamp(min=1e-30))
            assert err < 1e-5, (key, err)
        else:
            assert torch.equal(a[key], b[key]), key


def test_given_spikes_drive_the_recurrence():
    """bt_engine_run_given: the published spikes are the given ones; the step's own only reset the neuron."""
    import scipy.sparse as sp

    from btorch_b200.models._ops import neuron_desc

    for n in (64, 33):  # the vectorised and the per-neuron step
        B, T = 3, 6
        g = torch.Generator(device=DEV).manual_seed(n)
        conn = SparseConn(sp.coo_array(np.eye(n, k=1, dtype=np.float32) * 0.5)).to(DEV)
        psc = ExponentialPSC(n, tau_syn=5.0, linear=conn).to(DEV)
        neuron = LIF(n, tau=20.0, hard_reset=True).to(DEV)
        d, keep = neuron_desc(neuron, 1.0)
        with environ.context(dt=1.0):
            coef, tau = psc.coefficients(1.0)
        zero = torch.zeros((B, n), device=DEV)
        eng = bptt._Run(neuron, d, psc, coef, tau, conn.layout(DEV), "scatter", conn.magnitude.detach(), B, n, zero, zero,
                        None, None)
        given = (torch.rand((T, B, n), generator=g, device=DEV) < 0.3).float()
        trace, own = torch.empty((T, B, n), device=DEV), torch.empty((T, B, n), device=DEV)
        from btorch_b200 import _lib as L

        eng.steps(torch.zeros((T, B, n), device=DEV), T, L.stream_of(trace.device), spikes=own, given=given, psc=trace)
        p = torch.zeros((B, n), device=DEV)
        for t in range(T):
            p = p + coef * (-p / tau)
            p[:, 1:] += 0.5 * given[t][:, :-1]
            torch.testing.assert_close(trace[t], p, rtol=2e-6, atol=1e-6)
