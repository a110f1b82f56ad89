"""What a user of this package runs, as measurable cases.

Every case is one call (or one short sequence of calls) through the public
modules: a closed-loop single step, the sparse connection alone (forward, and
forward + backward), whole simulations of the kinds the benchmark and the
tests build (a small network alone, a batch with ragged durations and a dense
input layer, a delayed connectome, receptor channels, a small network with
every state traced), truncated-BPTT training windows, a served mix of
requests and the raster export.

listed() gives the fixed cases, draw(rng) another one of the same ranges,
prepare(case, seed) the state a program holds before the call, run(state) one
pass, work(case) the bytes and operations the pass cannot do without, and
exact(case, seed) the outputs in 64 bits where they have such a value.

Recurrent weights of whole simulations lie on a dyadic grid (as the benchmark's
connectome and training networks do), so that spike rasters do not depend on
the order of a sum.
"""

import numpy as np
import torch

from btorch_b200.io import raster_to_sparse_repr
from btorch_b200.models import (ALIF, LIF, DelayedPSC, DenseConn, ExponentialPSC, HeterSynapsePSC, RecurrentNN,
                                Sigmoid, SparseConn, environ)
from btorch_b200.models.functional import init_net_state, reset_net
from btorch_b200.serving import NetworkPool, SimRequest, SimulationServer


def listed():
    return [
        # closed-loop stepping: one module-by-module step per call of the plain network, an environment in
        # between; the smallest call there is
        dict(name="cell_step", kind="cell", neuron="lif", n=4096, indeg=82, batch=1),
        # a graded (rate) signal through the connection alone, inference
        dict(name="conn_graded", kind="conn", n=8192, indeg=160, batch=32, activity=1.0, grad=False),
        # spikes through the connection alone with both gradients: a module-by-module training step
        dict(name="conn_spikes_grad", kind="conn", n=8192, indeg=410, batch=128, activity=0.02, grad=True),
        # the plain forward simulation: one network, one sample, 1000 channels, 1000 steps
        dict(name="sim_plain", kind="sim", neuron="lif", n=4096, indeg=82, batch=1, steps=1000, c_in=1000),
        # a small odd-sized network with a synaptic delay, default outputs: dense spikes and every state traced
        dict(name="sim_traces", kind="traces", n=1000, indeg=50, batch=3, steps=300, delay=3),
        # batched simulation: adaptive neurons, dense input layer, ragged durations, captured chunks
        dict(name="sim_batched", kind="sim", neuron="alif", n=32768, indeg=250, batch=64, steps=400, c_in=2000),
        # connectome-shaped: lognormal in-degree, per-synapse delays, background drive on every neuron
        dict(name="sim_connectome", kind="connectome", n=140000, indeg=128, batch=8, steps=504, receptors=1),
        # the same with four E/I receptor channels
        dict(name="sim_receptors", kind="connectome", n=16384, indeg=200, batch=8, steps=300, receptors=4),
        # one truncated-BPTT window of the training network, chunks of 20 recomputed in backward
        dict(name="train_window", kind="train", neuron="lif", n=8192, indeg=410, batch=128, steps=100, c_in=256,
             chunk=20),
        # a small adaptive network trained with every step's buffers kept
        dict(name="train_small", kind="train", neuron="alif", n=2000, indeg=100, batch=16, steps=50, c_in=100,
             chunk=0),
        # a mix of requests served by continuous batching on one network
        dict(name="serve_mix", kind="serve", n=16384, indeg=128, slots=8, requests=16, steps=500, c_in=500),
        # export of a spike raster as sparse coordinates
        dict(name="raster_export", kind="raster", n=20000, batch=4, steps=1000, activity=0.01),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["cell", "conn", "conn", "sim", "sim", "traces", "connectome", "connectome", "train", "train",
                       "serve", "raster"])
    if kind == "cell":
        n = _log(rng, 256, 8192)
        return dict(kind=kind, neuron=rng.choice(["lif", "alif"]), n=n, indeg=_log(rng, 8, min(200, n // 4)),
                    batch=_log(rng, 1, 32))
    if kind == "conn":
        n = _log(rng, 512, 8192)
        return dict(kind=kind, n=n, indeg=_log(rng, 16, min(410, n // 4)), batch=_log(rng, 1, 128),
                    activity=rng.choice([0.01, 0.02, 0.1, 1.0]), grad=rng.random() < 0.5)
    if kind == "sim":
        if rng.random() < 0.5:
            n = _log(rng, 512, 4096)
            return dict(kind=kind, neuron="lif", n=n, indeg=_log(rng, 16, 82), batch=rng.choice([1, 1, 2, 4]),
                        steps=_log(rng, 100, 1000), c_in=_log(rng, 50, 1000))
        n = _log(rng, 2048, 32768)
        return dict(kind=kind, neuron="alif", n=n, indeg=_log(rng, 50, 250), batch=_log(rng, 16, 64),
                    steps=_log(rng, 100, 400), c_in=_log(rng, 200, 2000))
    if kind == "traces":
        n = _log(rng, 200, 3000)
        return dict(kind=kind, n=n, indeg=_log(rng, 10, 50), batch=_log(rng, 1, 8), steps=_log(rng, 50, 300),
                    delay=rng.randint(1, 6))
    if kind == "connectome":
        c = rng.choice([1, 1, 2, 3, 4])
        n = _log(rng, 4096, 140000 if c == 1 else 16384)
        return dict(kind=kind, n=n, indeg=_log(rng, 50, 128 if c == 1 else 200), batch=_log(rng, 1, 8),
                    steps=_log(rng, 100, 500), receptors=c)
    if kind == "train":
        n = _log(rng, 512, 8192)
        steps = _log(rng, 20, 100)
        return dict(kind=kind, neuron=rng.choice(["lif", "lif", "alif"]), n=n, indeg=_log(rng, 20, min(410, n // 8)),
                    batch=_log(rng, 4, 128), steps=steps, c_in=_log(rng, 20, 256), chunk=rng.choice([0, 10, 20]))
    if kind == "serve":
        return dict(kind=kind, n=_log(rng, 4096, 16384), indeg=_log(rng, 50, 128), slots=rng.choice([4, 8, 16]),
                    requests=_log(rng, 4, 16), steps=_log(rng, 150, 500), c_in=_log(rng, 100, 500))
    return dict(kind=kind, n=_log(rng, 1000, 20000), batch=_log(rng, 1, 8), steps=_log(rng, 100, 1000),
                activity=rng.choice([0.002, 0.01, 0.05]))


# ------------------------------------------------------------------ inputs --

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(7919 * int(seed) + 13)


def _edges(n, indeg, ragged=False):
    """Random connections in canonical (post, pre) order, on the device: a fixed in-degree (pairs drawn twice count
    once), or a lognormal one (sigma 1) of that mean.  Which pairs are connected goes by the sizes; weights and
    everything else by the seed."""
    g = _gen(1000003 * n + indeg)
    if ragged:
        k = torch.empty(n, device="cuda").log_normal_(float(np.log(indeg) - 0.5), 1.0, generator=g)
        k = k.round().clamp(1, n - 1).long()
    else:
        k = torch.full((n,), indeg, device="cuda", dtype=torch.long)
    post = torch.repeat_interleave(torch.arange(n, device="cuda"), k)
    pre = torch.randint(0, n, (post.numel(),), generator=g, device="cuda")
    key = torch.unique(post * n + pre)
    return key // n, key % n


def _counts(g, m):
    """Synapse counts: geometric, mean 4."""
    u = torch.rand(m, generator=g, device="cuda").clamp_(min=1e-7)
    return (torch.log(u) / float(np.log(0.75))).floor_() + 1.0


def _conn(post, src, w, shape, **kwargs):
    return SparseConn.from_canonical(post.cpu().numpy(), src.cpu().numpy(), w.cpu().numpy(), shape,
                                     enforce_dale=False, **kwargs)


def _dyadic_weights(g, pre, n, exc, inh, exc_frac=0.8):
    c = _counts(g, pre.numel())
    return c * torch.where(pre < int(exc_frac * n), exc, -inh)


def _neuron(case, **kwargs):
    n = case["n"]
    if case["neuron"] == "alif":
        return ALIF(n, v_threshold=1.0, v_reset=0.0, c_m=1.0, g_leak=0.05, E_leak=0.0, E_k=-1.0, tau_adapt=200.0,
                    dg_k=0.07, tau_ref=2.0, hard_reset=True, **kwargs)
    return LIF(n, v_threshold=1.0, v_reset=0.0, tau=20.0, tau_ref=2.0, hard_reset=True, **kwargs)


def _dense(g, c_in, n, std):
    return DenseConn(c_in, n, weight=torch.randn((c_in, n), generator=g, device="cuda").mul_(std).cpu())


def _prepare_cell(case, seed):
    g = _gen(seed)
    n, B = case["n"], case["batch"]
    post, pre = _edges(n, case["indeg"])
    w = torch.randn(pre.numel(), generator=g, device="cuda") * 0.1
    conn = _conn(post, pre, w, (n, n))
    net = RecurrentNN(_neuron(case), ExponentialPSC(n, tau_syn=5.0, linear=conn)).to("cuda")
    init_net_state(net, batch_size=B, dtype=torch.float32, device="cuda")
    # a network in operation: membranes anywhere below threshold, a tenth of the neurons refractory
    state = {"v": torch.rand((B, n), generator=g, device="cuda"),
             "refractory": (torch.rand((B, n), generator=g, device="cuda") < 0.1).float(),
             "psc": torch.randn((B, n), generator=g, device="cuda") * 0.1}
    if case["neuron"] == "alif":
        state["g_k"] = torch.rand((B, n), generator=g, device="cuda") * 0.3
    x = torch.randn((B, n), generator=g, device="cuda") * 0.1 + 0.1
    return {"net": net, "state": state, "x": x, "edges": (post, pre, w)}


def _run_cell(s):
    net, st = s["net"], s["state"]
    net.neuron.v, net.neuron.refractory, net.synapse.psc = st["v"], st["refractory"], st["psc"]
    if "g_k" in st:
        net.neuron.g_k = st["g_k"]
    with torch.no_grad(), environ.context(dt=1.0):
        z, states = net.single_step_forward(s["x"])
    return {"z": z, "states": states}


def _exact_cell(case, s):
    post, pre, w = s["edges"]
    d = lambda t: t.double()  # noqa: E731
    st = {k: d(v) for k, v in s["state"].items()}
    v, ref, psc = st["v"], st["refractory"], st["psc"]
    current = psc + d(s["x"])
    out = {}
    if case["neuron"] == "alif":
        gk = st["g_k"]
        lin = (-0.05 - gk) / 1.0
        v1 = v + torch.expm1(lin) / lin * (-0.05 * v - gk * (v + 1.0) + current)
        rate = -1.0 / 200.0
        gk = gk + float(np.expm1(rate) / rate) * (-gk / 200.0)
    else:
        v1 = v + (-v / 20.0 + current)
    z = (v1 >= 1.0).double() * (ref == 0).double()
    out["neuron.v"] = v1 - v1 * z
    out["neuron.refractory"] = (ref + 2.0 * z - 1.0).clamp(min=0.0)
    if case["neuron"] == "alif":
        out["neuron.g_k"] = gk + 0.07 * z
    rate = -1.0 / 5.0
    wz = torch.zeros_like(psc).index_add_(1, post, z[:, pre] * d(w))
    out["synapse.psc"] = psc + float(np.expm1(rate) / rate) * (-psc / 5.0) + wz
    return {"z": z, "states": out}


def _prepare_conn(case, seed):
    g = _gen(seed)
    n, B = case["n"], case["batch"]
    post, pre = _edges(n, case["indeg"])
    w = torch.randn(pre.numel(), generator=g, device="cuda") * 0.1
    conn = _conn(post, pre, w, (n, n)).to("cuda")
    if case["activity"] >= 1.0:
        x = torch.randn((B, n), generator=g, device="cuda")
    else:
        x = (torch.rand((B, n), generator=g, device="cuda") < case["activity"]).float()
    grad = torch.randn((B, n), generator=g, device="cuda") if case["grad"] else None
    return {"conn": conn, "x": x, "grad": grad, "edges": (post, pre, w)}


def _run_conn(s):
    conn = s["conn"]
    if s["grad"] is None:
        with torch.no_grad():
            return {"out": conn(s["x"])}
    x = s["x"].detach().requires_grad_(True)
    conn.magnitude.grad = None
    out = conn(x)
    out.backward(s["grad"])
    return {"out": out.detach(), "grad_x": x.grad, "grad_w": conn.magnitude.grad}


def _exact_conn(case, s):
    post, pre, w = s["edges"]
    n = case["n"]
    dense = torch.zeros((n, n), device="cuda", dtype=torch.float64)
    dense[pre, post] = w.double()
    x = s["x"].double()
    out = {"out": x @ dense}
    if s["grad"] is not None:
        gr = s["grad"].double()
        out["grad_x"] = gr @ dense.t()
        out["grad_w"] = (x.t() @ gr)[pre, post]
    return out


def _poisson(g, shape, rate):
    return torch.poisson(torch.full(shape, rate, device="cuda"), generator=g)


def _prepare_sim(case, seed):
    g = _gen(seed)
    n, B, T, c_in = case["n"], case["batch"], case["steps"], case["c_in"]
    post, pre = _edges(n, case["indeg"])
    batched = case["neuron"] == "alif"
    if batched:
        # weak lognormal weights with 80/20 excitation and inhibition, rounded to the grid
        w = torch.empty(pre.numel(), device="cuda").log_normal_(-1.0, 1.0, generator=g) * 0.003
        w = torch.round(torch.where(pre < int(0.8 * n), w, -0.4 * w) * 2.0**16) * 2.0**-16
        rates = (2.0 + 38.0 * torch.rand(B, generator=g, device="cuda")) * 1e-3
        x = torch.poisson(rates.view(1, B, 1).expand(T, B, c_in).contiguous(), generator=g)
        lens = torch.randint(max(1, T // 10), T + 1, (B,), generator=g, device="cuda")
    else:
        w = torch.empty(pre.numel(), device="cuda").log_normal_(-1.0, 1.0, generator=g) * 0.1
        w = torch.round(torch.where(pre < int(0.8 * n), w, -0.4 * w) * 2.0**12) * 2.0**-12
        x = _poisson(g, (T, B, c_in), 0.01)
        lens = None
    net = RecurrentNN(_neuron(case), ExponentialPSC(n, tau_syn=5.0, linear=_conn(post, pre, w, (n, n))),
                      neuron_inp_module=_dense(g, c_in, n, 0.05), update_state_names=(), cudagraph=batched).to("cuda")
    init_net_state(net, batch_size=B, dtype=torch.float32, device="cuda")
    return {"net": net, "x": x, "lens": lens, "bitmask": True}


def _prepare_traces(case, seed):
    g = _gen(seed)
    n, B, T = case["n"], case["batch"], case["steps"]
    post, pre = _edges(n, case["indeg"])
    w = _dyadic_weights(g, pre, n, 2.0**-6, 2.0**-5)
    psc = ExponentialPSC(n, tau_syn=5.0, linear=_conn(post, pre, w, (n, n)))
    syn = DelayedPSC(psc, max_delay_steps=case["delay"], use_circular_buffer=True) if case["delay"] > 1 else psc
    net = RecurrentNN(LIF(n, v_threshold=1.0, v_reset=0.0, tau=20.0, tau_ref=2.0, hard_reset=False), syn,
                      update_state_names=("neuron.v", "neuron.refractory",
                                          "synapse.psc_module.psc" if case["delay"] > 1 else "synapse.psc")).to("cuda")
    init_net_state(net, batch_size=B, dtype=torch.float32, device="cuda")
    return {"net": net, "x": _poisson(g, (T, B, n), 0.05) * 0.5, "lens": None, "bitmask": False}


def _heter(n, conn, bins, receptors):
    import pandas as pd

    if receptors == 1:
        table = pd.DataFrame({"receptor_type": ["syn"], "receptor_index": [0]})
        taus = 5.0
    else:
        table = pd.DataFrame({"receptor_type": [f"r{i}" for i in range(receptors)],
                              "receptor_index": list(range(receptors))})
        taus = torch.tensor([5.0, 3.0, 10.0, 2.5][:receptors]).repeat(n)
    return HeterSynapsePSC(n, receptors, table, conn, base_psc=ExponentialPSC, max_delay_steps=bins,
                           use_circular_buffer=True, tau_syn=taus)


def _connectome(g, n, indeg, bins, receptors=1):
    """Delay-expanded connection: lognormal in-degree, delays 1..bins, the sign by presynaptic type (70 %
    excitatory), the receptor channel of a synapse by chance."""
    post, pre = _edges(n, indeg, ragged=True)
    w = _dyadic_weights(g, pre, n, 2.0**-6, 2.0**-6, exc_frac=0.7)
    src = pre * bins + torch.randint(0, bins, (pre.numel(),), generator=g, device="cuda")
    if receptors > 1:
        col = post * receptors + torch.randint(0, receptors, (pre.numel(),), generator=g, device="cuda")
        order = torch.argsort(col * (n * bins) + src)
        post, src, w = col[order], src[order], w[order]
    return _conn(post, src, w, (n * bins, n * receptors))


def _prepare_connectome(case, seed):
    g = _gen(seed)
    n, B, T = case["n"], case["batch"], case["steps"]
    conn = _connectome(g, n, case["indeg"], 20, case["receptors"])
    neuron = LIF(n, v_threshold=1.0, v_reset=0.0, c_m=64.0, tau=20.0, tau_ref=2.0, hard_reset=True)
    net = RecurrentNN(neuron, _heter(n, conn, 20, case["receptors"]), update_state_names=(),
                      cudagraph=case["receptors"] == 1).to("cuda")
    init_net_state(net, batch_size=B, dtype=torch.float32, device="cuda")
    x = _poisson(g, (T, B, n), 0.25).mul_(8.0)
    return {"net": net, "x": x, "lens": None, "bitmask": True}


def _run_sim(s):
    net = s["net"]
    reset_net(net, batch_size=s["x"].shape[1])
    with torch.no_grad(), environ.context(dt=1.0):
        if s["bitmask"]:
            z, states = net(s["x"], sample_len=s["lens"], spikes_out="bitmask")
        else:
            z, states = net(s["x"])
    out = {"z": z, "states": states, "v": net.neuron.v, "psc": net.synapse.psc}
    if hasattr(net.neuron, "g_k"):
        out["g_k"] = net.neuron.g_k
    return out


def _prepare_train(case, seed):
    g = _gen(seed)
    n, B, T, c_in = case["n"], case["batch"], case["steps"], case["c_in"]
    post, pre = _edges(n, case["indeg"])
    w = _dyadic_weights(g, pre, n, 2.0**-9, 6.0 * 2.0**-9)
    chunk = case["chunk"]
    net = RecurrentNN(_neuron(case, surrogate_function=Sigmoid(alpha=5.0)),
                      ExponentialPSC(n, tau_syn=5.0, linear=_conn(post, pre, w, (n, n))),
                      neuron_inp_module=_dense(g, c_in, n, 0.1), update_state_names=(),
                      grad_checkpoint=chunk > 0, chunk_size=chunk or None, unroll=10).to("cuda")
    readout = torch.nn.Linear(n, 10, device="cuda")
    with torch.no_grad():
        readout.weight.copy_(torch.randn((10, n), generator=g, device="cuda") * n**-0.5)
        readout.bias.zero_()
    x = _poisson(g, (T, B, c_in), 0.02)
    freq = 1.0 + 19.0 * torch.rand((1, B, 10), generator=g, device="cuda")
    phase = 2.0 * np.pi * torch.rand((1, B, 10), generator=g, device="cuda")
    t = torch.arange(T, device="cuda").view(T, 1, 1) * 1e-3
    return {"net": net, "readout": readout, "x": x, "target": torch.sin(2.0 * np.pi * freq * t + phase)}


def _run_train(s):
    net, readout = s["net"], s["readout"]
    for p in (*net.parameters(), *readout.parameters()):
        p.grad = None
    reset_net(net, batch_size=s["x"].shape[1])
    with environ.context(dt=1.0):
        z, _ = net(s["x"])
        loss = ((readout(z) - s["target"]) ** 2).mean()
        loss.backward()
    return {"loss": loss.detach(), "z": z.detach(), "v": net.neuron.v.detach(), "psc": net.synapse.psc.detach(),
            "grad_w": net.synapse.linear.magnitude.grad, "grad_in": net.neuron_inp_module.weight.grad,
            "grad_out": readout.weight.grad}


def _prepare_serve(case, seed):
    g = _gen(seed)
    n, c_in = case["n"], case["c_in"]
    conn = _connectome(g, n, case["indeg"], 20)
    w_in = torch.round(torch.randn((c_in, n), generator=g, device="cuda").abs_() * 0.05 * 256.0) / 256.0 * 16.0
    neuron = LIF(n, v_threshold=1.0, v_reset=0.0, c_m=64.0, tau=20.0, tau_ref=2.0, hard_reset=True)
    net = RecurrentNN(neuron, _heter(n, conn, 20, 1), neuron_inp_module=DenseConn(c_in, n, weight=w_in.cpu()),
                      update_state_names=()).to("cuda")
    pool = NetworkPool("net", net, slots=case["slots"], chunk=128, device="cuda")
    # durations spread evenly over [steps / 5, steps]: the same work whatever the seed
    low, most, m = max(1, case["steps"] // 5), case["steps"], case["requests"]
    steps = [low + (i * 7 % m) * (most - low) // max(1, m - 1) for i in range(m)]
    stimuli = [_poisson(g, (t, c_in), 0.02) for t in steps]
    return {"pools": {"net": pool}, "stimuli": stimuli}


def _run_serve(s):
    server = SimulationServer(s["pools"], hbm_budget_bytes=4 << 30)
    requests = [SimRequest(network="net", stimulus=x, rid=i) for i, x in enumerate(s["stimuli"])]
    server.run(requests)
    return [r.raster for r in requests]


def _prepare_raster(case, seed):
    g = _gen(1)  # as many spikes whatever the seed, which shuffles the steps
    T, B, n = case["steps"], case["batch"], case["n"]
    words = (n + 31) // 32
    bit = torch.arange(32, device="cuda", dtype=torch.int32)
    raster = torch.empty((T, B, words), dtype=torch.int32, device="cuda")
    for t in range(0, T, 100):
        on = torch.rand((min(100, T - t), B, words, 32), generator=g, device="cuda") < case["activity"]
        on.view(on.shape[0], B, -1)[..., n:] = False
        raster[t:t + 100] = (on.int() << bit).sum(-1, dtype=torch.int32)
    return {"raster": raster[torch.randperm(T, generator=_gen(seed), device="cuda")], "n": n}


def _run_raster(s):
    rep = raster_to_sparse_repr(s["raster"], s["n"])
    return [np.asarray(rep[k][1]) for k in sorted(rep)]


_PREPARE = {"cell": _prepare_cell, "conn": _prepare_conn, "sim": _prepare_sim, "traces": _prepare_traces,
            "connectome": _prepare_connectome, "train": _prepare_train, "serve": _prepare_serve,
            "raster": _prepare_raster}
_RUN = {"cell": _run_cell, "conn": _run_conn, "sim": _run_sim, "traces": _run_sim, "connectome": _run_sim,
        "train": _run_train, "serve": _run_serve, "raster": _run_raster}
_EXACT = {"cell": _exact_cell, "conn": _exact_conn}


def prepare(case, seed):
    return dict(_PREPARE[case["kind"]](case, seed), kind=case["kind"])


def run(state):
    return _RUN[state["kind"]](state)


def exact(case, seed):
    """Single steps and single layers have a value in 64 bits.  A simulation's spikes do not (one rounding at the
    threshold moves every later step), and a raster export holds whole numbers."""
    if case["kind"] not in _EXACT:
        return None
    return _EXACT[case["kind"]](case, prepare(case, seed))


def work(case):
    kind, n = case["kind"], case["n"]
    if kind == "raster":
        rows = case["steps"] * case["batch"]
        spikes = rows * n * case["activity"]
        return {"bytes": 4 * rows * ((n + 31) // 32) + 16 * spikes, "flops": 0}
    nnz = n * case["indeg"]
    words = (n + 31) // 32
    if kind == "cell":
        return {"bytes": 8 * nnz + 4 * case["batch"] * n * 8, "flops": 30 * case["batch"] * n}
    if kind == "conn":
        B, a = case["batch"], case["activity"]
        both = 2 if case["grad"] else 1
        return {"bytes": 8 * nnz * both + (4 * nnz if case["grad"] else 0) + 8 * B * n * both,
                "flops": 2 * nnz * B * a + (2 * nnz * B + 2 * nnz * B * a if case["grad"] else 0)}
    if kind == "serve":
        steps, batch = int(0.6 * case["steps"]) * case["requests"], 1
        fed = case["c_in"]
    else:
        steps, batch = case["steps"], case["batch"]
        fed = case.get("c_in", n)
    cells = steps * batch * n
    traced = 4 if kind == "traces" else 0
    data = 8 * nnz + 4 * steps * batch * fed + 4 * steps * batch * words + 4 * traced * cells
    data += 4 * fed * n if "c_in" in case else 0
    flops = (60 if case.get("neuron") == "alif" else 25) * cells
    if kind == "train":
        # spikes out, gradient of every stored weight, the transposed product of every step
        data += 4 * cells + 4 * nnz + 4 * fed * n
        flops = 3 * flops + 2 * nnz * steps * batch
    return {"bytes": data, "flops": flops}
