"""The fused BPTT's memory gate on a device that is nearly full: the call steps
module by module, with the same gradients, instead of running out of memory."""
import time

import pytest
import torch

from btorch_b200.models import LIF, ExponentialPSC, RecurrentNN, Sigmoid, SparseConn, bptt, environ
from btorch_b200.models.functional import init_net_state

pytestmark = pytest.mark.gpu
DEV = "cuda"


def step(net, x):
    init_net_state(net, batch_size=x.shape[1], dtype=torch.float32, device=DEV)
    net.zero_grad()
    with environ.context(dt=1.0):
        z, _ = net(x)
        z.sum().backward()
    return net.last_path, z.detach(), net.synapse.linear.magnitude.grad.clone()


def network(n=64):
    g = torch.Generator().manual_seed(0)
    w = (torch.rand((n, n), generator=g) < 0.3).float() * 2.0**-4
    return RecurrentNN(LIF(n, surrogate_function=Sigmoid(alpha=2.0)), ExponentialPSC(n, 5.0, SparseConn(w.numpy())),
                       update_state_names=()).to(DEV)


def same(a, b):
    assert torch.equal(a[1], b[1])
    assert float((a[2] - b[2]).norm()) <= 1e-5 * float(b[2].norm())


def test_nearly_full_device_steps_module_by_module(monkeypatch):
    net = network()
    x = (torch.rand((12, 4, 64), device=DEV) < 0.4).float() * 2.0
    getattr(bptt, "_FREE", {}).clear()
    want = step(net, x)
    assert want[0] == "fused-bptt" and want[1].sum() > 0
    asked = []
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda dev=None: asked.append(dev) or (1 << 16, 180 << 30))
    time.sleep(getattr(bptt, "FREE_AGE", 0.0) + 0.1)
    got = step(net, x)
    assert got[0] != "fused-bptt" and asked
    same(got, want)


def test_running_out_of_memory_steps_module_by_module(monkeypatch):
    net = network()
    x = (torch.rand((12, 4, 64), device=DEV) < 0.4).float() * 2.0
    want = step(net, x)

    def full(*a):
        raise torch.OutOfMemoryError("no memory left")

    monkeypatch.setattr(bptt._FusedBPTT, "apply", full)
    got = step(net, x)
    assert got[0] != "fused-bptt"
    same(got, want)


def test_small_calls_do_not_ask_the_driver_each_time(monkeypatch):
    asked = []
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda dev=None: asked.append(dev) or (1 << 34, 180 << 30))
    monkeypatch.setattr(bptt, "FREE_AGE", 60.0)
    dev = torch.device(DEV, 0)
    bptt._FREE.clear()
    assert all(bptt.fits(dev, 1 << 20) for _ in range(5)) and len(asked) == 1
    assert bptt.fits(dev, 1 << 31) and len(asked) == 2  # a call of a size that matters
    assert not bptt.fits(dev, 1 << 33) and len(asked) == 3
    bptt._FREE.clear()
