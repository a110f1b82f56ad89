"""Cluster engine, waits that run into their limit: the call raises, no word or
bulk copy is left under way (the drain behind the loop), and the next call of the
same network is right.  Both time loops: a warp per item, and several items per
warp with per-neuron divisors.  Small limits, so that the waits give up at
different steps; a limit that suffices gives the right result."""
import numpy as np
import pytest
import torch

from btorch_b200.models import environ
from btorch_b200.models.functional import init_net_state
from tests.test_gpu_cluster import GATHER, _dyadic, _model, cluster

pytestmark = pytest.mark.gpu


def reset(rnn, batch):
    init_net_state(rnn, batch_size=batch, dtype=torch.float32, device="cuda")


@pytest.mark.parametrize("n,batch,steps,per_neuron", [(4096, 1, 60, False), (1000, 3, 61, False), (1500, 4, 30, True),
                                                      (700, 24, 7, True), (96, 1, 1, False), (64, 2, 2, True)])
def test_waits_that_give_up(n, batch, steps, per_neuron):
    rng = np.random.default_rng(n)
    rnn = _model(_dyadic(rng, n, min(0.2, 60 / n)), n, 0, batch, names=())
    if per_neuron:
        rnn.neuron.tau = torch.linspace(10.0, 30.0, n, device="cuda")
    x = torch.tensor((rng.random((steps, batch, n)) < 0.1).astype(np.float32) * 8.0, device="cuda")
    reset(rnn, batch)
    with torch.no_grad(), environ.context(dt=1.0):
        want, _ = rnn(x, engine_choice=GATHER)
        assert want.sum() > 0
        gave_up = 0
        for limit in (1, 1, 2, 4, 8, 16, 40, 100, 250, 600):
            reset(rnn, batch)
            rnn.engine_spin_limit = limit
            try:
                z, _ = rnn(x, engine_choice=cluster())
                assert torch.equal(z, want)
            except RuntimeError as e:
                assert "gave up" in str(e)
                gave_up += 1
            torch.cuda.synchronize()
            rnn.engine_spin_limit = 0
            reset(rnn, batch)
            z, _ = rnn(x, engine_choice=cluster())
            assert torch.equal(z, want)
    if n >= 1000:
        assert gave_up >= 1
