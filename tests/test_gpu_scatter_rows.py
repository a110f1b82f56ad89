"""The scatter that sums a sample's rows in shared memory (32-lane choice, 32
samples and more, up to 16384 neurons) against the one that reduces in L2 (the
8-lane choice): on dyadic weights, whose sums are exact in any order, rasters,
traces and final state are equal bit for bit.  Sizes: below a warp, not a
multiple of 4 or 32, the largest of the range; batches that are not a multiple
of the mask word; shares with more rows than the block's list holds; uneven
lengths, a uniform delay, dense steps, several calls in a row."""

import numpy as np
import pytest
import scipy.sparse as sp
import torch

from btorch_b200 import _lib as L
from btorch_b200.models import ALIF, LIF, DelayedPSC, ExponentialPSC, RecurrentNN, SparseConn, environ
from btorch_b200.models.autotune import EngineChoice
from btorch_b200.models.functional import init_net_state

pytestmark = pytest.mark.gpu


def _net(n, indeg, batch, delay, alif):
    rng = np.random.default_rng(n + batch)
    post = np.repeat(np.arange(n), indeg)
    src = rng.integers(0, n, n * indeg)
    w = rng.integers(1, 5, n * indeg) * 2.0**-7 * np.where(src < 0.8 * n, 1.0, -2.0)
    conn = SparseConn(sp.coo_array((w.astype(np.float32), (src, post)), shape=(n, n)),
                      sparse_config={"direction": "scatter"})
    psc = ExponentialPSC(n, 5.0, conn)
    neuron = ALIF(n, g_leak=0.05, E_leak=0.0, E_k=-1.0, dg_k=0.0625, tau_adapt=200.0, tau_ref=2.0,
                  hard_reset=True) if alif else LIF(n, tau_ref=2.0, hard_reset=True)
    rnn = RecurrentNN(neuron, DelayedPSC(psc, max_delay_steps=delay) if delay else psc,
                      update_state_names=("neuron.v",)).cuda()
    init_net_state(rnn, batch_size=batch, dtype=torch.float32, device="cuda")
    return rnn


# n, in-degree, batch, steps, uniform delay, ALIF, dense rows, drive
@pytest.mark.parametrize("n, indeg, batch, steps, delay, alif, dense, drive", [
    (7, 3, 32, 20, 0, False, 0, 2.0),
    (33, 20, 33, 20, 0, False, 0, 1.0),
    (1000, 60, 64, 24, 0, True, 0, 0.3),
    (2050, 60, 100, 16, 0, False, 0, 0.5),
    (4100, 60, 129, 12, 3, False, 0, 0.5),
    (1001, 50, 40, 16, 2, False, 0, 0.5),
    (2000, 60, 64, 16, 0, False, -1, 3.0),      # dense steps among the others
    (16384, 60, 32, 8, 0, False, 0, 1.0),
    (16384, 20, 256, 5, 0, False, 0, 30.0),     # every neuron fires: more rows a share than the list holds
])
def test_scatter_rows_equals_reductions(n, indeg, batch, steps, delay, alif, dense, drive):
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randint(0, 9, (steps, batch, n), generator=g, device="cuda").float() * (drive / 8.0)
    lens = torch.arange(batch, device="cuda") % steps + 1
    lens[::2] = steps
    outs = []
    for lanes in (8, 32):
        rnn = _net(n, indeg, batch, delay, alif)
        choice = EngineChoice(L.BT_MODE_SCATTER, scatter_lanes=lanes, neuron_spt=4, dense_rows=dense)
        got = []
        with torch.no_grad(), environ.context(dt=1.0):
            for a, b in ((0, steps // 2), (steps // 2, steps)):  # two calls: pending delays cross them
                z, st = rnn(x[a:b], sample_len=(lens - a).clamp(0, b - a), engine_choice=choice)
                got += [z, st["neuron.v"]]
        assert rnn.last_path == "fused"
        psc = rnn.synapse.psc_module.psc if delay else rnn.synapse.psc
        outs.append([t.cpu().numpy() for t in (*got, rnn.neuron.v, psc)])
    assert outs[0][0].sum() > 0
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)
