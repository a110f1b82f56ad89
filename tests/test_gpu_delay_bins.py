"""Scatter delivery over wide delay ranges: as many delay bins as the engine
takes, around 64 of them, all of them occupied or a range that starts late,
against the ordered gather.  Dyadic weights: sums are exact in any order, so
rasters, traces and final state are equal bit for bit."""
import numpy as np
import pandas as pd
import pytest
import scipy.sparse as sp
import torch

from btorch_b200 import _lib as L
from btorch_b200.models import LIF, DelayedPSC, ExponentialPSC, HeterSynapsePSC, RecurrentNN, SparseConn, environ
from btorch_b200.models.autotune import EngineChoice
from btorch_b200.models.functional import init_net_state

pytestmark = pytest.mark.gpu
GATHER = EngineChoice(L.BT_MODE_GATHER)


def run(rnn, x, choice, batch, names):
    init_net_state(rnn, batch_size=batch, dtype=torch.float32, device="cuda")
    T, got = x.shape[0], []
    with torch.no_grad(), environ.context(dt=1.0):
        for a, b in ((0, T // 3), (T // 3, T)):  # two calls: pending delays cross them
            z, st = rnn(x[a:b], engine_choice=choice)
            got += [z, st["neuron.v"]]
    assert rnn.last_path == "fused"
    return [t.cpu().numpy() for t in (*got, rnn.neuron.v, names(rnn))]


def compare(make, x, batch, names, **choice):
    want = run(make(), x, GATHER, batch, names)
    got = run(make(), x, EngineChoice(L.BT_MODE_SCATTER, neuron_spt=1, **choice), batch, names)
    assert want[0].sum() > 0
    for a, b in zip(want, got):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("lanes", [1, 8, 32])
@pytest.mark.parametrize("bins,first,receptors,batch", [(63, 0, 1, 2), (64, 0, 1, 2), (65, 0, 3, 2), (128, 0, 1, 3),
                                                        (128, 0, 2, 130), (120, 57, 1, 2), (128, 63, 1, 1)])
def test_wide_delay_ranges_equal_gather(lanes, bins, first, receptors, batch):
    rng = np.random.default_rng(bins + first)
    n, nnz, T = 96, 12000, 150
    pre, post = rng.integers(0, n, nnz), rng.integers(0, n * receptors, nnz)
    delay = rng.integers(first, bins, nnz)
    delay[0], delay[1] = first, bins - 1
    key = np.unique((pre * bins + delay) * (n * receptors) + post)
    src, post = key // (n * receptors), key % (n * receptors)
    w = (rng.integers(1, 5, key.size) * 2.0**-6 * np.where(rng.random(key.size) < 0.8, 1.0, -2.0)).astype(np.float32)
    m = sp.coo_array((w, (src, post)), shape=(n * bins, n * receptors))
    rti = pd.DataFrame({"receptor_type": [f"r{r}" for r in range(receptors)], "receptor_index": list(range(receptors))})

    def make():
        conn = SparseConn(m, enforce_dale=False, sparse_config={"direction": "scatter"})
        syn = HeterSynapsePSC(n, receptors, rti, conn, max_delay_steps=bins, use_circular_buffer=True, tau_syn=5.0)
        return RecurrentNN(LIF(n, tau_ref=2.0, hard_reset=True), syn, update_state_names=("neuron.v",)).cuda()

    x = torch.tensor((rng.random((T, batch, n)) < 0.05).astype(np.float32) * 1.5, device="cuda")
    compare(make, x, batch, lambda rnn: rnn.synapse.base_psc.psc, scatter_lanes=lanes)


@pytest.mark.parametrize("lanes", [1, 8, 32])
@pytest.mark.parametrize("dense", [0, -1])
@pytest.mark.parametrize("delay,n,batch", [(0, 300, 3), (2, 96, 40), (127, 200, 33)])
def test_one_plane_with_and_without_dense_steps(lanes, dense, delay, n, batch):
    rng = np.random.default_rng(n)
    w = np.where(rng.random((n, n)) < 0.2, rng.integers(1, 5, (n, n)) * 2.0**-6, 0.0).astype(np.float32)

    def make():
        psc = ExponentialPSC(n, 5.0, SparseConn(w, sparse_config={"direction": "scatter"}))
        return RecurrentNN(LIF(n, tau_ref=2.0, hard_reset=True), DelayedPSC(psc, max_delay_steps=delay) if delay else psc,
                           update_state_names=("neuron.v",)).cuda()

    x = torch.tensor((rng.random((delay + 30, batch, n)) < 0.3).astype(np.float32) * 8.0, device="cuda")
    x[1::7] = 16.0  # steps in which most neurons fire in every sample
    compare(make, x, batch, lambda rnn: (rnn.synapse.psc_module if delay else rnn.synapse).psc, scatter_lanes=lanes,
            dense_rows=dense)


@pytest.mark.parametrize("batch,every", [(1, 1), (1, 3), (33, 1)])
def test_more_rows_than_one_pass_takes(batch, every):
    """Bursts that list more rows than the grid's warps take at once (32 each): several passes, equal shares."""
    n, bins, T = 16384, 20, 26
    rng = np.random.default_rng(7)
    pre, post, delay = (rng.integers(0, k, 40 * n) for k in (n, n, bins))
    key = np.unique((pre * bins + delay) * n + post)
    w = (rng.integers(1, 5, key.size) * 2.0**-8).astype(np.float32)
    m = sp.coo_array((w, (key // n, key % n)), shape=(n * bins, n))
    rti = pd.DataFrame({"receptor_type": ["syn"], "receptor_index": [0]})

    def make():
        conn = SparseConn(m, enforce_dale=False, sparse_config={"direction": "scatter"})
        syn = HeterSynapsePSC(n, 1, rti, conn, max_delay_steps=bins, use_circular_buffer=True, tau_syn=5.0)
        return RecurrentNN(LIF(n, hard_reset=True), syn, update_state_names=("neuron.v",)).cuda()

    x = torch.zeros((T, batch, n), device="cuda")
    x[:, :, ::every] = 32.0  # they fire in every step
    compare(make, x, batch, lambda rnn: rnn.synapse.base_psc.psc, scatter_lanes=1)
