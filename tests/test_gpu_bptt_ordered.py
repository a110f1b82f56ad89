"""Ordered (gather) training at batches around the engine's choice between a warp
and a lane per neuron: the same spikes, states and gradients as the single-step
kernels, stored and recomputed."""
import pytest
import torch

from btorch_b200.models import bptt
from tests.test_gpu_bptt_native import run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,B", [(33, 3), (33, 4), (65, 31), (500, 200), (40, 260)])
@pytest.mark.parametrize("chunk", [0, 5])
def test_ordered_training_equals_single_steps(monkeypatch, n, B, chunk):
    modes = []
    steps = bptt._Run.steps

    def seen(self, *a, **k):
        modes.append(self.desc.mode)
        return steps(self, *a, **k)

    monkeypatch.setattr(bptt._Run, "steps", seen)
    with pytest.MonkeyPatch.context() as inner:
        a = run(inner, True, n, B, "lif", True, True, 7, chunk, "gather", True, False)
    assert set(modes) == {bptt.L.BT_MODE_PULL if B >= 4 else bptt.L.BT_MODE_GATHER}
    with pytest.MonkeyPatch.context() as inner:
        b = run(inner, False, n, B, "lif", True, True, 7, chunk, "gather", True, False)
    assert a["z"].sum() > 0
    for key in a:
        if key.startswith("g"):
            assert float((a[key] - b[key]).double().norm()) <= 1e-5 * float(b[key].double().norm().clamp(min=1e-30)), key
        else:
            assert torch.equal(a[key], b[key]), key
