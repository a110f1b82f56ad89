"""A run that overwrites a circular spike history in place says so to autograd:
a gradient that needs the old values is refused, not computed from the new."""
import pytest
import torch

from btorch_b200.models.history import SpikeHistory

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("circular", [True, False])
@pytest.mark.parametrize("inference", [False, True])
def test_from_ring_counts_as_a_write(circular, inference):
    n, batch, depth = 40, 2, 3
    hist = SpikeHistory(n, max_delay_steps=depth, use_circular_buffer=circular)
    with torch.inference_mode(inference):
        hist.init_state(batch, device=DEV, dtype=torch.float32)
        ring = torch.randint(-2**31, 2**31 - 1, (depth + 2, batch, 2), dtype=torch.int32, device=DEV)
        old = hist.history
        if inference:
            hist.from_ring(ring, batch, 20, 3)
            return
    w = torch.ones((), device=DEV, requires_grad=True)
    loss = (old * w).sum()  # its backward needs the history of now
    cursor = hist._cursor._version if circular else None
    hist.from_ring(ring, batch, 20, 3)
    if circular:
        assert hist.history is old and hist._cursor._version > cursor
        with pytest.raises(RuntimeError, match="modified by an inplace operation"):
            loss.backward()
    else:
        assert hist.history is not old
        loss.backward()
