"""Spike history to and from the engine's ring (bt_history_load / bt_history_store)
against the module's own tensor moves, and the packed edge records against
indexing: whole numbers, so equal."""
import pytest
import torch

from btorch_b200.models._ops import pack_edges
from btorch_b200.models.history import SpikeHistory

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("circular", [True, False])
@pytest.mark.parametrize("n,batch,depth,advance", [(1, 1, 1, 0), (31, 2, 3, 1), (32, 1, 5, 5), (33, 3, 4, 2),
                                                   (100, 2, 20, 7), (65, 1, 2, 1000)])
def test_history_ring_round_trip(circular, n, batch, depth, advance):
    g = torch.Generator(device=DEV).manual_seed(n + depth)
    hist = SpikeHistory(n, max_delay_steps=depth, use_circular_buffer=circular)
    hist.init_state(batch, device=DEV, dtype=torch.float32)
    for _ in range(depth + 2):
        hist.update((torch.rand((batch, n), generator=g, device=DEV) < 0.3).float())
    want = hist.recent_block(depth)  # [d][batch][n]
    H, words, t0 = depth + 2, (n + 31) // 32, 40 * (depth + 2)
    ring = torch.zeros((H, batch, words), dtype=torch.int32, device=DEV)
    hist.to_ring(ring, batch, t0)
    bit = torch.arange(32, device=DEV, dtype=torch.int32)
    for d in range(depth):
        row = ring[(t0 - 1 - d) % H]
        got = ((row[..., None] >> bit) & 1).reshape(batch, -1)[:, :n].float()
        torch.testing.assert_close(got, want[d], rtol=0, atol=0)
    # new spikes in the ring, read back as the state after `advance` steps
    new = torch.randint(0, 2, (H, batch, words * 32), generator=g, device=DEV)
    new[..., n:] = 0
    ring.copy_((new.view(H, batch, words, 32).int() << bit).sum(-1, dtype=torch.int32))
    before = hist._cursor.clone() if circular else None
    hist.from_ring(ring, batch, t0 + advance, advance)
    for d in range(depth):
        torch.testing.assert_close(hist.get_delay(d).reshape(batch, n), new[(t0 + advance - 1 - d) % H, :, :n].float(),
                                   rtol=0, atol=0)
    if circular:
        assert int(hist._cursor) == (int(before) + advance) % depth


@pytest.mark.parametrize("nnz", [0, 1, 3, 4, 5, 1023, 1030])
def test_pack_edges(nnz):
    from types import SimpleNamespace

    from btorch_b200.models._ops import pad4

    padded = pad4(nnz)
    lay = SimpleNamespace(nnz=nnz, csr_dst=torch.randint(0, 1 << 30, (padded,), dtype=torch.int32, device=DEV),
                          csr_perm=torch.randperm(max(nnz, 1), device=DEV)[:nnz])
    w = torch.randn(max(nnz, 1), device=DEV)
    rec = pack_edges(lay, w).view(-1, 2)
    assert torch.equal(rec[:, 0], lay.csr_dst)
    assert torch.equal(rec[:nnz, 1], w[lay.csr_perm].view(torch.int32))
    assert (rec[nnz:, 1] == 0).all()
