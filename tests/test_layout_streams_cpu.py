"""A layout's index arrays are the host builder's own: what a launch reads is
never derived later on one caller's stream and kept for the others."""
import numpy as np
import pytest
import torch

from btorch_b200 import _lib as L
from btorch_b200.models import SparseConn, _ops


class Recorder:
    """The library with its launching entries replaced by records of their arguments."""

    def __init__(self, real):
        self.real, self.calls = real, {}

    def __getattr__(self, name):
        if name.startswith("bt_pack_edges") or name.startswith("bt_spmv_push") and not name.endswith("words"):
            return lambda *a: self.calls.setdefault(name, []).append(a) or 0
        return getattr(self.real, name)


@pytest.mark.parametrize("nnz_mask", [0.0, 0.3])
def test_launches_read_the_layouts_own_permutation(monkeypatch, nnz_mask):
    rng = np.random.default_rng(1)
    post, src = np.nonzero(rng.random((9, 13)) < nnz_mask)
    m = SparseConn.from_canonical(post, src, np.ones(post.size, np.float32), (13, 9), enforce_dale=False)
    lay = m.layout("cpu")
    lib = Recorder(L.lib())
    monkeypatch.setattr(L, "lib", lambda: lib)
    monkeypatch.setattr(L, "stream_of", lambda dev: 0)
    before = dict(lay.__dict__)
    for _ in range(2):
        _ops._spmv("scatter", lay, torch.ones(2, 13), m.magnitude.detach(), None)
        _ops.pack_edges(lay, m.magnitude.detach())
    own = lay.csr_perm.data_ptr()
    assert lay.csr_perm.dtype == torch.int32
    assert [c[6] for c in lib.calls["bt_spmv_push"]] == [own, own]
    assert [c[3] for c in lib.calls["bt_pack_edges"]] == [own, own]
    assert lay.__dict__.keys() == before.keys()  # the calls added nothing to the layout
