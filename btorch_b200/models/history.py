"""Rolling spike history (API and layout of btorch/models/history.py:28-358).

Memory ``history`` has shape (*batch, max_delay, *n_neuron).  Circular mode
keeps a cursor (slot cursor-1 is the most recent spike); cat mode keeps the
most recent spike at index 0.  ``get_flattened(D)`` interleaves neurons and
delays [n0_d0, n0_d1, ..., n1_d0, ...], the row order of
expand_conn_for_delays.  The fused engine reads and writes this state when a
run starts and ends; stepping module by module uses these tensor moves.
"""

from __future__ import annotations

import torch

from .. import _lib as L
from .base import MemoryModule, normalize_n_neuron


class SpikeHistory(MemoryModule):
    def __init__(self, n_neuron, max_delay_steps: int = 5, use_circular_buffer: bool = True):
        super().__init__()
        self.n_neuron, self.size = normalize_n_neuron(n_neuron)
        self.max_delay = int(max_delay_steps)
        self.use_circular_buffer = use_circular_buffer
        self.register_memory("history", torch.tensor(0.0, dtype=torch.float32), (self.max_delay, *self.n_neuron))
        if use_circular_buffer:
            self.register_buffer("_cursor", torch.tensor(0, dtype=torch.long), persistent=False)

    def init_state(self, batch_size=None, dtype=None, device=None, persistent=False, skip_mem_name=()):
        super().init_state(batch_size, dtype, device, persistent, skip_mem_name)
        if self.use_circular_buffer:
            self._cursor = torch.tensor(0, dtype=torch.long, device=device)

    def reset(self, batch_size=None, dtype=None, device=None, skip_mem_name=(), inplace: bool = False):
        super().reset(batch_size, dtype, device, skip_mem_name, inplace=inplace)
        if self.use_circular_buffer:
            if inplace:
                self._cursor.zero_()
            else:
                self._cursor = torch.tensor(0, dtype=torch.long, device=self._cursor.device)

    def _nb(self) -> int:
        return self.history.ndim - 1 - len(self.n_neuron)

    def _delay_first(self) -> torch.Tensor:
        h = self.history
        nb = self._nb()
        if nb <= 0:
            return h
        return h.movedim(nb, 0)

    def update(self, spike: torch.Tensor) -> "SpikeHistory":
        if getattr(self, "history", None) is None:
            raise RuntimeError("SpikeHistory buffer not initialized. Call init_state() before first update().")
        spike = spike.to(self.history.dtype)
        nb = self._nb()
        if self.use_circular_buffer:
            # index ops with a device-side index: no host sync, so the update
            # can be captured in a CUDA graph
            h = self._delay_first()
            h.index_copy_(0, self._cursor.view(1), spike.unsqueeze(0))
            self._cursor.copy_((self._cursor + 1) % self.max_delay)
        else:
            h = self._delay_first()
            new = torch.cat([spike.unsqueeze(0), h[:-1]], dim=0)
            self.history = new.movedim(0, nb) if nb > 0 else new
        return self

    def get_delay(self, delay_steps: int) -> torch.Tensor:
        if delay_steps >= self.max_delay:
            raise IndexError(f"delay_steps ({delay_steps}) >= max_delay ({self.max_delay}). "
                             "Increase max_delay_steps or use smaller delays.")
        h = self._delay_first()
        if self.use_circular_buffer:
            return h.index_select(0, ((self._cursor - 1 - delay_steps) % self.max_delay).view(1)).squeeze(0)
        return h[delay_steps]

    def get_recent(self, n_steps: int) -> list[torch.Tensor]:
        if n_steps > self.max_delay:
            raise IndexError(f"n_steps ({n_steps}) > max_delay ({self.max_delay})")
        return [self.get_delay(d) for d in range(n_steps)]

    def get_flattened(self, n_delays: int) -> torch.Tensor:
        if n_delays > self.max_delay:
            raise IndexError(f"n_delays ({n_delays}) > max_delay ({self.max_delay})")
        st = torch.stack([self.get_delay(d) for d in range(n_delays)], dim=0)  # (D, *batch, *n)
        st = st.reshape(n_delays, *st.shape[1: st.ndim - len(self.n_neuron)], self.size)
        return st.movedim(0, -1).reshape(*st.shape[1:-1], self.size * n_delays)

    # -- engine interface: the last `k` spikes as [k][batch][n], index d = d steps ago
    def recent_block(self, k: int) -> torch.Tensor:
        return torch.stack([self.get_delay(d).reshape(-1, self.size) for d in range(k)])

    def store_recent_block(self, block: torch.Tensor, advance: int) -> None:
        """Set the history to what the reference holds after `advance` more
        update() calls whose last max_delay spikes are `block` [max_delay][batch][n]
        (index d = d steps ago).  Circular mode advances the cursor by `advance`."""
        k = block.shape[0]
        assert k == self.max_delay
        nb = self._nb()
        new = block.reshape(k, *self.history.shape[:nb], *self.n_neuron).to(self.history.dtype)
        if self.use_circular_buffer:
            self._cursor.copy_((self._cursor + advance) % k)
            order = (self._cursor - 1 - torch.arange(k, device=self._cursor.device)) % k
            h = self._delay_first()
            h[order] = new
        else:
            self.history = new.movedim(0, nb).contiguous() if nb > 0 else new.clone()

    def _kernel_state(self, batch: int) -> bool:
        """The history is [batch][max_delay][n] contiguous fp32 on the device."""
        h = self.history
        return (h.is_cuda and h.dtype == torch.float32 and h.is_contiguous()
                and h.numel() == batch * self.max_delay * self.size
                and (not self.use_circular_buffer or self._cursor.device == h.device))

    def to_ring(self, ring: torch.Tensor, batch: int, t0: int) -> None:
        """The spikes d = 0 .. max_delay - 1 steps ago as bitmaps in slots
        (t0 - 1 - d) mod H of the engine's history ring [H][batch][words]."""
        H, words = ring.shape[0], ring.shape[-1]
        s = L.stream_of(ring.device)
        if self._kernel_state(batch):
            cursor = self._cursor.data_ptr() if self.use_circular_buffer else None
            L.check(L.lib().bt_history_load(batch, self.max_delay, self.size, self.history.data_ptr(), cursor, t0, H,
                                            ring.data_ptr(), s), "bt_history_load")
            return
        block = self.recent_block(self.max_delay).float().contiguous()
        bits = torch.empty((self.max_delay, batch, words), device=ring.device, dtype=torch.int32)
        L.check(L.lib().bt_float_to_bits(self.max_delay * batch, self.size, block.data_ptr(), bits.data_ptr(), s),
                "bt_float_to_bits")
        for d in range(self.max_delay):
            ring[(t0 - 1 - d) % H] = bits[d]

    def from_ring(self, ring: torch.Tensor, batch: int, t_end: int, advance: int) -> None:
        """The state after `advance` steps from the ring's bitmaps of steps
        t_end - 1 - d (as store_recent_block)."""
        H = ring.shape[0]
        s = L.stream_of(ring.device)
        if self._kernel_state(batch):
            if self.use_circular_buffer:
                cursor = self._cursor.data_ptr()
            else:
                cursor, self.history = None, torch.empty_like(self.history)
            L.check(L.lib().bt_history_store(batch, self.max_delay, self.size, ring.data_ptr(), t_end, H, cursor,
                                             advance, self.history.data_ptr(), s), "bt_history_store")
            if self.use_circular_buffer:  # written in place: as the tensor moves below, a new version
                written = [t for t in (self.history, self._cursor) if not t.is_inference()]
                if written:
                    torch.autograd.graph.increment_version(written)
            return
        block = torch.empty((self.max_delay, batch, self.size), device=ring.device, dtype=torch.float32)
        sel = torch.stack([ring[(t_end - 1 - d) % H] for d in range(self.max_delay)]).contiguous()
        L.check(L.lib().bt_bits_to_float(self.max_delay * batch, self.size, sel.data_ptr(), block.data_ptr(), s),
                "bt_bits_to_float")
        self.store_recent_block(block, advance)
