"""Fused surrogate-gradient BPTT for RecurrentNN calls that need gradients.

The per-module path builds one autograd node per module per step (neuron,
sparse product, synapse), so a truncated-BPTT window of T steps costs ~6 T
Python-level autograd nodes in the forward and as many backward calls.  For
the common training model -- LIF/ALIF neurons, an ExponentialPSC over a
SparseConn whose weight is its magnitude parameter, an optional DenseConn /
nn.Linear input layer -- this module runs the whole call as ONE autograd
Function: the forward is the multi-step engine with its state traces
(bt_engine_run), the backward one native call per chunk of steps:

    forward, step t:  P_t = x_t W_in^T (+ b)                  (bt_input_project)
                      I_t = psc_{t-1} + P_t                  (rnn.py:524)
                      z_t, v_t, gk_t = neuron(I_t, v_{t-1}, gk_{t-1})
                      psc_t = psc_{t-1} + coef*((-psc_{t-1})/tau) + W z_t
    backward, step t: dz_t  = gZ_t + W^T dpsc_t
                      dI_t, dv_{t-1}, dgk_{t-1} = neuron'(dz_t, dv_t, dgk_t)
                      dpsc_{t-1} = dpsc_t + coef*((-dpsc_t)/tau) + dI_t
                                                             (bt_bptt_backward)
    weight gradients: dW = sum over (t, b) of z_t[b, pre] dpsc_t[b, post]
                      (bt_spmv_grad_weight_rows, stored nonzeros only);
                      dW_in = sum over (t, b) of x_t[b]^T dI_t[b], over the
                      nonzero inputs only (bt_input_grad_weight).

A smooth (non-spiking) surrogate forward, which the engine does not run, and
shapes outside its limits step through the single-step kernels instead
(_Steps), with the same results.

Checkpointed recompute (RecurrentNN(grad_checkpoint=True), the reference's
per-chunk checkpoint, rnn.py:177-197): with chunks of C steps (chunk_size,
or unroll when chunk_size is None) the forward keeps only the spikes, the
requested state stacks and the state at every chunk start; the backward
recomputes each chunk's forward from its start state into chunk-sized
buffers (driving the synaptic recurrence with the stored spikes) and runs
that chunk's backward, accumulating the weight gradients chunk by chunk.
Memory is O(C batch n) for the step buffers instead of O(T batch n).
Without checkpointing every step's buffers are kept and nothing is
recomputed.  Gradients equal the per-module path's up to fp32 summation
order (tests compare both with the reference's autograd within 1e-4).
"""

from __future__ import annotations

import ctypes as CT
import time

import torch
import torch.nn as nn

from .. import _lib as L
from . import _ops, environ
from ._ops import _csr_weights_cached, _spmv, neuron_desc, pack_csr_weights, pack_edges, scalar_values
from .functional import named_hidden_states
from .linear import DenseConn, SparseConn
from .neurons.alif import ALIF
from .neurons.lif import LIF
from .synapse import ExponentialPSC

MEMORY_FRACTION = 0.25  # largest share of free device memory the step buffers may take
FREE_AGE = 0.5  # seconds for which a figure of the free memory serves calls far below it
_FREE: dict = {}  # device -> (when, free bytes) as last asked for


def fits(device, need: int) -> bool:
    """`need` bytes are at most MEMORY_FRACTION of the free device memory.
    Asking the driver takes up to milliseconds, as long as a small call: one
    that needs less than a sixteenth of what is allowed goes by a figure up to
    FREE_AGE seconds old."""
    when, free = _FREE.get(device, (float("-inf"), 0))
    now = time.monotonic()
    if now - when > FREE_AGE or 16 * need > MEMORY_FRACTION * free:
        free = torch.cuda.mem_get_info(device)[0]
        _FREE[device] = (now, free)
    return need <= MEMORY_FRACTION * free


def match(rnn) -> tuple[dict | None, str]:
    """The state kinds to stack (key -> "v" / "psc" / "gk" / "ref") when the
    call can run through the fused BPTT, else (None, reason)."""
    neuron, syn = rnn.neuron, rnn.synapse
    if type(neuron) not in (LIF, ALIF) or neuron.pre_spike_v:
        return None, "neuron"
    if any(p.requires_grad for p in neuron.parameters(recurse=False)):
        return None, "neuron parameter gradients"
    if type(syn) is not ExponentialPSC or type(syn.linear) is not SparseConn or syn.linear.bias is not None:
        return None, "synapse"
    if rnn.syn_inp_module is not None:
        return None, "syn_inp_module"
    if rnn.neuron_inp_module is not None and type(rnn.neuron_inp_module) not in (nn.Linear, DenseConn):
        return None, "neuron_inp_module"
    if rnn.cpu_offload or rnn.cudagraph or rnn.save_grad_history:
        return None, "offload / graphs / grad history"
    if syn.linear.in_features != neuron.size or syn.linear.out_features != neuron.size:
        return None, "connectivity shape"
    if syn.linear.indices.shape[1] == 0:
        return None, "no synapses"
    paths = {}
    npath = next(name for name, m in rnn.named_modules() if m is neuron)
    spath = next(name for name, m in rnn.named_modules() if m is syn)
    for key in named_hidden_states(rnn, rnn.update_state_names, allow_buffer=rnn.allow_buffer):
        kind = {f"{npath}.v": "v", f"{npath}.g_k": "gk", f"{npath}.refractory": "ref", f"{spath}.psc": "psc"}.get(key)
        if kind is None:
            return None, f"state '{key}'"
        paths[key] = kind
    return paths, ""


def checkpoint_chunk(rnn, T: int) -> int:
    """Steps per recomputed chunk: the reference's checkpoint chunk (chunk_size,
    else unroll) with grad_checkpoint, else T (nothing recomputed)."""
    if not rnn.grad_checkpoint:
        return T
    if rnn.chunk_size is not None:
        return max(1, min(T, int(rnn.chunk_size)))
    return T if rnn.unroll is False else max(1, min(T, int(rnn.unroll)))


class _Steps:
    """The forward of one chunk into chunk-sized buffers (shared by the
    forward pass and the backward recomputation)."""

    def __init__(self, B, n, Cb, has_gk, has_ref, proj, c_in, dev):
        new = lambda *shape: torch.empty(shape, device=dev, dtype=torch.float32)  # noqa: E731
        self.I, self.U, self.M, self.VCH = new(Cb, B, n), new(Cb, B, n), new(Cb, B, n), new(Cb, B, n)
        self.Vs, self.Ps = new(Cb + 1, B, n), new(Cb + 1, B, n)
        self.GKs = new(Cb + 1, B, n) if has_gk else None
        self.REFs = new(Cb + 1, B, n) if has_ref else None
        self.Pc = new(Cb, B, n) if proj else None
        self.pw = torch.empty(max(1, Cb * B * (2 * c_in + 1)), device=dev, dtype=torch.int32) if proj else None
        self.zr = new(B, n)

    def load(self, v, p, gk, ref):
        self.Vs[0].copy_(v)
        self.Ps[0].copy_(p)
        if self.GKs is not None:
            self.GKs[0].copy_(gk)
        if self.REFs is not None:
            self.REFs[0].copy_(ref)

    def run(self, k, kc, xin, w_t, bias, Z, z_given, d, coef, tau, direction, lay, w, w_csr, s, stacks=None):
        """Steps 0 .. kc-1 of the chunk starting at step k.  z_given: drive the
        synaptic recurrence with the stored spikes Z[k + t] (recomputation)."""
        B, n = self.Vs.shape[1:]
        if self.Pc is not None:
            L.check(L.lib().bt_input_project(kc * B, xin.shape[-1], n, xin[k:k + kc].data_ptr(), w_t.data_ptr(),
                                             L.ptr(bias), self.Pc.data_ptr(), self.pw.data_ptr(), s),
                    "bt_input_project")
            P = self.Pc
        else:
            P = xin[k:k + kc]
        ptr = lambda A, t: None if A is None else A[t].data_ptr()  # noqa: E731
        for t in range(kc):
            torch.add(self.Ps[t], P[t], out=self.I[t])
            zt = self.zr if z_given else Z[k + t]
            L.check(L.lib().bt_neuron_step(d, B, n, self.I[t].data_ptr(), self.Vs[t].data_ptr(), ptr(self.REFs, t),
                                           ptr(self.GKs, t), self.Vs[t + 1].data_ptr(), ptr(self.REFs, t + 1),
                                           ptr(self.GKs, t + 1), zt.data_ptr(), self.U[t].data_ptr(),
                                           self.M[t].data_ptr(), self.VCH[t].data_ptr(), s), "bt_neuron_step")
            wz = _spmv(direction, lay, Z[k + t], w, w_csr)
            L.check(L.lib().bt_psc_step(B, n, L.param(coef), L.param(tau), self.Ps[t].data_ptr(), wz.data_ptr(),
                                        self.Ps[t + 1].data_ptr(), s), "bt_psc_step")
            if stacks is not None:
                for kind, A in (("v", self.Vs), ("psc", self.Ps), ("gk", self.GKs), ("ref", self.REFs)):
                    if stacks.get(kind) is not None:
                        stacks[kind][k + t].copy_(A[t + 1])

    def roll(self, kc):
        """The chunk's last state becomes the next chunk's first."""
        for A in (self.Vs, self.Ps, self.GKs, self.REFs):
            if A is not None:
                A[0].copy_(A[kc])


def native_steps(rnn, B: int, n: int, direction: str) -> bool:
    """The engine and the native backward run this call (else the single-step
    kernels do): a spiking forward within the engine's limits."""
    if not getattr(rnn.neuron.surrogate_function, "spiking", True) or n >= 1 << 25:
        return False
    return B <= (256 if direction != "gather" else 12288) and B * n < 1 << 31


class _Run:
    """The engine as the forward of a BPTT call: scatter or ordered (a warp per
    neuron, "gather", or a lane, "pull"), one delay bin, state in this object's
    own [B][n] buffers, successive `steps` calls continuing one run."""

    def __init__(self, neuron, d, psc_mod, coef, tau, lay, direction, w, B, n, v, psc, gk, ref):
        dev = w.device
        new = lambda *shape: torch.empty(shape, device=dev, dtype=torch.float32)  # noqa: E731
        self.v, self.psc = new(B, n), new(B, n)
        self.gk = new(B, n) if gk is not None else None
        self.ref = new(B, n) if ref is not None else None
        self.load(v, psc, gk, ref)
        self.B, self.n, self.dev = B, n, dev
        e = self.desc = L.BtEngineDesc()
        self.keep = [coef, tau, w, lay]
        e.neuron, e.psc_coef, e.psc_tau = d, L.param(coef), L.param(tau)
        vals = scalar_values([coef, psc_mod.tau_syn])
        if vals is not None:
            e.psc_uniform, e.psc_coef_s, e.psc_tau_s = 1, vals[0], vals[1]
            ok, r = _ops.fast_division(vals[1], psc_mod.tau_syn.device)
            e.psc_fast_div, e.psc_rcp = int(ok), r
        e.n, e.batch, e.n_bins, e.n_rec, e.hist_len, e.t0 = n, B, 1, 1, 3, 3
        e.v, e.psc, e.g_k, e.refractory = self.v.data_ptr(), self.psc.data_ptr(), L.ptr(self.gk), L.ptr(self.ref)
        hist = torch.zeros((3, B, (n + 31) // 32), device=dev, dtype=torch.int32)
        e.hist = hist.data_ptr()
        self.keep.append(hist)
        self.ordered = direction in ("gather", "pull")
        if direction == "pull":
            e.mode = L.BT_MODE_PULL
            sl = getattr(lay, "slices", None)
            if sl is None:
                sl = lay.slices = _ops.build_slices(lay, dev)
            sl_w = _ops.pack_slice_weights(sl, w)
            masks = torch.zeros((3, n + 1, L.lib().bt_mask_stride(B)), device=dev, dtype=torch.int32)
            self.keep += [sl, sl_w, masks]
            e.sl_ptr, e.sl_src, e.sl_w = sl.sl_ptr.data_ptr(), sl.sl_src.data_ptr(), sl_w.data_ptr()
            e.masks = masks.data_ptr()
            return
        if direction == "gather":
            e.mode = L.BT_MODE_GATHER
            e.csc_ptr, e.csc_src, e.csc_w = lay.csc_ptr.data_ptr(), lay.csc_src.data_ptr(), w.data_ptr()
            return
        e.mode = L.BT_MODE_SCATTER
        edges = pack_edges(lay, w)
        ring = new(B, n)
        work = torch.empty(L.lib().bt_engine_work_words(n, B, 1), device=dev, dtype=torch.int32)
        self.keep += [edges, ring, work]
        e.csr_ptr, e.csr_edges = lay.csr_ptr.data_ptr(), edges.data_ptr()
        e.ring, e.work = ring.data_ptr(), work.data_ptr()
        rows = max(1, lay.csr_ptr.numel() - 1)
        e.scatter_lanes = 1 if lay.nnz < 48 * rows else 32
        L.check(L.lib().bt_engine_prime(CT.byref(e), L.stream_of(dev)), "bt_engine_prime")

    def load(self, v, psc, gk, ref):
        self.v.copy_(v)
        self.psc.copy_(psc)
        if self.gk is not None:
            self.gk.copy_(gk)
        if self.ref is not None:
            self.ref.copy_(ref)

    def steps(self, x, kc, s, spikes=None, given=None, v=None, psc=None, gk=None, ref=None):
        """kc steps on the drive x [kc][B][n]; spikes and state traces into the
        given [kc][B][n] tensors.  given: the spikes that drive the recurrence
        (a scatter's sums may round differently than in the first run; the
        ordered gather's cannot)."""
        e = self.desc
        e.x, e.n_steps, e.spikes = x.data_ptr(), kc, L.ptr(spikes)
        e.v_trace, e.psc_trace, e.gk_trace, e.ref_trace = L.ptr(v), L.ptr(psc), L.ptr(gk), L.ptr(ref)
        if given is not None and not self.ordered:
            L.check(L.lib().bt_engine_run_given(CT.byref(e), given.data_ptr(), s), "bt_engine_run_given")
        else:
            L.check(L.lib().bt_engine_run(CT.byref(e), s), "bt_engine_run")
        e.t0 += kc


class _Traces:
    """State before the first and after every step of a chunk ([Cb + 1][B][n]),
    and the chunk's projected drive."""

    def __init__(self, B, n, Cb, has_gk, has_ref, proj, c_in, dev):
        new = lambda *shape: torch.empty(shape, device=dev, dtype=torch.float32)  # noqa: E731
        self.V, self.P = new(Cb + 1, B, n), new(Cb + 1, B, n)
        self.GK = new(Cb + 1, B, n) if has_gk else None
        self.REF = new(Cb + 1, B, n) if has_ref else None
        self.x = new(Cb, B, n) if proj else None
        self.pw = _projection_scratch(Cb, B, c_in, dev) if proj else None

    def start(self, run):
        for A, t in ((self.V, run.v), (self.P, run.psc), (self.GK, run.gk), (self.REF, run.ref)):
            if A is not None:
                A[0].copy_(t)

    def into(self):
        return {"v": self.V[1:], "psc": self.P[1:], "gk": self.GK[1:] if self.GK is not None else None,
                "ref": self.REF[1:] if self.REF is not None else None}


def _projection_scratch(steps, B, c_in, dev):
    return torch.empty(max(1, steps * B * (2 * c_in + 1)), device=dev, dtype=torch.int32)


def _drive(xin, k, kc, w_t, bias, out, pw, s):
    """The drive of steps k .. k + kc - 1: the projected input, or the input itself."""
    if out is None:
        return xin[k:k + kc]
    B, n = out.shape[1:]
    L.check(L.lib().bt_input_project(kc * B, xin.shape[-1], n, xin[k].data_ptr(), w_t.data_ptr(), L.ptr(bias),
                                     out.data_ptr(), pw.data_ptr(), s), "bt_input_project")
    return out


class _FusedBPTT(torch.autograd.Function):
    @staticmethod
    def forward(ctx, xin, w_in, b_in, mag, v0, psc0, gk0, ref0, rnn, kinds, C):
        T, B = xin.shape[:2]
        dev = xin.device
        neuron, psc_mod, conn = rnn.neuron, rnn.synapse, rnn.synapse.linear
        n = neuron.size
        proj = w_in is not None
        c_in = int(xin.shape[-1]) if proj else 0
        dt = float(environ.get("dt"))
        d, keep = neuron_desc(neuron, dt)
        coef, tau = psc_mod.coefficients(dt)
        lay = conn.layout(dev)
        direction = conn.direction(B)
        w = mag.detach().float().contiguous()
        native = native_steps(rnn, B, n, direction)
        w_csr = pack_csr_weights(lay, w) if direction != "gather" and not native else None
        w_t = w_in.detach().float().t().contiguous() if proj else None
        bias = b_in.detach().float().contiguous() if b_in is not None else None
        s = L.stream_of(dev)
        new = lambda *shape: torch.empty(shape, device=dev, dtype=torch.float32)  # noqa: E731
        n_ch = -(-T // C)
        ckpt = n_ch > 1
        Cb = C if ckpt else T
        Z = new(T, B, n)
        stacks = {kind: new(T, B, n) if kind in kinds else None for kind in ("v", "psc", "gk", "ref")}
        if gk0 is None:
            stacks["gk"] = None
        if ref0 is None:
            stacks["ref"] = None
        bounds = None
        if ckpt:
            bounds = {"v": new(n_ch, B, n), "psc": new(n_ch, B, n),
                      "gk": new(n_ch, B, n) if gk0 is not None else None,
                      "ref": new(n_ch, B, n) if ref0 is not None else None}
        if native:
            # (the engine's own choice for the ordered modes: a warp per neuron walks the
            # samples one after the other)
            engine = "pull" if direction == "gather" and B >= conn.sparse_config.pull_min_batch else direction
            run = _Run(neuron, d, psc_mod, coef, tau, lay, engine, w, B, n, v0, psc0, gk0, ref0)
            ctx.engine = engine
            st = None if ckpt else _Traces(B, n, T, gk0 is not None, ref0 is not None, proj, c_in, dev)
            out = new(Cb, B, n) if proj and ckpt else None
            pw = _projection_scratch(Cb, B, c_in, dev) if out is not None else None
            for ci in range(n_ch):
                k = ci * C
                kc = min(C, T - k)
                if ckpt:
                    for kind, t in (("v", run.v), ("psc", run.psc), ("gk", run.gk), ("ref", run.ref)):
                        if t is not None:
                            bounds[kind][ci].copy_(t)
                    at = {kind: t[k:] for kind, t in stacks.items() if t is not None}
                    run.steps(_drive(xin, k, kc, w_t, bias, out, pw, s), kc, s, spikes=Z[k:], **at)
                else:
                    st.start(run)
                    run.steps(_drive(xin, 0, T, w_t, bias, st.x, st.pw, s), T, s, spikes=Z, **st.into())
                    for kind, t in st.into().items():
                        if stacks[kind] is not None:
                            stacks[kind].copy_(t)
            last = (run.v, run.psc, run.gk, run.ref)
        else:
            st = _Steps(B, n, Cb, gk0 is not None, ref0 is not None, proj, c_in, dev)
            st.load(v0, psc0, gk0, ref0)
            for ci in range(n_ch):
                k = ci * C
                kc = min(C, T - k)
                if ckpt:
                    for kind, A in (("v", st.Vs), ("psc", st.Ps), ("gk", st.GKs), ("ref", st.REFs)):
                        if bounds[kind] is not None:
                            bounds[kind][ci].copy_(A[0])
                st.run(k, kc, xin, w_t, bias, Z, False, d, coef, tau, direction, lay, w, w_csr, s, stacks)
                if ci + 1 < n_ch:
                    st.roll(kc)
            kT = T - (n_ch - 1) * C  # steps of the last chunk
            last = tuple(A[kT].clone() if A is not None else None for A in (st.Vs, st.Ps, st.GKs, st.REFs))
        outs = [Z, stacks["v"], stacks["psc"], stacks["gk"], stacks["ref"], *last]
        # no reference to the module itself: the module's state will hold this
        # Function's outputs, and a cycle would keep the step buffers alive
        ctx.d, ctx.keep, ctx.coef, ctx.tau, ctx.lay, ctx.direction = d, keep, coef, tau, lay, direction
        ctx.detach_reset = int(bool(neuron.detach_reset))
        ctx.C, ctx.n_ch, ctx.proj, ctx.c_in = C, n_ch, proj, c_in
        ctx.has_gk, ctx.has_ref = gk0 is not None, ref0 is not None
        ctx.bias, ctx.native = bias, native
        # (the synapse and the neuron, without their states' graph: their
        # time constants, for the engine's descriptor in backward)
        ctx.tau_syn = psc_mod.tau_syn
        if ckpt:
            ctx.bounds = bounds
            ctx.steps = None  # recomputed chunk by chunk in backward
            del st
        else:
            ctx.bounds = None
            ctx.steps = st
        # saved through autograd, so they are freed after backward (unless
        # retain_graph) and Z, also returned, is checked for in-place changes
        ctx.save_for_backward(xin, w_in, mag, Z)
        ctx.set_materialize_grads(False)
        for o in (outs[4], outs[8]):
            if o is not None:
                ctx.mark_non_differentiable(o)
        return tuple(outs)

    @staticmethod
    def backward(ctx, gZ, gV, gP, gGK, _gR, gvT, gpT, ggT, _grT):
        xin, w_in, mag, Z = ctx.saved_tensors
        T, B, n = Z.shape
        dev = Z.device
        lay, d, C = ctx.lay, ctx.d, ctx.C
        s = L.stream_of(dev)
        w = mag.detach().float().contiguous()
        w_csr = _csr_weights_cached(lay, mag)
        native, ckpt = ctx.native, ctx.bounds is not None
        w_fwd = pack_csr_weights(lay, w) if ctx.direction != "gather" and not native else None
        w_t = w_in.detach().float().t().contiguous() if ctx.proj else None
        new = lambda *shape: torch.empty(shape, device=dev, dtype=torch.float32)  # noqa: E731
        st = ctx.steps
        if st is None:
            st = (_Traces if native else _Steps)(B, n, C, ctx.has_gk, ctx.has_ref, ctx.proj, ctx.c_in, dev)
        Cb = C if ckpt else T
        # dL/dpsc_t (state after step t) and dL/dI_t of one chunk; the projected
        # drive of a recomputed chunk is used up step by step as dL/dI_t is formed
        G_psc = new(Cb, B, n)
        G_I = st.x if native and ckpt and ctx.proj else new(Cb, B, n)
        gz, gT_work = new(B, n), new((B + 3) // 4 * 4 * n)
        g_psc = torch.zeros((B, n), device=dev) if gpT is None else gpT.reshape(B, n).contiguous().clone()
        cur_v = None if gvT is None else gvT.reshape(B, n).contiguous()
        cur_gk = None if (ggT is None or not ctx.has_gk) else ggT.reshape(B, n).contiguous()
        detach_reset = ctx.detach_reset
        want_mag, want_x = ctx.needs_input_grad[3], ctx.needs_input_grad[0]
        want_w, want_b = ctx.proj and ctx.needs_input_grad[1], ctx.proj and ctx.needs_input_grad[2]
        g_mag = torch.empty(lay.nnz, device=dev, dtype=torch.float32) if want_mag else None
        mag_work = torch.empty(L.lib().bt_grad_weight_work_words(Cb * B, n, 0), device=dev,
                               dtype=torch.int32) if want_mag else None
        g_wt = new(ctx.c_in, n) if want_w else None
        gw_work = torch.empty(max(1, ctx.c_in * (Cb * B + 1)), device=dev, dtype=torch.int32) if want_w else None
        g_b = torch.zeros(n, device=dev) if want_b else None
        g_x = torch.empty_like(xin) if want_x else None
        if native:
            cur_v = torch.zeros((B, n), device=dev) if cur_v is None else cur_v.clone()
            if ctx.has_gk:
                cur_gk = torch.zeros((B, n), device=dev) if cur_gk is None else cur_gk.clone()
            bd_desc = L.BtBpttDesc()
            bd_desc.batch, bd_desc.n, bd_desc.neuron = B, n, d
            bd_desc.psc_coef, bd_desc.psc_tau, bd_desc.detach_reset = L.param(ctx.coef), L.param(ctx.tau), detach_reset
            bd_desc.csr_ptr, bd_desc.csr_dst, bd_desc.csr_w = lay.csr_ptr.data_ptr(), lay.csr_dst.data_ptr(), w_csr.data_ptr()
            bd_desc.cur_psc, bd_desc.cur_v, bd_desc.cur_gk = g_psc.data_ptr(), cur_v.data_ptr(), L.ptr(cur_gk)
            bd_desc.G_psc, bd_desc.G_I, bd_desc.gz, bd_desc.gT = (t.data_ptr() for t in (G_psc, G_I, gz, gT_work))
            stack_grads = [g.contiguous() if g is not None else None for g in (gZ, gV, gP, gGK if ctx.has_gk else None)]
            run = None
        else:
            g_v = [new(B, n), new(B, n)]
            g_gk = [new(B, n), new(B, n)] if ctx.has_gk else None
        for ci in reversed(range(ctx.n_ch)):
            k = ci * C
            kc = min(C, T - k)
            if native:
                if ckpt:
                    start = [t[ci] if t is not None else None for t in map(ctx.bounds.get, ("v", "psc", "gk", "ref"))]
                    if run is None:
                        run = _Run(None, d, ctx, ctx.coef, ctx.tau, lay, ctx.engine, w, B, n, *start)
                    else:
                        run.load(*start)
                    st.start(run)
                    x = _drive(xin, k, kc, w_t, ctx.bias, st.x, st.pw, s)
                    run.steps(x, kc, s, given=Z[k:], **st.into())
                else:
                    x = st.x if ctx.proj else xin
                bd_desc.n_steps, bd_desc.x, bd_desc.z = kc, x.data_ptr(), Z[k].data_ptr()
                bd_desc.v, bd_desc.psc = st.V.data_ptr(), st.P.data_ptr()
                bd_desc.ref, bd_desc.gk = L.ptr(st.REF), L.ptr(st.GK)
                bd_desc.g_z, bd_desc.g_v, bd_desc.g_psc, bd_desc.g_gk = (g[k].data_ptr() if g is not None else None
                                                                         for g in stack_grads)
                L.check(L.lib().bt_bptt_backward(CT.byref(bd_desc), s), "bt_bptt_backward")
            elif ctx.bounds is not None:
                bd = ctx.bounds
                st.load(bd["v"][ci], bd["psc"][ci], bd["gk"][ci] if bd["gk"] is not None else None,
                        bd["ref"][ci] if bd["ref"] is not None else None)
                st.run(k, kc, xin, w_t, ctx.bias, Z, True, d, ctx.coef, ctx.tau, ctx.direction, lay, w, w_fwd, s)
            for tl in reversed(range(kc)) if not native else ():
                t = k + tl
                gp = G_psc[tl]
                torch.add(g_psc, gP[t], out=gp) if gP is not None else gp.copy_(g_psc)
                if gV is not None:
                    cur_v = gV[t] if cur_v is None else cur_v + gV[t]
                if gGK is not None and ctx.has_gk:
                    cur_gk = gGK[t] if cur_gk is None else cur_gk + gGK[t]
                L.check(L.lib().bt_spmv_grad_input_pad(B, n, n, lay.csr_ptr.data_ptr(), lay.csr_dst.data_ptr(),
                                                       w_csr.data_ptr(), gp.data_ptr(), gz.data_ptr(),
                                                       gT_work.data_ptr(), s), "bt_spmv_grad_input_pad")
                if gZ is not None:
                    gz.add_(gZ[t])
                out_v = g_v[tl & 1]
                out_gk = g_gk[tl & 1] if g_gk is not None else None
                L.check(L.lib().bt_neuron_step_backward(
                    d, B, n, st.I[tl].data_ptr(), gz.data_ptr(), L.ptr(cur_v), L.ptr(cur_gk), st.U[tl].data_ptr(),
                    Z[t].data_ptr(), st.M[tl].data_ptr(), st.VCH[tl].data_ptr(), st.Vs[tl].data_ptr(),
                    st.GKs[tl].data_ptr() if st.GKs is not None else None, G_I[tl].data_ptr(), out_v.data_ptr(),
                    L.ptr(out_gk), detach_reset, s), "bt_neuron_step_backward")
                # dpsc_{t-1} = dpsc_t + coef*((-dpsc_t)/tau) + dI_t
                nxt = torch.empty_like(g_psc)
                L.check(L.lib().bt_psc_step(B, n, L.param(ctx.coef), L.param(ctx.tau), gp.data_ptr(),
                                            G_I[tl].data_ptr(), nxt.data_ptr(), s), "bt_psc_step")
                # step t - 1 reads what step t wrote and writes the other buffer of
                # each pair (one stream: the kernels run in order); the pair
                # parity restarts per chunk, so copy out of the pair first
                g_psc, cur_v, cur_gk = nxt, out_v, out_gk
            if not native:
                cur_v = cur_v.clone() if cur_v is not None else None
                cur_gk = cur_gk.clone() if cur_gk is not None else None
            rows = kc * B
            if want_mag:
                L.check(L.lib().bt_spmv_grad_weight_rows(rows, n, n, lay.csc_ptr.data_ptr(), lay.csc_src.data_ptr(),
                                                         Z[k].data_ptr(), G_psc.data_ptr(), g_mag.data_ptr(),
                                                         int(ci != ctx.n_ch - 1), 0, mag_work.data_ptr(), s),
                        "bt_spmv_grad_weight_rows")
            if want_w:
                L.check(L.lib().bt_input_grad_weight(rows, ctx.c_in, n, xin[k].data_ptr(), G_I.data_ptr(),
                                                     g_wt.data_ptr(), int(ci != ctx.n_ch - 1), gw_work.data_ptr(),
                                                     s), "bt_input_grad_weight")
            if want_b:
                g_b.add_(G_I[:kc].sum(dim=(0, 1)))
            if want_x:
                gi = G_I[:kc]
                # the input's own gradient (data rarely needs one): a plain GEMM
                g_x[k:k + kc] = (gi.reshape(rows, n) @ w_in.detach().float()).reshape(kc, B, -1) if ctx.proj else gi
        g_w = g_wt.t().contiguous().to(w_in.dtype) if want_w else None
        if g_mag is not None:
            g_mag = g_mag.to(mag.dtype)
        return g_x, g_w, g_b, g_mag, cur_v, g_psc, cur_gk, None, None, None, None


def _bytes_needed(T, B, n, C, kinds, has_gk, has_ref, proj, c_in, native, nnz=0):
    """Device bytes of the call's buffers (spikes, stacks, step buffers,
    chunk-start states, gradients of one chunk, the weight gradient's row
    lists, the edges packed for the forward and the backward)."""
    n_ch = -(-T // C)
    ckpt = n_ch > 1
    Cb = C if ckpt else T
    states = 2 + int(has_gk) + int(has_ref)
    per = T * (1 + len(kinds))  # spikes + requested stacks
    per += states * (Cb + 1) + (Cb if proj else 0)  # states of every step, projected drive
    per += 0 if native else 4 * Cb  # I, u, mask, v_charged
    per += states * (n_ch if ckpt else 0)  # chunk-start states
    per += Cb if native and ckpt and proj else 2 * Cb  # gradients of a chunk (dI over its drive)
    lists = L.lib().bt_grad_weight_work_words(Cb * B, n, 0)
    return 4 * (B * n * per + (Cb * B * (2 * c_in + 1) if proj else 0) + lists + 3 * nnz)


def run(rnn, x: torch.Tensor, paths: dict):
    """One call through the fused BPTT, or None when its buffers would not
    fit (the caller then steps module by module)."""
    neuron, syn = rnn.neuron, rnn.synapse
    n = neuron.size
    inp = rnn.neuron_inp_module
    T = x.shape[0]
    v = neuron.v
    B = v.numel() // n
    if inp is not None:
        c_in = inp.in_features
        if x.shape[-1] != c_in:
            raise RuntimeError(f"RecurrentNN input has shape {tuple(x.shape)}; its input layer takes {c_in} channels.")
        xin = torch.broadcast_to(x.reshape(T, -1, c_in), (T, B, c_in)).float().contiguous()
        w_in, b_in = inp.weight, inp.bias
    else:
        c_in = 0
        xin = torch.broadcast_to(x.reshape(T, -1, n), (T, B, n)).float().contiguous()
        w_in = b_in = None
    C = checkpoint_chunk(rnn, T)
    kinds = frozenset(paths.values())
    need = _bytes_needed(T, B, n, C, kinds, isinstance(neuron, ALIF), neuron._use_refractory, inp is not None, c_in,
                         native_steps(rnn, B, n, syn.linear.direction(B)), int(syn.linear.indices.shape[1]))
    if not fits(x.device, need):
        return None
    shape = v.shape
    v0 = v.reshape(B, n)
    psc0 = syn.psc.reshape(B, n)
    gk0 = neuron.g_k.reshape(B, n) if isinstance(neuron, ALIF) else None
    ref0 = neuron.refractory.reshape(B, n).detach() if neuron._use_refractory else None
    syn.linear._edge_weight()  # one weight per stored nonzero, or an error before any launch
    try:
        outs = _FusedBPTT.apply(xin, w_in, b_in, syn.linear.magnitude, v0, psc0, gk0, ref0, rnn, kinds, C)
    except torch.OutOfMemoryError:  # (the free memory was less than the figure; no state has changed)
        _FREE.pop(x.device, None)
        return None
    Z, Vst, Pst, GKst, REFst, vT, pT, gT, rT = outs
    neuron.v = vT.reshape(shape)
    syn.psc = pT.reshape(syn.psc.shape)
    if gT is not None:
        neuron.g_k = gT.reshape(shape)
    if rT is not None:
        neuron.refractory = rT.reshape(shape)
    stacks = {"v": Vst, "psc": Pst, "gk": GKst, "ref": REFst}
    states = {key: stacks[kind].reshape(T, *shape) for key, kind in paths.items()}
    rnn.last_path = "fused-bptt"
    rnn.last_bptt = {"chunk": C, "recomputed": C < T, "bytes": need}
    return Z.reshape(T, *shape), states


__all__ = ["match", "run", "checkpoint_chunk"]
