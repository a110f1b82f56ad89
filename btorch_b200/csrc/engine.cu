// Fused multi-step recurrent engine: RecurrentNN(neuron, synapse, inp) for
// LIF/ALIF neurons with exponential (optionally delayed) synapses on a sparse
// connectivity, btorch/models/rnn.py:517-528 repeated over time
// (rnn.py:200-332).
//
// Reference step t (per sample b, neuron i):
//   I     = psc_{t-1} + x_t                     (rnn.py:524)
//   z_t   = neuron(I)                           (base.py:1108-1116)
//   psc_t = decay(psc_{t-1}) + sum_d W_d z_{t-d} (synapse.py:99-103, delay bins
//                                                 via history.py:299-345 and
//                                                 connection.py:973-1027)
//
// SCATTER mode, two launches per step:
//   k_eng_neuron  (step t): P = stored + acc; zero acc; neuron update with
//                 I = P + x_t; stored = decay(P); spike bitmaps; the step's
//                 spike set: a mask of spiking samples per neuron and the
//                 compacted list of neurons that spiked in any sample (warp
//                 ballot + one warp-aggregated atomic on one of 64 counters).
//   k_eng_scatter (step t): for every delay bin d and every neuron j in the
//                 spike set of step t - d, stream the out-edges of row
//                 j * R + d of the delay-expanded matrix with 128-bit loads
//                 and add w into acc[b][post] for every sample b in j's mask
//                 (fp32 reductions, resolved in L2: acc is [B][n], the size
//                 of one state variable, whatever the delay range).
//   The spike sets of the last R steps live in a ring of R + 1 slots (slot =
//   step mod (R + 1)) in the scratch; the last reader of a set clears it.
//   "stored" holds decay(psc_{t-1}) during a run and acc the sum W z of the
//   step, so the reference's rounding of psc = decay(psc) + Wz is kept
//   (exact sums when weights are dyadic).
//
// GATHER mode, one launch per step (k_eng_gather): each warp owns a neuron,
//   computes P_{t-1} = decay(P_{t-2}) + sum over its in-edges (pre, bin) in
//   ascending canonical order of w * z_{t-1-bin}[pre] (fmaf chain, exactly the
//   reference's CPU rounding), then runs the neuron update of step t.  The
//   last synapse update of a run is k_eng_gather_final.
//
// RECEPTOR CHANNELS (HeterSynapsePSC with n_receptor = C > 1,
// synapse.py:626-847): the matrix has C columns per neuron (post * C + r, the
// layout make_hetersynapse_conn builds, connection.py:218-587); PSC state,
// acc and the PSC coefficients are [batch][n * C], and the neuron's input is
// the receptor sum of its C channels (receptor_sum, the reference's
// psc.reshape(..., n, C).sum(-1) rounding).  Scatter and gather modes.
#include <algorithm>
#include <climits>
#include <cstring>
#include <type_traits>

#include "neuron.cuh"

namespace bt {

constexpr int kEngThreads = 256;
constexpr int kMaxRec = 16;  // receptor channels per neuron

// Receptor columns per neuron (0 in the descriptor means 1).
__host__ __device__ __forceinline__ int n_rec(const bt_engine_desc& d) { return d.n_rec > 1 ? d.n_rec : 1; }

// Sum of one neuron's C receptor PSCs p[0..C) in the order torch's CPU sum
// reduces a contiguous row of C floats, which the reference runs as
// psc.reshape(..., n, C).sum(-1) (synapse.py:744-747):
//   C < 4       left to right;
//   4 <= C < 8  a_j = p_j (j < 4), p_4 .. p_{C-1} added to a_0 in turn, then
//               ((a_0 + a_1) + a_2) + a_3;
//   C >= 8      a_j = p_j + p_{8+j} + ... over the whole groups of 8, the
//               left-to-right sum of the remaining tail added to a_0, then
//               a_0 + a_1 + ... + a_7 left to right.
// (Established against torch.sum for every C up to 39; the host mirror in
// btorch_b200/models/synapse.py is checked against torch.sum in the CPU
// tests.)  p holds M >= C values; indices are compile-time after unrolling.
template <int M>
__device__ __forceinline__ float receptor_sum(const float (&p)[M], int C) {
  if (C < 4 || M < 4) {
    float s = p[0];
#pragma unroll
    for (int r = 1; r < 4 && r < M; ++r)
      if (r < C) s = add(s, p[r]);
    return s;
  }
  if constexpr (M >= 4) {
    if (C < 8 || M < 8) {
      float a0 = p[0];
#pragma unroll
      for (int r = 4; r < 8 && r < M; ++r)
        if (r < C) a0 = add(a0, p[r]);
      return add(add(add(a0, p[1]), p[2]), p[3]);
    }
  }
  if constexpr (M >= 8) {
    const int full = C & ~7;
    float a[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] = p[j];
#pragma unroll
    for (int r = 8; r < M; ++r)
      if (r < full) a[r & 7] = add(a[r & 7], p[r]);
    if (full < C) {
      float t = 0.0f;
      bool first = true;
#pragma unroll
      for (int r = 8; r < M; ++r)
        if (r >= full && r < C) {
          t = first ? p[r] : add(t, p[r]);
          first = false;
        }
      a[0] = add(a[0], t);
    }
    float s = a[0];
#pragma unroll
    for (int j = 1; j < 8; ++j) s = add(s, a[j]);
    return s;
  }
  return p[0];  // not reached: C <= M
}

__host__ __device__ __forceinline__ int mask_words(int64_t batch) { return int((batch + 31) >> 5); }

// Words per neuron in the pull engine's sample masks: the word count rounded up
// to the vector width the kernel loads with (1, 2 or 4 words), unchanged above 4.
__host__ __device__ __forceinline__ int mask_stride(int64_t batch) {
  const int mw = mask_words(batch);
  return mw <= 1 ? 1 : mw <= 2 ? 2 : mw <= 4 ? 4 : mw;
}

// Slot indices of one step, computed on the host per launch so that no kernel
// evaluates a 64-bit modulo per element.
struct StepIdx {
  int q_t;     // t mod (R + 1): spike-set slot of step t (scatter)
  int h_t;     // t mod H:       history slot written at step t
  int h_prev;  // (t - 1) mod H: history slot of step t - 1
};

inline StepIdx step_idx(int64_t t, int R, int H) {
  StepIdx s;
  s.q_t = int(t % (R + 1));
  s.h_t = int(t % H);
  s.h_prev = int((t - 1) % H);
  return s;
}

// ---------------------------------------------------------------- scatter --

// Scatter-mode scratch (d.work, int32 words), Q = R + 1 spike-set slots:
//   [0, 2*Q*kSub)                  active-list counts and spike totals,
//                                  [slot][count | spikes][sub-list]
//   next Q*n                       "listed" flags, [slot][neuron]
//   next Q*kSub*cap                list entries, [slot][sub-list][cap]
//   next Q n S                     sample masks, [slot][neuron][S words], S = mask_stride(batch)
//   next kSub                      control words (ctrl[0]: blocks done with a dense step)
// Sub-list s only lists neurons [s*cap, (s+1)*cap) and each neuron is listed at
// most once per step (its flag), so a sub-list never holds more than cap
// entries.  cap is a multiple of 32, so the 32 neurons of a warp share one
// sub-list.
constexpr int kSub = 64;
// Dense delivery needs at least this many spiking samples per listed neuron on
// average: below it the per-event reductions of the list path are cheaper
// than the dense pull's random mask reads (measured crossover about 2.5).
constexpr int kDenseSpikesPerRow = 3;

// A power of two (>= 32), so the sub-list of neuron i is i >> log2(cap).
__host__ __device__ __forceinline__ int64_t sub_cap(int64_t n) {
  const int64_t c = (n + kSub - 1) / kSub;
  int64_t p = 32;
  while (p < c) p <<= 1;
  return p;
}

__host__ __device__ __forceinline__ int64_t scatter_work_words(int64_t n, int64_t batch, int n_bins) {
  const int64_t Q = int64_t(n_bins) + 1;
  return Q * (2 * kSub + n + kSub * sub_cap(n) + n * mask_stride(batch)) + kSub;
}

struct ScatterScratch {
  int32_t* count;
  int32_t* spk;   // spikes (sample-neuron pairs) listed per sub-list
  int32_t* flag;
  int32_t* list;
  uint32_t* mask;
  int32_t* ctrl;
  int64_t cap;
  int cap_shift;  // log2(cap)
  int ms;
};

__host__ __device__ __forceinline__ int log2_pow2(int64_t c) {
  int s = 0;
  while ((int64_t(1) << s) < c) ++s;
  return s;
}

__host__ __device__ __forceinline__ ScatterScratch scatter_scratch(const bt_engine_desc& d, int q) {
  ScatterScratch w;
  const int64_t n = d.n;
  const int64_t Q = int64_t(d.n_bins) + 1;
  w.ms = mask_stride(d.batch);
  w.cap = sub_cap(n);
  w.cap_shift = log2_pow2(w.cap);
  w.count = d.work + q * 2 * kSub;
  w.spk = w.count + kSub;
  w.flag = d.work + Q * 2 * kSub + q * n;
  w.list = d.work + Q * 2 * kSub + Q * n + q * kSub * w.cap;
  w.mask = reinterpret_cast<uint32_t*>(d.work + Q * 2 * kSub + Q * n + Q * kSub * w.cap) + int64_t(q) * n * w.ms;
  w.ctrl = d.work + Q * (2 * kSub + n + kSub * w.cap + n * w.ms);
  return w;
}

// Publish neuron i's spikes of step t in the step's spike set `ws` (bit u of
// `spiked`: sample b0 + u): the samples' bits in the neuron's mask -- one
// atomic, the S samples lie in one 32-sample word (b0 % S == 0, S | 32) --
// and the neuron in the compacted list if this warp's samples are the first
// to spike (one warp-aggregated atomic on one of kSub counters).  Called by
// every lane of the warp.
__device__ __forceinline__ void publish_spikes_ws(const ScatterScratch& ws, int i, int b0, uint32_t spiked) {
  if (__ballot_sync(0xffffffffu, spiked != 0) == 0) return;  // warp-uniform
  const unsigned lane = lane_id();
  bool first = false;
  if (spiked) {
    atomicOr(ws.mask + int64_t(i) * ws.ms + (b0 >> 5), spiked << (b0 & 31));
    first = atomicOr(ws.flag + i, 1) == 0;
  }
  const uint32_t fb = __ballot_sync(0xffffffffu, first);
  const int sub = (i - int(lane)) >> ws.cap_shift;  // same for the whole warp (cap % 32 == 0)
  const int nspk = __reduce_add_sync(0xffffffffu, unsigned(__popc(spiked)));
  if (lane == 0 && nspk) atomicAdd(ws.spk + sub, nspk);
  if (fb == 0) return;
  int32_t base = 0;
  if (lane == 0) base = atomicAdd(ws.count + sub, __popc(fb));
  base = __shfl_sync(0xffffffffu, base, 0);
  if (first) ws.list[int64_t(sub) * ws.cap + base + __popc(fb & ((1u << lane) - 1u))] = i;
}

// The same for a kernel that derives the spike set from the descriptor.
template <int S>
__device__ __forceinline__ void publish_spikes(const bt_engine_desc& d, const StepIdx& si, int64_t i, int64_t b0,
                                               uint32_t spiked) {
  if (__ballot_sync(0xffffffffu, spiked != 0) == 0) return;  // warp-uniform
  const unsigned lane = lane_id();
  const ScatterScratch ws = scatter_scratch(d, si.q_t);
  bool first = false;
  if (spiked) {
    uint32_t* mrow = ws.mask + i * ws.ms;
#pragma unroll
    for (int u = 0; u < S; ++u)
      if (spiked & (1u << u)) atomicOr(mrow + ((b0 + u) >> 5), 1u << ((b0 + u) & 31));
    first = atomicOr(ws.flag + i, 1) == 0;
  }
  const uint32_t fb = __ballot_sync(0xffffffffu, first);
  const int sub = int((i - lane) >> ws.cap_shift);  // same for the whole warp (cap % 32 == 0)
  const int nspk = __reduce_add_sync(0xffffffffu, unsigned(__popc(spiked)));
  if (lane == 0 && nspk) atomicAdd(ws.spk + sub, nspk);
  if (fb == 0) return;
  int32_t base = 0;
  if (lane == 0) base = atomicAdd(ws.count + sub, __popc(fb));
  base = __shfl_sync(0xffffffffu, base, 0);
  if (first) ws.list[sub * ws.cap + base + __popc(fb & ((1u << lane) - 1u))] = int32_t(i);
}

// Grid (ceil(n / 256), ceil(batch / S)): a thread owns neuron i for S
// consecutive samples; a warp covers one 32-neuron bitmap word of each of
// them.  All S samples' state is loaded before any is updated (memory-level
// parallelism), and the neuron's parameters are read once for the S samples.
// `ws` is the step's spike set, its pointers computed on the host; indices
// are 32-bit (batch * n < 2^31 in scatter mode, checked on the host) except
// into the per-step input and trace arrays.
template <int KIND, bool HARD, bool USE_REF, int S, bool FAST>
__global__ void __launch_bounds__(kEngThreads) k_eng_neuron(bt_engine_desc d, int k, StepIdx si, ScatterScratch ws,
                                                          const float* __restrict__ z_given) {
  step_wait();
  const int n = int(d.n), B = int(d.batch);
  const int words = (n + 31) >> 5;
  const int i = int(blockIdx.x) * kEngThreads + int(threadIdx.x);
  const int b0 = int(blockIdx.y) * S;
  if ((i & ~31) >= n) return;  // whole warps past the last word
  const bool valid = i < n;
  const int nb = B - b0 < S ? B - b0 : S;  // samples of this block (uniform)
  const int off0 = b0 * n + (valid ? i : 0);
  float* ring_p = d.ring + off0;  // acc: W z of the previous step
  float* psc_p = d.psc + off0;
  float* v_p = d.v + off0;
  float* ref_p = USE_REF ? d.refractory + off0 : nullptr;
  float* gk_p = KIND == BT_NEURON_ALIF ? d.g_k + off0 : nullptr;
  const float* x_p = d.x ? d.x + int64_t(k) * B * n + off0 : nullptr;
  const uint64_t pol_stream = l2_evict_first(), pol_keep = l2_evict_last();
  // Every load before the first store: a load behind a store through a
  // pointer that may alias it waits for the store.  A sample past its length
  // (k > len) reads and writes no state unless state traces are requested:
  // its state is frozen and its accumulator is not read again in this call.
  const bool traces = d.v_trace || d.psc_trace || d.ref_trace || d.gk_trace || d.spikes;
  const bool st_traces = d.v_trace || d.psc_trace || d.ref_trace || d.gk_trace;
  float pend[S], pv[S], xv[S], vv[S], rv[S], gv[S];
  int lenv[S];
#pragma unroll
  for (int u = 0; u < S; ++u) lenv[u] = (valid && u < nb && d.sample_len) ? d.sample_len[b0 + u] : INT_MAX;
#pragma unroll
  for (int u = 0; u < S; ++u) {
    const bool in = valid && u < nb;
    const bool live = in && k < lenv[u], edge = in && k <= lenv[u], frozen = in && st_traces;
    const int o = u * n;
    pend[u] = edge ? ld_f32(ring_p + o, pol_keep) : 0.0f;
    pv[u] = (edge || frozen) ? psc_p[o] : 0.0f;
    xv[u] = (live && x_p) ? ld_nc_f32(x_p + o, pol_stream) : 0.0f;
    vv[u] = (live || frozen) ? v_p[o] : 0.0f;
    rv[u] = ((live || frozen) && USE_REF) ? ref_p[o] : 0.0f;
    gv[u] = ((live || frozen) && KIND == BT_NEURON_ALIF) ? gk_p[o] : 0.0f;
  }
  const int ip = valid ? i : 0;
  const NeuronParams prm = load_params<KIND, USE_REF>(d.neuron, ip);
  const float pc = d.psc_uniform ? d.psc_coef_s : ld(d.psc_coef, ip);
  const float pt = d.psc_uniform ? d.psc_tau_s : ld(d.psc_tau, ip);
  const Div dpt = make_div(pt, d.psc_uniform && d.psc_fast_div, d.psc_rcp);
  const unsigned lane = lane_id();
  uint32_t* hist_p = d.hist + (int64_t(si.h_t) * B + b0) * words + (i >> 5);
  uint32_t* raster_p = d.raster ? d.raster + (int64_t(k) * B + b0) * words + (i >> 5) : nullptr;
  uint32_t spiked = 0;  // bit u: spiked in sample b0 + u
#pragma unroll
  for (int u = 0; u < S; ++u) {
    if (u >= nb) break;  // uniform across the block
    const int o = u * n;
    float s = 0.0f;
    if (valid) {
      const int len = lenv[u];
      if (k <= len) st_f32(ring_p + o, 0.0f, pol_keep);
      float v = vv[u], ref = rv[u], gk = gv[u];
      float P;
      if (k < len) {
        P = add(pv[u], pend[u]);
        const float I = x_p ? add(P, xv[u]) : P;
        const NeuronOut out = neuron_update<KIND, HARD, USE_REF, true, FAST>(prm, I, v, ref, gk);
        s = out.spike;
        v_p[o] = v;
        if (USE_REF) ref_p[o] = ref;
        if (KIND == BT_NEURON_ALIF) gk_p[o] = gk;
        psc_p[o] = psc_decay_k<FAST>(pc, dpt, P);
      } else {
        // Finished sample: its state freezes at its last step.  On the first
        // step past the end the pending sum completes psc of that last step;
        // later arrivals are dropped.
        P = pv[u];
        if (k == len) {
          P = add(P, pend[u]);
          psc_p[o] = P;
        }
      }
      if (traces) {
        const int64_t tix = (int64_t(k) * B + b0 + u) * n + i;
        if (d.psc_trace && k > 0) d.psc_trace[tix - int64_t(B) * n] = P;
        if (d.v_trace) d.v_trace[tix] = v;
        if (USE_REF && d.ref_trace) d.ref_trace[tix] = ref;
        if (KIND == BT_NEURON_ALIF && d.gk_trace) d.gk_trace[tix] = gk;
        if (d.spikes) d.spikes[tix] = s;
      }
    }
    const uint32_t word = __ballot_sync(0xffffffffu, s != 0.0f);
    if (lane == 0) {
      hist_p[u * words] = word;
      if (raster_p) raster_p[u * words] = word;
    }
    // z_given: publish these spikes instead of the step's own
    if (z_given && valid) s = z_given[(int64_t(k) * B + b0 + u) * n + i];
    if (s != 0.0f) spiked |= 1u << u;
  }
  publish_spikes_ws(ws, i, b0, spiked);
}

// x / d for 4 values by a divisor of kind 1 or 2 (divk<true>, bit for bit): one
// uniform branch on the kind and one on the rare cases for the four of them.  A
// zero takes the fast path (its quotient is x r, sign included): silent synapses
// and freshly reset neurons are in every warp, and the out-of-line path for one
// lane costs the whole warp.
__device__ __forceinline__ void divk4(const float (&x)[4], const Div& d, float (&out)[4]) {
  if (d.kind == 1) {
#pragma unroll
    for (int q = 0; q < 4; ++q) out[q] = mul(x[q], d.r);
    return;
  }
  bool rare = false;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float y = mul(x[q], d.r), ay = fabsf(y);
    const float e = __fmaf_rn(-y, d.c, x[q]);
    out[q] = x[q] == 0.0f ? y : __fmaf_rn(e, d.r, y);
    rare |= !(ay >= 0x1p-100f && ay <= 0x1p100f) && x[q] != 0.0f;
  }
  if (rare) {
#pragma unroll
    for (int q = 0; q < 4; ++q) out[q] = div_recip(x[q], d.c, d.r);
  }
}

// neuron_update<KIND, HARD, USE_REF, true, true> for 4 neurons with the same
// (scalar) parameters, the same operations in the same order per neuron.
template <int KIND, bool HARD, bool USE_REF>
__device__ __forceinline__ void neuron_update4(const NeuronParams& pr, const float (&I)[4], float (&v)[4], float (&ref)[4],
                                               float (&gk)[4], float (&s)[4]) {
  float v1[4], t[4], a[4], b[4];
  if (KIND == BT_NEURON_LIF) {
#pragma unroll
    for (int q = 0; q < 4; ++q) t[q] = -sub(v[q], pr.vr);
    divk4(t, pr.d_tau, a);
    divk4(I, pr.d_cm, b);
#pragma unroll
    for (int q = 0; q < 4; ++q) v1[q] = add(v[q], mul(pr.dt, add(a[q], b[q])));
  } else {
#pragma unroll
    for (int q = 0; q < 4; ++q)
      t[q] = add(add(mul(pr.ngl, sub(v[q], pr.El)), mul(-gk[q], sub(v[q], pr.Ek))), I[q]);
    divk4(t, pr.d_cm, a);  // derivative
#pragma unroll
    for (int q = 0; q < 4; ++q) t[q] = sub(pr.ngl, gk[q]);
    divk4(t, pr.d_cm, b);  // linear
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float coef = div(expm1f(mul(pr.dt, b[q])), b[q]);
      v1[q] = add(v[q], mul(coef, a[q]));
      t[q] = -gk[q];
    }
    divk4(t, pr.d_tau_a, a);
#pragma unroll
    for (int q = 0; q < 4; ++q) gk[q] = add(gk[q], mul(pr.cgk, a[q]));
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) t[q] = sub(v1[q], pr.vth);
  divk4(t, pr.d_den, a);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    s[q] = (a[q] >= 0.0f && (!USE_REF || ref[q] == 0.0f)) ? 1.0f : 0.0f;
    v[q] = HARD ? sub(v1[q], mul(sub(v1[q], pr.vr), s[q])) : sub(v1[q], mul(pr.den, s[q]));
    if (KIND == BT_NEURON_ALIF) gk[q] = add(gk[q], mul(pr.dgk, s[q]));
    if (USE_REF) ref[q] = relu_keep_nan(sub(add(ref[q], mul(s[q], pr.tau_ref)), pr.dt));
  }
}

// Publish the spikes of one sample for the 4 neurons i0 .. i0 + 3 of this
// thread (bit q of `nib`: neuron i0 + q), as publish_spikes_ws.  The warp's
// 128 neurons share a sub-list when cap >= 128 (one atomic for the warp),
// otherwise every lane appends its own.  Called by every lane of the warp.
__device__ __forceinline__ void publish_nibble(const ScatterScratch& ws, int i0, int b, uint32_t nib) {
  const unsigned lane = lane_id();
  // The four neurons' mask bits are all issued before the first result is looked at.
  // The first spike in a word of the mask asks the flag whether it is the neuron's
  // first; a mask of one word needs none.
  uint32_t was[4];
#pragma unroll
  for (int q = 0; q < 4; ++q)
    was[q] = nib & (1u << q) ? atomicOr(ws.mask + int64_t(i0 + q) * ws.ms + (b >> 5), 1u << (b & 31)) : 1u;
  if (ws.ms > 1) {
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (was[q] == 0u) was[q] = uint32_t(atomicOr(ws.flag + i0 + q, 1));
  }
  uint32_t first = 0;
#pragma unroll
  for (int q = 0; q < 4; ++q) first |= (was[q] == 0u ? 1u : 0u) << q;
  const int cnt = __popc(first), nspk = __popc(nib);
  int64_t at;
  if (ws.cap_shift >= 7) {
    int incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, incl, o);
      if (int(lane) >= o) incl += y;
    }
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    const int sub = (i0 - 4 * int(lane)) >> ws.cap_shift;  // the same for the whole warp
    const int spk = __reduce_add_sync(0xffffffffu, unsigned(nspk));
    int base = 0;
    if (lane == 0) {
      atomicAdd(ws.spk + sub, spk);
      if (total) base = atomicAdd(ws.count + sub, total);
    }
    base = __shfl_sync(0xffffffffu, base, 0);
    at = int64_t(sub) * ws.cap + base + incl - cnt;
  } else {
    const int sub = i0 >> ws.cap_shift;
    if (nspk) atomicAdd(ws.spk + sub, nspk);
    at = int64_t(sub) * ws.cap + (cnt ? atomicAdd(ws.count + sub, cnt) : 0);
  }
#pragma unroll
  for (int q = 0; q < 4; ++q)
    if (first & (1u << q)) ws.list[at++] = i0 + q;
}

// The same step for n a multiple of 4 and 16-byte aligned arrays: a thread
// owns 4 consecutive neurons of one sample, so every array moves in 16-byte
// accesses (6 in flight per thread, all before the first store) and the
// bookkeeping -- sample length, addresses, bitmap words, publication -- is paid
// once per 4 neurons instead of once per neuron-sample, which is what the
// per-neuron kernel's time went to (its issue slots, 71 %).  A block of a
// finished sample only writes its zero words.  A warp covers 4 bitmap words;
// publication runs only in warps with a spike.  Grid (ceil(n / 512), batch),
// 128 threads.  z_given: publish these spikes instead of the step's own (a
// recomputation driven by the spikes of its first run).
constexpr int kVecThreads = 128;
template <int KIND, bool HARD, bool USE_REF, bool FAST>
__global__ void __launch_bounds__(kVecThreads) k_eng_neuron_vec(bt_engine_desc d, int k, StepIdx si, ScatterScratch ws,
                                                                const float* __restrict__ z_given) {
  step_wait();
  const int n = int(d.n), B = int(d.batch);
  const int words = (n + 31) >> 5;
  const int i0 = (int(blockIdx.x) * kVecThreads + int(threadIdx.x)) * 4;
  const int b = int(blockIdx.y);
  const unsigned lane = lane_id();
  if (i0 - 4 * int(lane) >= n) return;  // whole warps past the end
  const bool valid = i0 < n;            // n % 4 == 0: all four or none
  const int len = d.sample_len ? d.sample_len[b] : INT_MAX;
  const bool st_traces = d.v_trace || d.psc_trace || d.ref_trace || d.gk_trace;
  uint32_t* hist_p = d.hist + (int64_t(si.h_t) * B + b) * words + (i0 >> 5);
  uint32_t* raster_p = d.raster ? d.raster + (int64_t(k) * B + b) * words + (i0 >> 5) : nullptr;
  if (k > len && !st_traces && !d.spikes) {  // block-uniform: frozen, nothing to read
    if (valid && (lane & 7) == 0) {
      *hist_p = 0u;
      if (raster_p) *raster_p = 0u;
    }
    return;
  }
  const int o = b * n + (valid ? i0 : 0);
  const int64_t tix = int64_t(k) * B * n + o;
  const uint64_t pol_stream = l2_evict_first(), pol_keep = l2_evict_last();
  const bool live = k < len, edge = k <= len;
  const bool want = valid && (edge || st_traces);
  const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  float4 aq = zero, pq = zero, xq = zero, vq = zero, rq = zero, gq = zero, zq = zero;
  if (want) {
    if (edge) aq = ld_f4(d.ring + o, pol_keep);
    pq = *reinterpret_cast<const float4*>(d.psc + o);
    if (live && d.x) xq = ld_nc_f4(d.x + tix, pol_stream);
    vq = *reinterpret_cast<const float4*>(d.v + o);
    if (USE_REF) rq = *reinterpret_cast<const float4*>(d.refractory + o);
    if (KIND == BT_NEURON_ALIF) gq = *reinterpret_cast<const float4*>(d.g_k + o);
    if (z_given) zq = ld_nc_f4(z_given + tix, pol_stream);
  }
  float acc[4] = {aq.x, aq.y, aq.z, aq.w}, P[4] = {pq.x, pq.y, pq.z, pq.w}, x[4] = {xq.x, xq.y, xq.z, xq.w};
  float v[4] = {vq.x, vq.y, vq.z, vq.w}, ref[4] = {rq.x, rq.y, rq.z, rq.w}, gk[4] = {gq.x, gq.y, gq.z, gq.w};
  float s[4] = {0.0f, 0.0f, 0.0f, 0.0f}, stored[4];
  if constexpr (FAST) {  // every parameter a scalar
    const NeuronParams prm = load_params<KIND, USE_REF>(d.neuron, 0);
    const Div dpt = make_div(d.psc_tau_s, d.psc_fast_div, d.psc_rcp);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (edge) P[q] = add(P[q], acc[q]);
      stored[q] = P[q];
    }
    if (live) {
      float I[4], t[4], a[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        I[q] = d.x ? add(P[q], x[q]) : P[q];
        t[q] = -P[q];
      }
      neuron_update4<KIND, HARD, USE_REF>(prm, I, v, ref, gk, s);
      divk4(t, dpt, a);
#pragma unroll
      for (int q = 0; q < 4; ++q) stored[q] = add(P[q], mul(d.psc_coef_s, a[q]));
    }
  } else {
    NeuronParams prm = load_params<KIND, USE_REF>(d.neuron, valid ? i0 : 0);
    float pc = d.psc_uniform ? d.psc_coef_s : 0.0f;
    Div dpt = make_div(d.psc_uniform ? d.psc_tau_s : 1.0f, d.psc_uniform && d.psc_fast_div, d.psc_rcp);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int i = valid ? i0 + q : 0;
      if (q > 0 && !d.neuron.uniform) prm = load_params<KIND, USE_REF>(d.neuron, i);
      if (!d.psc_uniform) {
        pc = ld(d.psc_coef, i);
        dpt = make_div(ld(d.psc_tau, i), false, 0.0f);
      }
      if (edge) P[q] = add(P[q], acc[q]);
      stored[q] = P[q];
      if (live) {
        const float I = d.x ? add(P[q], x[q]) : P[q];
        s[q] = neuron_update<KIND, HARD, USE_REF, true, false>(prm, I, v[q], ref[q], gk[q]).spike;
        stored[q] = psc_decay_k<false>(pc, dpt, P[q]);
      }
    }
  }
  uint32_t nib = 0, own = 0;
  if (valid) {
    if (edge) {
      st_f4(d.ring + o, zero, pol_keep);
      *reinterpret_cast<float4*>(d.psc + o) = make_float4(stored[0], stored[1], stored[2], stored[3]);
    }
    if (live) {
      *reinterpret_cast<float4*>(d.v + o) = make_float4(v[0], v[1], v[2], v[3]);
      if (USE_REF) *reinterpret_cast<float4*>(d.refractory + o) = make_float4(ref[0], ref[1], ref[2], ref[3]);
      if (KIND == BT_NEURON_ALIF) *reinterpret_cast<float4*>(d.g_k + o) = make_float4(gk[0], gk[1], gk[2], gk[3]);
    }
    if (st_traces) {
      auto put = [&](float* t, int64_t at, const float(&q)[4]) {
        if (t) *reinterpret_cast<float4*>(t + at) = make_float4(q[0], q[1], q[2], q[3]);
      };
      if (k > 0) put(d.psc_trace, tix - int64_t(B) * n, P);
      put(d.v_trace, tix, v);
      if (USE_REF) put(d.ref_trace, tix, ref);
      if (KIND == BT_NEURON_ALIF) put(d.gk_trace, tix, gk);
    }
    if (d.spikes) *reinterpret_cast<float4*>(d.spikes + tix) = make_float4(s[0], s[1], s[2], s[3]);
#pragma unroll
    for (int q = 0; q < 4; ++q) own |= (s[q] != 0.0f ? 1u : 0u) << q;
    nib = own;
    if (z_given)
      nib = (zq.x != 0.0f ? 1u : 0u) | (zq.y != 0.0f ? 2u : 0u) | (zq.z != 0.0f ? 4u : 0u) | (zq.w != 0.0f ? 8u : 0u);
  }
  const bool any = __any_sync(0xffffffffu, nib != 0);
  uint32_t word = nib << (4 * (lane & 7));
  if (any) {  // the word of the 8 lanes' 32 neurons
#pragma unroll
    for (int w = 1; w < 8; w <<= 1) word |= __shfl_xor_sync(0xffffffffu, word, w);
  }
  if (valid && (lane & 7) == 0) {
    *hist_p = word;
    if (raster_p) *raster_p = word;
  }
  if (any) publish_nibble(ws, i0, b, nib);
}

// SCATTER neuron step with receptor channels (n_rec = C > 1): for each
// channel column c = i * C + r, P_r = stored + acc (acc zeroed); the neuron's
// input is receptor_sum(P) (+ x); stored = decay_r(P_r).  Grid
// (ceil(n / 256), batch): a thread owns (neuron i, sample b).  CT = C known
// at compile time (2 or 4: the channels of (b, i) are one 8- or 16-byte
// vector) or 0 (any C up to kMaxRec).  Every load of the thread is issued
// before its first store: a load behind a store through a pointer that may
// alias it waits for the store, which made this step latency bound.
template <int KIND, bool HARD, bool USE_REF, int CT>
__global__ void __launch_bounds__(kEngThreads) k_eng_neuron_rec(bt_engine_desc d, int64_t k, StepIdx si) {
  step_begin();
  constexpr int M = CT > 0 ? CT : kMaxRec;
  const int64_t n = d.n, B = d.batch;
  const int C = CT > 0 ? CT : n_rec(d);
  const int64_t nc = n * C;
  const int64_t words = (n + 31) >> 5;
  const int64_t i = int64_t(blockIdx.x) * kEngThreads + threadIdx.x;
  const int64_t b = blockIdx.y;
  if ((i & ~int64_t(31)) >= n) return;  // whole warps past the last word
  float s = 0.0f;
  const int64_t len = (i < n && d.sample_len) ? d.sample_len[b] : INT64_MAX;
  const bool st_traces = d.v_trace || d.psc_trace || d.ref_trace || d.gk_trace;
  if (i < n && (k <= len || st_traces)) {  // else: past its length, nothing to read or write
    const int64_t idx = b * n + i, c0 = b * nc + i * C;
    float* ring = d.ring + c0;
    float* psc = d.psc + c0;
    // loads
    float pend[M], stv[M], pc[M], pt[M];
    if constexpr (CT == 4) {
      const float4 a = *reinterpret_cast<const float4*>(ring), q = *reinterpret_cast<const float4*>(psc);
      pend[0] = a.x, pend[1] = a.y, pend[2] = a.z, pend[3] = a.w;
      stv[0] = q.x, stv[1] = q.y, stv[2] = q.z, stv[3] = q.w;
    } else if constexpr (CT == 2) {
      const float2 a = *reinterpret_cast<const float2*>(ring), q = *reinterpret_cast<const float2*>(psc);
      pend[0] = a.x, pend[1] = a.y;
      stv[0] = q.x, stv[1] = q.y;
    } else {
      for (int r = 0; r < C; ++r) {
        pend[r] = ring[r];
        stv[r] = psc[r];
      }
    }
#pragma unroll
    for (int r = 0; r < M; ++r) {
      if (r >= C) break;
      pc[r] = d.psc_uniform ? d.psc_coef_s : ld(d.psc_coef, i * C + r);
      pt[r] = d.psc_uniform ? d.psc_tau_s : ld(d.psc_tau, i * C + r);
    }
    float v = d.v[idx];
    float ref = USE_REF ? d.refractory[idx] : 0.0f;
    float gk = KIND == BT_NEURON_ALIF ? d.g_k[idx] : 0.0f;
    const float xv = d.x ? d.x[(k * B) * n + idx] : 0.0f;
    const NeuronParams prm = load_params<KIND, USE_REF>(d.neuron, i);
    // past a sample's end: the first step completes psc of its last step,
    // later arrivals are dropped (as k_eng_neuron)
    float P[M];
#pragma unroll
    for (int r = 0; r < M; ++r) {
      if (r >= C) break;
      P[r] = k <= len ? add(stv[r], pend[r]) : stv[r];
    }
    // stores
    if constexpr (CT == 4) {
      *reinterpret_cast<float4*>(ring) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    } else if constexpr (CT == 2) {
      *reinterpret_cast<float2*>(ring) = make_float2(0.0f, 0.0f);
    } else {
      for (int r = 0; r < C; ++r) ring[r] = 0.0f;
    }
    float out[M];
    bool write = k <= len;
    if (k < len) {
      const float I0 = receptor_sum(P, C);
      const float I = d.x ? add(I0, xv) : I0;
      const NeuronOut o = neuron_update<KIND, HARD, USE_REF, true>(prm, I, v, ref, gk);
      s = o.spike;
      d.v[idx] = v;
      if (USE_REF) d.refractory[idx] = ref;
      if (KIND == BT_NEURON_ALIF) d.g_k[idx] = gk;
#pragma unroll
      for (int r = 0; r < M; ++r) {
        if (r >= C) break;
        out[r] = psc_decay(pc[r], make_div(pt[r], d.psc_uniform && d.psc_fast_div, d.psc_rcp), P[r]);
      }
    } else {
#pragma unroll
      for (int r = 0; r < M; ++r) {
        if (r >= C) break;
        out[r] = P[r];
      }
    }
    if (write) {
      if constexpr (CT == 4) {
        *reinterpret_cast<float4*>(psc) = make_float4(out[0], out[1], out[2], out[3]);
      } else if constexpr (CT == 2) {
        *reinterpret_cast<float2*>(psc) = make_float2(out[0], out[1]);
      } else {
        for (int r = 0; r < C; ++r) psc[r] = out[r];
      }
    }
    if (d.psc_trace && k > 0) {
      float* tr = d.psc_trace + ((k - 1) * B) * nc + c0;
#pragma unroll
      for (int r = 0; r < M; ++r) {
        if (r >= C) break;
        tr[r] = P[r];
      }
    }
    const int64_t tix = (k * B) * n + idx;
    if (d.v_trace) d.v_trace[tix] = v;
    if (USE_REF && d.ref_trace) d.ref_trace[tix] = ref;
    if (KIND == BT_NEURON_ALIF && d.gk_trace) d.gk_trace[tix] = gk;
  }
  if (i < n && d.spikes) d.spikes[(k * B + b) * n + i] = s;
  const uint32_t word = __ballot_sync(0xffffffffu, s != 0.0f);
  if (lane_id() == 0) {
    d.hist[(int64_t(si.h_t) * B + b) * words + (i >> 5)] = word;
    if (d.raster) d.raster[(k * B + b) * words + (i >> 5)] = word;
  }
  publish_spikes<1>(d, si, i, b, s != 0.0f ? 1u : 0u);
}

// Offsets of the sub-lists of every delivered spike set (planes x kSub, plane y
// = delay bin bin_lo + y, the set of step t - bin) in shared memory: s_off[c] =
// rows listed before counter c, s_off[planes * kSub] = rows of the step.  One
// list over all planes lets every warp of the grid take its share of the rows
// whatever bin they belong to.  *s_spk: spikes listed (one plane only).
template <int T = kEngThreads>
__device__ __forceinline__ void plane_offsets(const bt_engine_desc& d, const StepIdx& si, int planes, int32_t* s_off,
                                              int32_t* s_spk) {
  __shared__ int32_t s_warp[T / 32];
  const int Q = d.n_bins + 1, total = planes * kSub;
  const int per = (total + T - 1) / T;
  const int c0 = int(threadIdx.x) * per, c1 = c0 + per < total ? c0 + per : total;
  int32_t sum = 0, spk = 0;
#pragma unroll 4
  for (int c = c0; c < c1; ++c) {
    int q = si.q_t - d.bin_lo - c / kSub;
    if (q < 0) q += Q;
    const int32_t* cnt = d.work + q * 2 * kSub + c % kSub;
    const int32_t v = cnt[0];
    if (planes == 1) spk += cnt[kSub];
    s_off[c] = v;
    sum += v;
  }
  const int lane = int(lane_id()), warp = int(threadIdx.x >> 5);
  int32_t incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int32_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) s_warp[warp] = incl;
  if (threadIdx.x == 0) *s_spk = 0;
  __syncthreads();
  if (planes == 1 && spk) atomicAdd(s_spk, spk);
  int32_t run = incl - sum;
#pragma unroll
  for (int w = 0; w < T / 32; ++w) run += w < warp ? s_warp[w] : 0;
  for (int c = c0; c < c1; ++c) {
    const int32_t v = s_off[c];
    s_off[c] = run;
    run += v;
  }
  if (threadIdx.x == T - 1) s_off[total] = run;
  __syncthreads();
}

// Counter holding item `it`: the last c with s_off[c] <= it (s_off[total] > it).
__device__ __forceinline__ int find_sub(const int32_t* s_off, int total, int32_t it) {
  int lo = 0, hi = total - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (s_off[mid] <= it) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// One listed row of the step: its neuron, delay bin and sample mask.
struct ListedRow {
  int32_t j;
  int bin;
  uint32_t* mask;
  int32_t* flag;
};

__device__ __forceinline__ ListedRow listed_row(const bt_engine_desc& d, const StepIdx& si, const ScatterScratch& ws0,
                                                const int32_t* s_off, int planes, int32_t it) {
  const int c = find_sub(s_off, planes * kSub, it);
  ListedRow r;
  r.bin = d.bin_lo + c / kSub;
  int q = si.q_t - r.bin;
  if (q < 0) q += d.n_bins + 1;
  r.j = ws0.list[(int64_t(q) * kSub + c % kSub) * ws0.cap + (it - s_off[c])];
  r.mask = ws0.mask + (int64_t(q) * d.n + r.j) * ws0.ms;
  r.flag = ws0.flag + int64_t(q) * d.n + r.j;
  return r;
}

// The counts of slot (t + 1) mod Q, i.e. of step t - R, were last read by the
// previous step's scatter: clear them for the next neuron launch.
__device__ __forceinline__ void clear_oldest_counts(const bt_engine_desc& d, const StepIdx& si) {
  if (blockIdx.x == 0 && threadIdx.x < 2 * kSub) {
    const int qc = si.q_t + 1 == d.n_bins + 1 ? 0 : si.q_t + 1;
    d.work[qc * 2 * kSub + threadIdx.x] = 0;
  }
}

// Block-level sum of per-thread event / edge counts, one pair of atomics per
// block (same-address atomics serialise in L2).  Every thread of the block
// must call it.
__device__ __forceinline__ void block_stats(const bt_engine_desc& d, int64_t k, long long ev, long long ed) {
  __shared__ long long s_ev[kEngThreads / 32], s_ed[kEngThreads / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ev += __shfl_xor_sync(0xffffffffu, ev, o);
    ed += __shfl_xor_sync(0xffffffffu, ed, o);
  }
  if (lane_id() == 0) {
    s_ev[threadIdx.x >> 5] = ev;
    s_ed[threadIdx.x >> 5] = ed;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    long long tev = 0, ted = 0;
    for (int w = 0; w < kEngThreads / 32; ++w) {
      tev += s_ev[w];
      ted += s_ed[w];
    }
    if (ted) {
      atomicAdd(reinterpret_cast<unsigned long long*>(d.stats + k * 4 + 1), (unsigned long long)tev);
      atomicAdd(reinterpret_cast<unsigned long long*>(d.stats + k * 4 + 2), (unsigned long long)ted);
    }
  }
}

// Dense delivery of one spike set (single delay bin): a block owns a slice of
// 32 posts (lane = post); its W warps split the slice's rows of the sliced
// in-edge view and accumulate, one 32-sample mask word per pass, into
// per-warp shared-memory columns (no conflicts, no atomics); the block then
// sums the W partial columns and stores the totals into acc with plain
// stores (acc is zero on entry, each (sample, post) has one writer).  s_acc:
// W columns of 32 x 32 in shared memory, W the block's warps.  Used
// for steps where most neurons spike in some sample, where per-event
// reductions would cost more than reading every in-edge once.  The spike
// set's masks and flags are then cleared by the last block to finish
// (block-completion counter in ctrl[0]; no block waits for another).
template <int MS, int W = kEngThreads / 32>
__device__ void scatter_dense(const bt_engine_desc& d, const ScatterScratch& ws, float (*s_acc)[32][32], long long& ev,
                              long long& ed) {
  const int lane = int(lane_id()), wid = int(threadIdx.x >> 5);
  const int64_t n = d.n, B = d.batch;
  const int64_t nc = n * n_rec(d);  // acc columns (post * C + r)
  const int n32 = int(nc);
  const int64_t n_slices = (nc + 31) >> 5;
  const int64_t nblocks = gridDim.x, bid = blockIdx.x;
  float(*acc)[32] = s_acc[wid];
  const uint64_t pol_stream = l2_evict_first();
  const uint32_t sentinel = uint32_t(n);
  for (int64_t sl = bid; sl < n_slices; sl += nblocks) {  // uniform per block
    const int64_t r0 = d.sl_ptr[sl], r1 = d.sl_ptr[sl + 1];
    const int64_t per = (r1 - r0 + W - 1) / W;
    const int64_t ra = r0 + wid * per, rb = ra + per < r1 ? ra + per : r1;
    for (int w = 0; w < ws.ms; ++w) {
#pragma unroll 8
      for (int l = 0; l < 32; ++l) acc[l][lane] = 0.0f;
      __syncwarp();
      constexpr int U = 8;
      for (int64_t r = ra; r < rb; r += U) {
        uint32_t src[U];
        float wg[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const bool in = r + u < rb;
          src[u] = in ? ld_nc_u32(d.sl_src + (r + u) * 32 + lane, pol_stream) & kIdMask : sentinel;
          wg[u] = in ? ld_nc_f32(d.sl_w + (r + u) * 32 + lane, pol_stream) : 0.0f;
        }
        uint32_t m[U];
#pragma unroll
        for (int u = 0; u < U; ++u) m[u] = src[u] < sentinel ? ws.mask[int64_t(src[u]) * ws.ms + w] : 0u;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (w == 0 && src[u] < sentinel) {
            bool any = m[u] != 0;
            for (int x = 1; x < ws.ms && !any; ++x) any = ws.mask[int64_t(src[u]) * ws.ms + x] != 0;
            ed += any ? 1 : 0;
          }
          ev += __popc(m[u]);
          uint32_t mm = m[u];
          while (mm) {
            const int l = __ffs(mm) - 1;
            mm &= mm - 1;
            acc[l][lane] = add(acc[l][lane], wg[u]);
          }
        }
      }
      __syncthreads();
      for (int idx = threadIdx.x; idx < 32 * 32; idx += blockDim.x) {
        const int l = idx >> 5, ln = idx & 31;
        float sum = 0.0f;
#pragma unroll
        for (int v = 0; v < W; ++v) sum = add(sum, s_acc[v][l][ln]);
        const int64_t b = int64_t(w) * 32 + l, p = sl * 32 + ln;
        if (b < B && p < nc && sum != 0.0f) d.ring[b * n32 + p] = sum;
      }
      __syncthreads();
    }
  }
  // the last block to finish clears the spike set (no other block reads it)
  __shared__ int s_last;
  if (threadIdx.x == 0) {
    __threadfence();
    const int done = atomicAdd(ws.ctrl, 1);
    s_last = done == int(nblocks) - 1;
  }
  __syncthreads();
  if (s_last) {
    __threadfence();
    for (int64_t i = threadIdx.x; i < n * ws.ms; i += blockDim.x) ws.mask[i] = 0u;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) ws.flag[i] = 0;
    if (threadIdx.x == 0) ws.ctrl[0] = 0;
  }
}

// Delivery of one step: for every listed neuron j of the spike set of step
// t - bin, for every delay bin, row j * R + bin.  G lanes share one row, each
// lane loading 4 edges with two 128-bit loads of records, then adding them for
// every sample in the row's mask (MS words; the sample loop is outside the edge
// loop, so a lane issues 4 reductions per mask bit).  The grid is one wave of
// resident blocks over the rows of all bins: a step is a
// chain of dependent loads per row (list, row pointers and mask, edges), so a
// second wave, or planes of a bin each with idle warps beside busy ones, costs
// the whole chain again (20 bins, 120k rows of 6 edges: 12.9 us a step with a
// plane of blocks per bin and two waves).
// Launch bounds: at least 4 (MS <= 4) or 3 resident blocks per SM, which
// leaves ptxas 64 / 85 registers -- without a bound its occupancy heuristic
// has settled on 48 registers and spilled the reduction loop.
constexpr size_t kScatterStatic = 33 * 1024;  // at least the static shared memory of k_eng_scatter and k_eng_scatter_flat
template <int G, int MS>
__global__ void __launch_bounds__(kEngThreads, MS <= 4 ? 4 : 3) k_eng_scatter(bt_engine_desc d, int64_t k, StepIdx si) {
  step_begin();
  extern __shared__ int32_t s_off[];  // [planes * kSub + 1]
  const int64_t n = d.n;
  const int R = d.n_bins, planes = d.bin_hi - d.bin_lo + 1;
  const ScatterScratch ws0 = scatter_scratch(d, 0);
  __shared__ int32_t s_spk;
  plane_offsets(d, si, planes, s_off, &s_spk);
  const int32_t count = s_off[planes * kSub];
  clear_oldest_counts(d, si);
  if (blockIdx.x == 0 && threadIdx.x == 0 && d.stats)
    atomicAdd(reinterpret_cast<unsigned long long*>(d.stats + k * 4 + 0), (unsigned long long)count);
  // dense when most neurons spike and they do so in several samples each
  if (d.dense_rows > 0 && count >= d.dense_rows && s_spk >= kDenseSpikesPerRow * count) {  // grid-uniform
    int q = si.q_t - d.bin_lo;
    if (q < 0) q += R + 1;
    long long ev = 0, ed = 0;
    __shared__ float s_acc[kEngThreads / 32][32][32];  // (beside the offsets: overlaid on them, 1.4 % slower at 20 bins)
    scatter_dense<MS>(d, scatter_scratch(d, q), s_acc, ev, ed);
    if (d.stats) block_stats(d, k, ev, ed);
    return;
  }
  const unsigned lane = lane_id();
  const int grp = int(lane) / G, lig = int(lane) % G;
  constexpr int kPerWarp = 32 / G;
  const int64_t warps = (int64_t(gridDim.x) * blockDim.x) >> 5;
  const int n32 = int(n * n_rec(d));  // acc row stride; batch * n * C < 2^31 (checked on the host)
  // (as k_eng_scatter_flat: lines with the following rows, for the next steps)
  const uint64_t pol_edges = R > 1 ? l2_evict_normal() : l2_evict_first(), pol_keep = l2_evict_last();
  long long ev = 0, ed = 0;
  for (int64_t base = ((int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5) * kPerWarp; base < count;
       base += warps * kPerWarp) {
    const int64_t it = base + grp;
    uint32_t mw_local[MS];
    int32_t beg = 0, end = 0;
    uint32_t* mrow = nullptr;
    int32_t* flag = nullptr;
    if (it < count) {
      const ListedRow r = listed_row(d, si, ws0, s_off, planes, int32_t(it));
      mrow = r.mask;
      flag = r.bin == d.bin_hi ? r.flag : nullptr;  // this set is not read again: clear it
      const int64_t row = int64_t(r.j) * R + r.bin;
      beg = ld_nc_s32_line(d.csr_ptr + row);
      end = ld_nc_s32_line(d.csr_ptr + row + 1);
    }
    // MS is the compile-time bound (1, 2, 4 or 8); the row holds ms words
    // (5..8 samples words above 128 samples run with MS = 8)
    int nsamp = 0;
#pragma unroll
    for (int w = 0; w < MS; ++w) {
      mw_local[w] = (mrow && w < ws0.ms) ? mrow[w] : 0u;
      nsamp += __popc(mw_local[w]);
    }
    __syncwarp();
    if (flag && lig == 0) {
#pragma unroll
      for (int w = 0; w < MS; ++w)
        if (w < ws0.ms) mrow[w] = 0;
      *flag = 0;
    }
    if (lig == 0) {
      ev += (long long)nsamp * (end - beg);
      ed += end - beg;
    }
    // U quads per lane in flight: all loads of an iteration are issued before
    // its reductions
    constexpr int U = 2;
    for (int32_t g0 = (beg & ~3) + lig * 4; g0 < end; g0 += G * 4 * U) {
      uint4 dq[U], wq[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int32_t gi = g0 + u * G * 4;
        if (gi < end) {
          // edges gi .. gi+3 as (post, weight) records: two 128-bit loads
          const uint4 a = ld_nc_u4_line(d.csr_edges + 2 * int64_t(gi), pol_edges);
          const uint4 b = ld_nc_u4_line(d.csr_edges + 2 * int64_t(gi) + 4, pol_edges);
          dq[u] = make_uint4(a.x, a.z, b.x, b.z);
          wq[u] = make_uint4(a.y, a.w, b.y, b.w);
        } else {
          dq[u] = make_uint4(0u, 0u, 0u, 0u);
          wq[u] = dq[u];
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int32_t gidx = g0 + u * G * 4;
        // edges outside [beg, end) of the first and last quad add nothing
        const bool v0 = gidx >= beg && gidx < end, v1 = gidx + 1 >= beg && gidx + 1 < end,
                   v2 = gidx + 2 >= beg && gidx + 2 < end, v3 = gidx + 3 >= beg && gidx + 3 < end;
        const int p0 = int(dq[u].x & kIdMask), p1 = int(dq[u].y & kIdMask), p2 = int(dq[u].z & kIdMask),
                  p3 = int(dq[u].w & kIdMask);
#pragma unroll
        for (int w = 0; w < MS; ++w) {
          uint32_t m = mw_local[w];
          while (m) {
            const int l = __ffs(m) - 1;
            m &= m - 1;
            float* row = d.ring + (w * 32 + l) * n32;
            if (v0) red_add_f32(row + p0, __uint_as_float(wq[u].x), pol_keep);
            if (v1) red_add_f32(row + p1, __uint_as_float(wq[u].y), pol_keep);
            if (v2) red_add_f32(row + p2, __uint_as_float(wq[u].z), pol_keep);
            if (v3) red_add_f32(row + p3, __uint_as_float(wq[u].w), pol_keep);
          }
        }
      }
    }
  }
  if (d.stats) block_stats(d, k, ev, ed);
}

// Scatter for short rows (a wide delay range splits each neuron's out-edges
// into n_bins rows): a warp takes up to 32 rows -- the step's rows spread evenly
// over the grid's warps -- one per lane, scans their lengths and walks their
// edges as one flattened range, 32 consecutive edges per iteration: each lane
// finds its row by a 5-step binary search over the lanes' exclusive offsets
// (shuffles), so no lane idles on a short row and consecutive lanes load
// consecutive edges.  Grid as k_eng_scatter.
template <int MS>
__global__ void __launch_bounds__(kEngThreads, MS <= 4 ? 4 : 3) k_eng_scatter_flat(bt_engine_desc d, int64_t k,
                                                                              StepIdx si) {
  step_begin();
  extern __shared__ int32_t s_off[];  // [planes * kSub + 1]
  const int R = d.n_bins, planes = d.bin_hi - d.bin_lo + 1;
  const ScatterScratch ws0 = scatter_scratch(d, 0);
  __shared__ int32_t s_spk;
  plane_offsets(d, si, planes, s_off, &s_spk);
  const int32_t count = s_off[planes * kSub];
  clear_oldest_counts(d, si);
  if (blockIdx.x == 0 && threadIdx.x == 0 && d.stats)
    atomicAdd(reinterpret_cast<unsigned long long*>(d.stats + k * 4 + 0), (unsigned long long)count);
  // dense when most neurons spike and they do so in several samples each
  if (d.dense_rows > 0 && count >= d.dense_rows && s_spk >= kDenseSpikesPerRow * count) {  // grid-uniform
    int q = si.q_t - d.bin_lo;
    if (q < 0) q += R + 1;
    long long ev = 0, ed = 0;
    __shared__ float s_acc[kEngThreads / 32][32][32];  // (beside the offsets: overlaid on them, 1.4 % slower at 20 bins)
    scatter_dense<MS>(d, scatter_scratch(d, q), s_acc, ev, ed);
    if (d.stats) block_stats(d, k, ev, ed);
    return;
  }
  const int lane = int(lane_id());
  const int64_t warps = (int64_t(gridDim.x) * blockDim.x) >> 5;
  const int n32 = int(d.n * n_rec(d));  // acc row stride; batch * n * C < 2^31 (checked on the host)
  // a neuron's rows are consecutive and read in consecutive steps: whole lines
  // are brought in and kept for the next steps (one bin: read once, given up first)
  const uint64_t pol_edges = R > 1 ? l2_evict_normal() : l2_evict_first(), pol_keep = l2_evict_last();
  long long ev = 0, ed = 0;
  // rows per warp and pass, 32 at most: an even share of the step's rows, over as
  // many passes as it takes (passes of 32 leave the last one part empty: 140000
  // neurons, 17 edges a row, 240000 rows a step 58.8 us, 57.3 in equal passes)
  const int64_t share = (count + warps - 1) / warps, passes = (share + 31) / 32;
  const int rpw = int(passes > 1 ? (share + passes - 1) / passes : share);
  for (int64_t base = ((int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5) * rpw; base < count;
       base += warps * rpw) {
    const int64_t it = base + lane;
    uint32_t mw[MS];
    int32_t beg = 0, len = 0;
    if (lane < rpw && it < count) {
      const ListedRow r = listed_row(d, si, ws0, s_off, planes, int32_t(it));
      const int64_t row = int64_t(r.j) * R + r.bin;
      beg = ld_nc_s32_line(d.csr_ptr + row);
      len = ld_nc_s32_line(d.csr_ptr + row + 1) - beg;
      int nsamp = 0;
#pragma unroll
      for (int w = 0; w < MS; ++w) {
        mw[w] = w < ws0.ms ? r.mask[w] : 0u;
        nsamp += __popc(mw[w]);
      }
      if (r.bin == d.bin_hi) {  // this set is not read again: clear it
#pragma unroll
        for (int w = 0; w < MS; ++w)
          if (w < ws0.ms) r.mask[w] = 0;
        *r.flag = 0;
      }
      ev += (long long)nsamp * len;
      ed += len;
    } else {
#pragma unroll
      for (int w = 0; w < MS; ++w) mw[w] = 0u;
    }
    // exclusive offsets of the 32 rows in the flattened edge range
    int32_t incl = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    const int32_t excl = incl - len;
    const int32_t total = __shfl_sync(0xffffffffu, incl, 31);
    // U edges per lane in flight: the row searches and loads of an iteration
    // come before its reductions
    constexpr int U = 4;
    for (int32_t e0 = 0; e0 < total; e0 += 32 * U) {
      int pp[U];
      float wv[U];
      uint32_t mm[U][MS];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int32_t e = e0 + u * 32 + lane;
        // r = the last lane whose excl <= e (rows of length 0 are skipped over)
        int r = 0;
#pragma unroll
        for (int step = 16; step > 0; step >>= 1) {
          const int32_t x = __shfl_sync(0xffffffffu, excl, r + step);
          if (x <= e) r += step;
        }
        const int32_t rbeg = __shfl_sync(0xffffffffu, beg, r);
        const int32_t rexcl = __shfl_sync(0xffffffffu, excl, r);
#pragma unroll
        for (int w = 0; w < MS; ++w) mm[u][w] = __shfl_sync(0xffffffffu, mw[w], r);
        pp[u] = 0;
        wv[u] = 0.0f;
        if (e < total) {
          const int32_t g = rbeg + (e - rexcl);
          const uint2 e = ld_nc_u2_line(d.csr_edges + 2 * int64_t(g), pol_edges);
          pp[u] = int(e.x & kIdMask);
          wv[u] = __uint_as_float(e.y);
        } else {
#pragma unroll
          for (int w = 0; w < MS; ++w) mm[u][w] = 0u;
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
#pragma unroll
        for (int w = 0; w < MS; ++w) {
          uint32_t m = mm[u][w];
          while (m) {
            const int l = __ffs(m) - 1;
            m &= m - 1;
            red_add_f32(d.ring + (w * 32 + l) * n32 + pp[u], wv[u], pol_keep);
          }
        }
      }
    }
  }
  if (d.stats) block_stats(d, k, ev, ed);
}

// Delivery sample by sample, summed in shared memory: a block takes one of
// `parts` shares of a sample's spikes (listed from the step's bitmap), adds the
// rows' edges into n accumulators in shared memory and then adds those, four at
// a time, to the sample's row of acc.
// k_eng_scatter is bound by its reductions in L2 (150 G/s over the device, 31
// us for the 4.3M of a step at 8192 neurons, 410 edges a row, 128 samples, 1 %
// spiking); additions in shared memory are about three times as fast and the
// rows of acc are touched in whole lines: a training window of 100 such steps
// 25.4 -> 22.9 ms.  One share per sample instead of two takes 25.2 ms: the
// samples' spikes differ, and the busiest one is waited for; eight take 24.5,
// each share pays its zeros and its n sums.  Shares of posts instead of spikes
// read every edge in each of them (23.6 ms).
// The spike set of the step, which the neuron launch still publishes (the dense
// step reads it), is cleared whole.
constexpr int kRowThreads = 512, kRowWarps = kRowThreads / 32, kRowList = 4096;
constexpr int64_t kRowMaxN = 16384;  // accumulators and list of two blocks per SM: 160 KB
template <int MS>
__global__ void __launch_bounds__(kRowThreads, 2) k_eng_scatter_rows(bt_engine_desc d, StepIdx si, int parts) {
  step_begin();
  extern __shared__ __align__(16) float s_dyn[];  // [kRowList] row list, then accumulators or the dense step's columns
  int32_t* s_list = reinterpret_cast<int32_t*>(s_dyn);
  float* acc = s_dyn + kRowList;
  const int bin = d.bin_lo, R = d.n_bins, n = int(d.n), B = int(d.batch);
  int q = si.q_t - bin;
  if (q < 0) q += R + 1;
  const ScatterScratch ws = scatter_scratch(d, q);
  clear_oldest_counts(d, si);
  if (d.dense_rows > 0) {
    __shared__ int32_t s_off[kSub + 1], s_spk;
    plane_offsets<kRowThreads>(d, si, 1, s_off, &s_spk);
    const int32_t count = s_off[kSub];
    if (count >= d.dense_rows && s_spk >= kDenseSpikesPerRow * count) {  // grid-uniform
      long long ev = 0, ed = 0;
      scatter_dense<MS, kRowWarps>(d, ws, reinterpret_cast<float(*)[32][32]>(acc), ev, ed);
      return;
    }
  }
  const int tid = int(threadIdx.x), lane = int(lane_id()), wid = tid >> 5;
  for (int i = int(blockIdx.x) * kRowThreads + tid; i < n * ws.ms; i += int(gridDim.x) * kRowThreads) ws.mask[i] = 0u;
  for (int i = int(blockIdx.x) * kRowThreads + tid; i < n; i += int(gridDim.x) * kRowThreads) ws.flag[i] = 0;
  const int b = int(blockIdx.x) / parts, part = int(blockIdx.x) - b * parts;
  __shared__ int32_t s_warp[kRowWarps];
  const int words = (n + 31) >> 5, per = (words + kRowThreads - 1) / kRowThreads;
  const int w0 = tid * per < words ? tid * per : words, w1 = w0 + per < words ? w0 + per : words;
  int h = si.h_t - bin;
  if (h < 0) h += d.hist_len;
  const uint32_t* bits = d.hist + (int64_t(h) * B + b) * words;  // (this step's words: plain loads)
  int cnt = 0;
  for (int w = w0; w < w1; ++w) cnt += __popc(bits[w]);
  for (int i = tid; i < n; i += kRowThreads) acc[i] = 0.0f;
  int incl = cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) s_warp[wid] = incl;
  __syncthreads();
  const int wsum = lane < kRowWarps ? s_warp[lane] : 0;
  const int total = int(__reduce_add_sync(0xffffffffu, unsigned(wsum)));
  const int before = int(__reduce_add_sync(0xffffffffu, unsigned(lane < wid ? wsum : 0)));
  const int first = before + incl - cnt;  // this thread's first spike among the sample's
  // this block's share of the sample's spikes
  const int own0 = int(int64_t(total) * part / parts), own1 = int(int64_t(total) * (part + 1) / parts);
  if (own0 == own1) return;  // block-uniform
  const uint64_t pol = l2_evict_normal();
  for (int base = own0; base < own1; base += kRowList) {
    const int rows = own1 - base < kRowList ? own1 - base : kRowList;
    int at = first - base;
    for (int w = w0; w < w1; ++w) {
      uint32_t m = bits[w];
      while (m) {
        const int l = __ffs(m) - 1;
        m &= m - 1;
        if (at >= 0 && at < rows) s_list[at] = w * 32 + l;
        ++at;
      }
    }
    __syncthreads();
    // warp w takes rows w, w + kRowWarps, ...: 32 row pointers at a time, one per lane
    for (int r0 = wid; r0 < rows; r0 += kRowThreads) {
      int32_t beg = 0, end = 0;
      if (r0 + kRowWarps * lane < rows) {
        const int64_t row = int64_t(s_list[r0 + kRowWarps * lane]) * R + bin;
        beg = ld_nc_s32_line(d.csr_ptr + row);
        end = ld_nc_s32_line(d.csr_ptr + row + 1);
      }
      const int nr = (rows - r0 + kRowWarps - 1) / kRowWarps;
      for (int r = 0; r < (nr < 32 ? nr : 32); ++r) {
        const int32_t rb = __shfl_sync(0xffffffffu, beg, r), re = __shfl_sync(0xffffffffu, end, r);
        constexpr int U = 4;  // pairs of edges in flight per lane
        for (int32_t e0 = (rb & ~1) + 2 * lane; e0 - 2 * lane < re; e0 += 64 * U) {
          uint4 v[U];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int32_t e = e0 + 64 * u;
            v[u] = e < re ? ld_nc_u4_line(d.csr_edges + 2 * int64_t(e), pol) : make_uint4(0u, 0u, 0u, 0u);
          }
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int32_t e = e0 + 64 * u;
            if (e >= rb && e < re) atomicAdd(acc + (v[u].x & kIdMask), __uint_as_float(v[u].y));
            if (e + 1 < re) atomicAdd(acc + (v[u].z & kIdMask), __uint_as_float(v[u].w));
          }
        }
      }
    }
    __syncthreads();
  }
  // acc is zero on entry and holds a finite or infinite sum after it whatever the
  // order of the shares; zeros add nothing
  float* out = d.ring + int64_t(b) * n;
  if ((n & 3) == 0 && (reinterpret_cast<uintptr_t>(d.ring) & 15) == 0) {
    for (int i = 4 * tid; i < n; i += 4 * kRowThreads) {
      const float4 f = *reinterpret_cast<const float4*>(acc + i);
      if (f.x != 0.0f || f.y != 0.0f || f.z != 0.0f || f.w != 0.0f) atomicAdd(reinterpret_cast<float4*>(out + i), f);
    }
  } else {
    for (int i = tid; i < n; i += kRowThreads)
      if (acc[i] != 0.0f) atomicAdd(out + i, acc[i]);
  }
}

// Shares per sample of k_eng_scatter_rows, 0 where k_eng_scatter is taken: one
// delay bin, one channel, no statistics (they count the set's rows), long rows
// (the 32-lane choice) and enough samples for two blocks per SM.  Windows of 40
// training steps, k_eng_scatter against this one: 8192 neurons, batch 16: 3.76 /
// 3.70 ms, 32: 4.81 / 4.37, 64: 6.95 / 6.49, 128: 10.9 / 9.9, 200: 17.5 / 15.9;
// 2000 neurons, batch 64: 2.72 / 2.70, 4096, 128: 4.92 / 4.63, 16384, 128: 12.6 /
// 12.0; but 30000, 64: 9.4 / 10.2 (zeros and sums of n per share).  A run driven
// by given spikes needs them in the bitmap, which the vector neuron step writes.
int row_parts(const bt_engine_desc& d, const float* z_given, bool vec, int sms) {
  if (d.bin_lo != d.bin_hi || n_rec(d) != 1 || d.stats || d.scatter_lanes != 32 || (z_given && !vec)) return 0;
  if (d.batch < 32 || d.n > kRowMaxN) return 0;
  return int(std::max<int64_t>(2, 2 * sms / d.batch));
}

// psc_{t_end-1} = stored + acc; clears acc.
__global__ void k_eng_scatter_final(bt_engine_desc d) {
  const int64_t idx = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  const int64_t nc = d.n * n_rec(d), B = d.batch;  // one thread per PSC column
  if (idx >= B * nc) return;
  // all loads before the first store (see k_eng_neuron_rec)
  float* __restrict__ ring = d.ring;
  float* __restrict__ psc = d.psc;
  const float pending = ring[idx];
  const float stored = psc[idx];
  const int64_t b = idx / nc;
  const int64_t len = d.sample_len ? d.sample_len[b] : INT64_MAX;
  ring[idx] = 0.0f;
  const float P = d.n_steps - 1 < len ? add(stored, pending) : stored;
  if (d.n_steps - 1 < len) psc[idx] = P;
  if (d.psc_trace) d.psc_trace[((d.n_steps - 1) * B) * nc + idx] = P;
}

// ----------------------------------------------------------------- gather --

// Ordered in-edge gather of W z for (b, i) at arrival step `ta`:
// sum over in-edges (pre, bin) ascending of w * z_{ta - bin}[pre].
__device__ __forceinline__ float gather_in(const bt_engine_desc& d, int64_t i, int64_t b, int ta_mod_h, int64_t words) {
  const unsigned lane = lane_id();
  const int32_t beg = __ldg(d.csc_ptr + i), end = __ldg(d.csc_ptr + i + 1);
  const int H = d.hist_len;  // slot of bin b is ta_mod_h - b (mod H), b < H
  float acc = 0.0f;
  for (int32_t base = beg; base < end; base += 32) {
    const int32_t e = base + int32_t(lane);
    float w = 0.0f;
    bool act = false;
    if (e < end) {
      const uint32_t src = __ldg(d.csc_src + e);
      const uint32_t pre = src & kIdMask;
      int slot = ta_mod_h - int(src >> BT_BIN_SHIFT);
      if (slot < 0) slot += H;
      const uint32_t word = d.hist[(int64_t(slot) * d.batch + b) * words + (pre >> 5)];
      act = (word >> (pre & 31)) & 1u;
      if (act) w = __ldg(d.csc_w + e);
    }
    uint32_t m = __ballot_sync(0xffffffffu, act);
    while (m) {
      const int q = __ffs(m) - 1;
      m &= m - 1;
      acc = fmaf(__shfl_sync(0xffffffffu, w, q), 1.0f, acc);
    }
  }
  return acc;
}

// One launch per step.  Block = 32 warps = 32 consecutive neurons, so each
// (sample, 32-neuron word) of the spike bitmap is written by one thread.
// REC: receptor channels, the warp gathers the C columns i * C + r in turn.
template <int KIND, bool HARD, bool USE_REF, bool REC>
__global__ void __launch_bounds__(1024) k_eng_gather(bt_engine_desc d, int64_t k, StepIdx si) {
  extern __shared__ uint32_t sbits[];  // [batch]
  const int64_t n = d.n, B = d.batch;
  const int64_t words = (n + 31) >> 5;
  const int wid = threadIdx.x >> 5;
  const unsigned lane = lane_id();
  const int64_t i = int64_t(blockIdx.x) * 32 + wid;
  for (int64_t b = threadIdx.x; b < B; b += blockDim.x) sbits[b] = 0;
  __syncthreads();
  int nspk = 0;
  if (i < n) {
    for (int64_t b = 0; b < B; ++b) {
      const int64_t idx = b * n + i;
      const int64_t len = d.sample_len ? d.sample_len[b] : INT64_MAX;
      // synapse update of step t-1 (skipped on the first step of a call: the
      // stored psc already is psc_{t0-1}; skipped after a sample's last step)
      const bool syn = k > 0 && k - 1 < len;
      float P;
      float Pr[REC ? kMaxRec : 1];
      const int C = REC ? d.n_rec : 1;
      const int64_t c0 = (b * n + i) * C;  // first PSC column of (b, i)
      if constexpr (!REC) {
        P = d.psc[idx];
        if (syn) P = add(psc_decay(d.psc_coef, d.psc_tau, i, P), gather_in(d, i, b, si.h_prev, words));
      } else {
        for (int r = 0; r < C; ++r) {
          float q = d.psc[c0 + r];
          if (syn) q = add(psc_decay(d.psc_coef, d.psc_tau, i * C + r, q), gather_in(d, i * C + r, b, si.h_prev, words));
          Pr[r] = q;
        }
        P = receptor_sum(Pr, C);
      }
      float s = 0.0f;
      if (lane == 0) {
        if (k < len) {
          const float I = d.x ? add(P, d.x[(k * B) * n + idx]) : P;
          float v = d.v[idx];
          float ref = USE_REF ? d.refractory[idx] : 0.0f;
          float gk = KIND == BT_NEURON_ALIF ? d.g_k[idx] : 0.0f;
          const NeuronParams prm = load_params<KIND, USE_REF>(d.neuron, i);
          const NeuronOut o = neuron_update<KIND, HARD, USE_REF, true>(prm, I, v, ref, gk);
          s = o.spike;
          d.v[idx] = v;
          if (USE_REF) d.refractory[idx] = ref;
          if (KIND == BT_NEURON_ALIF) d.g_k[idx] = gk;
        }
        if constexpr (!REC) {
          d.psc[idx] = P;
          if (d.psc_trace && k > 0) d.psc_trace[((k - 1) * B) * n + idx] = P;
        } else {
          for (int r = 0; r < C; ++r) {
            d.psc[c0 + r] = Pr[r];
            if (d.psc_trace && k > 0) d.psc_trace[((k - 1) * B) * n * C + c0 + r] = Pr[r];
          }
        }
        if (d.v_trace) d.v_trace[(k * B) * n + idx] = d.v[idx];
        if (USE_REF && d.ref_trace) d.ref_trace[(k * B) * n + idx] = d.refractory[idx];
        if (KIND == BT_NEURON_ALIF && d.gk_trace) d.gk_trace[(k * B) * n + idx] = d.g_k[idx];
        if (d.spikes) d.spikes[(k * B) * n + idx] = s;
        if (s != 0.0f) {
          atomicOr(&sbits[b], 1u << (i & 31));
          ++nspk;
        }
      }
    }
  }
  __shared__ long long s_stat[32][3];  // per warp: union, events, edges
  if (d.stats && lane == 0) {
    const long long deg = (i < n && nspk && d.outdeg) ? d.outdeg[i] : 0;
    s_stat[wid][0] = nspk ? 1 : 0;
    s_stat[wid][1] = nspk * deg;
    s_stat[wid][2] = nspk ? deg : 0;
  }
  __syncthreads();
  if (d.stats && threadIdx.x < 3) {
    // one atomic per block and counter (same-address atomics serialise in L2)
    long long tot = 0;
    for (int q = 0; q < 32; ++q) tot += s_stat[q][threadIdx.x];
    if (tot) atomicAdd(reinterpret_cast<unsigned long long*>(d.stats + k * 4 + threadIdx.x), (unsigned long long)tot);
  }
  const int64_t w = int64_t(blockIdx.x);
  for (int64_t b = threadIdx.x; b < B; b += blockDim.x) {
    d.hist[(int64_t(si.h_t) * B + b) * words + w] = sbits[b];
    if (d.raster) d.raster[(k * B + b) * words + w] = sbits[b];
  }
}

// Synapse update of the last step of a call: psc_{t_end-1}.
__global__ void __launch_bounds__(1024) k_eng_gather_final(bt_engine_desc d, StepIdx si) {
  const int64_t n = d.n, B = d.batch;
  const int64_t words = (n + 31) >> 5;
  const int64_t k = d.n_steps - 1;
  const int64_t i = int64_t(blockIdx.x) * 32 + (threadIdx.x >> 5);
  if (i >= n) return;
  const int C = n_rec(d);
  const int64_t nc = n * C;
  for (int64_t b = 0; b < B; ++b) {
    const int64_t len = d.sample_len ? d.sample_len[b] : INT64_MAX;
    for (int r = 0; r < C; ++r) {
      const int64_t col = i * C + r, idx = b * nc + col;  // PSC column
      if (k >= len) {
        if (lane_id() == 0 && d.psc_trace) d.psc_trace[(k * B) * nc + idx] = d.psc[idx];
        continue;
      }
      const float wz = gather_in(d, col, b, si.h_t, words);
      if (lane_id() == 0) {
        const float P = add(psc_decay(d.psc_coef, d.psc_tau, col, d.psc[idx]), wz);
        d.psc[idx] = P;
        if (d.psc_trace) d.psc_trace[(k * B) * nc + idx] = P;
      }
    }
  }
}

// ------------------------------------------------------------ sliced pull --
//
// PULL mode, one launch per step for batched runs.  Warp = (slice of 32 posts,
// 32-sample word q); lane = post.  The warp walks the slice's SELL-32 rows
// (each post's in-edges in canonical order down its lane), looks up the
// presynaptic neuron's sample mask for the step the edge's delay bin points
// at, and adds w into acc[sample][lane] in shared memory -- conflict-free and
// in ascending in-edge order for every (sample, post), i.e. the reference's
// fma chain (acc + w == fma(w, 1, acc)).  Then each lane runs the neuron
// update of its post for the warp's 32 samples and publishes its new mask.
constexpr int kPullWarps = 8;
constexpr int kPullUnroll = 8;

template <int MW>
struct MaskVec;
template <>
struct MaskVec<1> {
  using T = uint32_t;
  __device__ static void split(T v, uint32_t* m) { m[0] = v; }
};
template <>
struct MaskVec<2> {
  using T = uint2;
  __device__ static void split(T v, uint32_t* m) { m[0] = v.x; m[1] = v.y; }
};
template <>
struct MaskVec<4> {
  using T = uint4;
  __device__ static void split(T v, uint32_t* m) { m[0] = v.x; m[1] = v.y; m[2] = v.z; m[3] = v.w; }
};

// MW: sample words a warp covers (1, 2 or 4 -> batch up to 32, 64, 128).  For
// larger batches MW = 1 and the grid has one warp per (slice, word): `split`.
template <int KIND, bool HARD, bool USE_REF, bool FINAL, int MW>
__global__ void __launch_bounds__(kPullWarps * 32, 3) k_eng_pull(bt_engine_desc d, int64_t k, int split, StepIdx si) {
  extern __shared__ float acc_dyn[];  // [kPullWarps][MW * 32][32]
  const int wid = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int64_t n = d.n, B = d.batch;
  const int mw_all = mask_stride(B);
  const int64_t n_slices = (n + 31) >> 5;
  const int64_t gw = int64_t(blockIdx.x) * kPullWarps + wid;
  const int64_t sl = split ? gw / mw_all : gw;
  const int q0 = split ? int(gw % mw_all) : 0;  // first sample word of this warp
  if (sl >= n_slices) return;  // warp-uniform; the kernel has no block barrier
  const int64_t p = sl * 32 + lane;
  const bool valid = p < n;
  const int H = d.hist_len;
  // history slot of the arrival step whose PSC this launch completes
  const int ta_mod_h = FINAL ? si.h_t : si.h_prev;
  const bool gather = FINAL || k > 0;
  float(*acc)[32] = reinterpret_cast<float(*)[32]>(acc_dyn + wid * (MW * 32 * 32));
  using V = typename MaskVec<MW>::T;
  const int64_t row_stride = int64_t(n + 1) * mw_all;  // words per history slot
  if (gather) {
#pragma unroll 8
    for (int l = 0; l < MW * 32; ++l) acc[l][lane] = 0.0f;
    __syncwarp();
    const int64_t r0 = d.sl_ptr[sl], r1 = d.sl_ptr[sl + 1];
    const uint32_t sentinel = uint32_t(n);
    for (int64_t r = r0; r < r1; r += kPullUnroll) {
      uint32_t src[kPullUnroll];
      float w[kPullUnroll];
      V mv[kPullUnroll];
#pragma unroll
      for (int u = 0; u < kPullUnroll; ++u) {
        const bool in = r + u < r1;
        src[u] = in ? __ldg(d.sl_src + (r + u) * 32 + lane) : sentinel;
        w[u] = in ? __ldg(d.sl_w + (r + u) * 32 + lane) : 0.0f;
      }
#pragma unroll
      for (int u = 0; u < kPullUnroll; ++u) {
        int slot = ta_mod_h - int(src[u] >> BT_BIN_SHIFT);
        if (slot < 0) slot += H;
        const uint32_t* mrow = d.masks + slot * row_stride + int64_t(src[u] & kIdMask) * mw_all + q0;
        mv[u] = __ldg(reinterpret_cast<const V*>(mrow));
      }
#pragma unroll
      for (int u = 0; u < kPullUnroll; ++u) {
        uint32_t m[MW];
        MaskVec<MW>::split(mv[u], m);
#pragma unroll
        for (int q = 0; q < MW; ++q) {
          uint32_t mm = m[q];
          while (mm) {
            const int l = __ffs(mm) - 1;
            mm &= mm - 1;
            acc[q * 32 + l][lane] = add(acc[q * 32 + l][lane], w[u]);
          }
        }
      }
    }
    __syncwarp();
  }
  const int64_t words = n_slices;
  uint32_t my_mask[MW];
#pragma unroll
  for (int q = 0; q < MW; ++q) my_mask[q] = 0;
  constexpr int U = 4;
  const float* __restrict__ xk = d.x ? d.x + (k * B) * n : nullptr;
  const NeuronParams prm = load_params<KIND, USE_REF>(d.neuron, valid ? p : 0);
  const float pc = ld(d.psc_coef, valid ? p : 0), pt = ld(d.psc_tau, valid ? p : 0), rpt = pow2_recip(pt);
#pragma unroll
  for (int q = 0; q < MW; ++q) {
    for (int l0 = 0; l0 < 32; l0 += U) {
      const int64_t b0 = int64_t(q0 + q) * 32 + l0;
      if (b0 >= B) break;  // warp-uniform
      // load phase: U samples' state at once (independent loads in flight)
      float pv[U], xv[U], vv[U], rv[U], gv[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int64_t b = b0 + u;
        const bool in = valid && b < B;
        const int64_t idx = b * n + p;
        pv[u] = in ? d.psc[idx] : 0.0f;
        xv[u] = (in && xk && !FINAL) ? xk[idx] : 0.0f;
        vv[u] = (in && !FINAL) ? d.v[idx] : 0.0f;
        rv[u] = (in && USE_REF && !FINAL) ? d.refractory[idx] : 0.0f;
        gv[u] = (in && KIND == BT_NEURON_ALIF && !FINAL) ? d.g_k[idx] : 0.0f;
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int64_t b = b0 + u;
        if (b >= B) break;  // warp-uniform
        const int l = l0 + u;
        float spk = 0.0f;
        if (valid) {
          const int64_t idx = b * n + p;
          const int64_t len = d.sample_len ? d.sample_len[b] : INT64_MAX;
          float P = pv[u];
          const bool syn_live = FINAL ? (k < len) : (k - 1 < len);
          if (gather && syn_live) P = add(psc_decay(pc, pt, rpt, P), acc[q * 32 + l][lane]);
          if (FINAL) {
            d.psc[idx] = P;
            if (d.psc_trace) d.psc_trace[(k * B) * n + idx] = P;
            continue;
          }
          float v = vv[u], ref = rv[u], gk = gv[u];
          if (k < len) {
            const float I = xk ? add(P, xv[u]) : P;
            const NeuronOut o = neuron_update<KIND, HARD, USE_REF, true>(prm, I, v, ref, gk);
            spk = o.spike;
            d.v[idx] = v;
            if (USE_REF) d.refractory[idx] = ref;
            if (KIND == BT_NEURON_ALIF) d.g_k[idx] = gk;
          }
          d.psc[idx] = P;
          if (d.v_trace) d.v_trace[(k * B) * n + idx] = v;
          if (USE_REF && d.ref_trace) d.ref_trace[(k * B) * n + idx] = ref;
          if (KIND == BT_NEURON_ALIF && d.gk_trace) d.gk_trace[(k * B) * n + idx] = gk;
          if (d.psc_trace && k > 0) d.psc_trace[((k - 1) * B) * n + idx] = P;
          if (d.spikes) d.spikes[(k * B) * n + idx] = spk;
        }
        if (!FINAL) {
          const uint32_t word = __ballot_sync(0xffffffffu, spk != 0.0f);
          if (lane == 0 && d.raster) d.raster[(k * B + b) * words + sl] = word;
          if (spk != 0.0f) my_mask[q] |= 1u << l;
        }
      }
    }
  }
  if (FINAL) return;
  if (valid) {
    uint32_t* mrow = d.masks + int64_t(si.h_t) * row_stride + p * mw_all + q0;
#pragma unroll
    for (int q = 0; q < MW; ++q) mrow[q] = my_mask[q];
  }
  if (d.stats) {
    // events = spikes x out-degree; union counted by the warp that owns word 0
    int nspk = 0;
#pragma unroll
    for (int q = 0; q < MW; ++q) nspk += __popc(my_mask[q]);
    const int deg = (valid && d.outdeg) ? d.outdeg[p] : 0;
    long long ev = (long long)nspk * deg;
    long long ed = (!split && nspk) ? deg : 0;
    long long un = (!split && nspk) ? 1 : 0;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      ev += __shfl_xor_sync(0xffffffffu, ev, off);
      ed += __shfl_xor_sync(0xffffffffu, ed, off);
      un += __shfl_xor_sync(0xffffffffu, un, off);
    }
    if (lane == 0) {
      if (ev) atomicAdd(reinterpret_cast<unsigned long long*>(d.stats + k * 4 + 1), (unsigned long long)ev);
      if (ed) atomicAdd(reinterpret_cast<unsigned long long*>(d.stats + k * 4 + 2), (unsigned long long)ed);
      if (un) atomicAdd(reinterpret_cast<unsigned long long*>(d.stats + k * 4 + 0), (unsigned long long)un);
    }
  }
}

// masks[i][q] bit l  <=>  in[(32 q + l) * n + i] != 0   (sample-minor from [B][n]).
__global__ void k_float_to_masks(int64_t batch, int64_t n, const float* __restrict__ in, uint32_t* __restrict__ masks) {
  const int64_t idx = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  const int mw = mask_stride(batch);
  if (idx >= n * mw) return;
  const int64_t i = idx / mw;
  const int q = int(idx % mw);
  uint32_t m = 0;
  for (int l = 0; l < 32 && int64_t(q) * 32 + l < batch; ++l)
    if (in[(int64_t(q) * 32 + l) * n + i] != 0.0f) m |= 1u << l;
  masks[idx] = m;
}

__global__ void k_masks_to_float(int64_t batch, int64_t n, const uint32_t* __restrict__ masks, float* __restrict__ out) {
  const int64_t idx = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (idx >= batch * n) return;
  const int64_t b = idx / n, i = idx % n;
  const int mw = mask_stride(batch);
  out[idx] = float((masks[i * mw + (b >> 5)] >> (b & 31)) & 1u);
}

// ---------------------------------------------------------- run priming --

// One thread per (steps ago a in 1..bin_hi, neuron i): the spike set of step
// t0 - a rebuilt from the history bitmaps -- the mask of samples in which i
// spiked, and i listed once if any did (warp-aggregated atomic).  Rows are
// padded to whole 32-neuron words, so every warp has a single a.
__global__ void k_prime_history(bt_engine_desc d) {
  const int64_t n = d.n, B = d.batch;
  const int64_t words = (n + 31) >> 5;
  const int64_t npad = words * 32;
  const int64_t gid = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  const int64_t a = 1 + gid / npad;
  const int64_t i = gid - (a - 1) * npad;
  if (a > d.bin_hi) return;  // whole warps
  const int64_t s = d.t0 - a;  // >= 0: t0 >= hist_len > n_bins > bin_hi
  const int64_t hs = s % d.hist_len;
  const int q = int(s % (d.n_bins + 1));
  const ScatterScratch ws = scatter_scratch(d, q);
  uint32_t mw[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  bool any = false;
  if (i < n) {
    const uint32_t* h = d.hist + hs * B * words + (i >> 5);
    for (int64_t b = 0; b < B; ++b) {
      if ((h[b * words] >> (i & 31)) & 1u) {
        mw[b >> 5] |= 1u << (b & 31);
        any = true;
      }
    }
    if (any) {
#pragma unroll
      for (int w = 0; w < 8; ++w)
        if (w < ws.ms) ws.mask[i * ws.ms + w] = mw[w];
      ws.flag[i] = 1;
    }
  }
  const unsigned lane = lane_id();
  const uint32_t fb = __ballot_sync(0xffffffffu, any);
  if (fb == 0) return;
  const int sub = int((i - lane) >> ws.cap_shift);
  int32_t base = 0;
  if (lane == 0) base = atomicAdd(ws.count + sub, __popc(fb));
  base = __shfl_sync(0xffffffffu, base, 0);
  if (any) ws.list[sub * ws.cap + base + __popc(fb & ((1u << lane) - 1u))] = int32_t(i);
}

// ------------------------------------------------------- input projection --

// Per row r: its nonzero inputs as (channel, value) pairs in ascending channel
// order (warp ballot + prefix), and their count.  With live_len, row
// r = t * batch + b of a sample past its length (t >= live_len[b]) gets
// count -1 and no pairs: nothing reads its projection.
__global__ void k_row_pairs(int64_t rows, int64_t c_in, const float* __restrict__ xin, int32_t* __restrict__ cnt,
                            int2* __restrict__ pairs, const int32_t* __restrict__ live_len, int64_t batch) {
  const int64_t r = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  if (r >= rows) return;
  const unsigned lane = lane_id();
  if (live_len && r / batch >= __ldg(live_len + r % batch)) {  // warp-uniform
    if (lane == 0) cnt[r] = -1;
    return;
  }
  int32_t total = 0;
  for (int64_t c0 = 0; c0 < c_in; c0 += 32) {
    const int64_t c = c0 + lane;
    const float v = c < c_in ? xin[r * c_in + c] : 0.0f;
    const bool nz = v != 0.0f;
    const uint32_t m = __ballot_sync(0xffffffffu, nz);
    if (nz) pairs[r * c_in + total + __popc(m & ((1u << lane) - 1u))] = make_int2(int(c), __float_as_int(v));
    total += __popc(m);
  }
  if (lane == 0) cnt[r] = total;
}

// out[r][i] = sum over the row's pairs (ascending channel) of v * w_t[c][i],
// as an fmaf chain (+ bias).  Each thread owns kProjNPT neurons spaced by the
// block size, so one broadcast pair load feeds kProjNPT coalesced weight loads
// and fmas.  grid.x walks row blocks fastest: the resident blocks then share a
// narrow column slice of w_t, which stays in L2.
constexpr int kProjRows = 8;
constexpr int kProjNPT = 4;
__global__ void __launch_bounds__(256) k_input_project(int64_t rows, int64_t c_in, int64_t n,
                                                       const float* __restrict__ w_t,
                                                       const float* __restrict__ bias,
                                                       const int32_t* __restrict__ cnt,
                                                       const int2* __restrict__ pairs, float* __restrict__ out) {
  const int64_t tile = int64_t(blockIdx.y) * (256 * kProjNPT);
  const int64_t r0 = int64_t(blockIdx.x) * kProjRows;
  int64_t ii[kProjNPT];
  bool ok[kProjNPT];
#pragma unroll
  for (int j = 0; j < kProjNPT; ++j) {
    ii[j] = tile + threadIdx.x + j * 256;
    ok[j] = ii[j] < n;
  }
  for (int64_t r = r0; r < r0 + kProjRows && r < rows; ++r) {
    const int32_t c_n = cnt[r];
    if (c_n < 0) continue;  // a finished sample's step: left unwritten
    const int2* rp = pairs + r * c_in;
    float acc[kProjNPT];
#pragma unroll
    for (int j = 0; j < kProjNPT; ++j) acc[j] = 0.0f;
    for (int32_t q = 0; q < c_n; ++q) {
      const int2 pr = __ldg(rp + q);
      const float v = __int_as_float(pr.y);
      const float* wr = w_t + int64_t(pr.x) * n;
#pragma unroll
      for (int j = 0; j < kProjNPT; ++j)
        if (ok[j]) acc[j] = fmaf(v, __ldg(wr + ii[j]), acc[j]);
    }
#pragma unroll
    for (int j = 0; j < kProjNPT; ++j)
      if (ok[j]) out[r * n + ii[j]] = bias ? add(acc[j], bias[ii[j]]) : acc[j];
  }
}

// Per channel c, the rows r (ascending) whose input x[r][c] is nonzero, and
// their count: one warp per channel (ballot + prefix keeps the order).
__global__ void k_channel_rows(int64_t rows, int64_t c_in, const float* __restrict__ x, int32_t* __restrict__ lists,
                               int32_t* __restrict__ counts) {
  const int64_t c = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  if (c >= c_in) return;
  const unsigned lane = lane_id();
  int32_t total = 0;
  for (int64_t r0 = 0; r0 < rows; r0 += 32) {
    const int64_t r = r0 + lane;
    const bool nz = r < rows && x[r * c_in + c] != 0.0f;
    const uint32_t m = __ballot_sync(0xffffffffu, nz);
    if (nz) lists[c * rows + total + __popc(m & ((1u << lane) - 1u))] = int32_t(r);
    total += __popc(m);
  }
  if (lane == 0) counts[c] = total;
}

// Gradient of the input layer's weight (w_t [c_in][n]) from the gradient of
// its projection g [rows][n]: out[c][i] = sum over the rows r of channel c
// (ascending) of x[r][c] * g[r][i] -- an fmaf chain over the nonzero inputs
// only; accumulate adds it to out.  Block = (channel, 1024 columns), each
// thread kProjNPT columns spaced by the block size (coalesced rows of g).
__global__ void __launch_bounds__(256) k_input_grad_weight(int64_t rows, int64_t c_in, int64_t n,
                                                           const float* __restrict__ x, const float* __restrict__ g,
                                                           const int32_t* __restrict__ lists,
                                                           const int32_t* __restrict__ counts,
                                                           float* __restrict__ out, int accumulate) {
  const int64_t c = blockIdx.x;
  const int64_t tile = int64_t(blockIdx.y) * (256 * kProjNPT);
  const int32_t cnt = counts[c];
  const int32_t* rl = lists + c * rows;
  float acc[kProjNPT];
#pragma unroll
  for (int j = 0; j < kProjNPT; ++j) acc[j] = 0.0f;
  for (int32_t q = 0; q < cnt; ++q) {
    const int64_t r = __ldg(rl + q);
    const float xv = __ldg(x + r * c_in + c);
    const float* gr = g + r * n;
#pragma unroll
    for (int j = 0; j < kProjNPT; ++j) {
      const int64_t i = tile + threadIdx.x + j * 256;
      if (i < n) acc[j] = fmaf(xv, __ldg(gr + i), acc[j]);
    }
  }
#pragma unroll
  for (int j = 0; j < kProjNPT; ++j) {
    const int64_t i = tile + threadIdx.x + j * 256;
    if (i < n) out[c * n + i] = accumulate ? add(out[c * n + i], acc[j]) : acc[j];
  }
}

// --------------------------------------------------------------- bitmaps --

__global__ void k_bits_to_float(int64_t rows, int64_t n, const uint32_t* __restrict__ bits, float* __restrict__ out) {
  const int64_t idx = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (idx >= rows * n) return;
  const int64_t r = idx / n, i = idx % n;
  const int64_t words = (n + 31) >> 5;
  out[idx] = float((bits[r * words + (i >> 5)] >> (i & 31)) & 1u);
}

__global__ void k_float_to_bits(int64_t rows, int64_t n, const float* __restrict__ in, uint32_t* __restrict__ bits) {
  const int64_t words = (n + 31) >> 5;
  const int64_t gw = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  if (gw >= rows * words) return;
  const int64_t r = gw / words, w = gw % words;
  const int64_t i = w * 32 + lane_id();
  const bool nz = i < n && in[r * n + i] != 0.0f;
  const uint32_t m = __ballot_sync(0xffffffffu, nz);
  if (lane_id() == 0) bits[gw] = m;
}

}  // namespace bt

using namespace bt;

namespace bt {
int run_tile(const bt_engine_desc& d, bool fast, cudaStream_t s);     // tile.cu
int run_cluster(const bt_engine_desc& d, bool fast, cudaStream_t s);  // cluster.cu
}

namespace {

int engine_check(const bt_engine_desc* d) {
  if (!d) return bt_set_error(BT_ERR_INVALID, "null engine descriptor");
  if (int st = bt_check_neuron_desc(&d->neuron)) return st;
  BT_CHECK_ARG(d->n > 0 && d->n < BT_MAX_NEURONS, "n=%lld outside (0, 2^25)", (long long)d->n);
  BT_CHECK_ARG(d->batch > 0 && d->batch * d->n < (int64_t(1) << 40), "bad batch");
  BT_CHECK_ARG(d->n_bins >= 1 && d->n_bins <= BT_MAX_BINS, "n_bins=%d outside [1, 128]", d->n_bins);
  BT_CHECK_ARG(d->hist_len >= d->n_bins + 2, "hist_len=%d must be >= n_bins + 2", d->hist_len);
  BT_CHECK_ARG(d->n_steps >= 0 && d->t0 >= 0, "negative step index");
  BT_CHECK_ARG(d->n_steps < (int64_t(1) << 31), "n_steps must be below 2^31");
  BT_CHECK_ARG(d->mode == BT_MODE_SCATTER || d->mode == BT_MODE_GATHER || d->mode == BT_MODE_PULL ||
                   d->mode == BT_MODE_TILE || d->mode == BT_MODE_CLUSTER,
               "mode=%d", d->mode);
  BT_CHECK_ARG(d->v && d->psc && d->hist, "state pointer missing (v / psc / hist)");
  BT_CHECK_ARG(!d->neuron.use_refractory || d->refractory, "refractory state missing");
  BT_CHECK_ARG(d->neuron.kind != BT_NEURON_ALIF || d->g_k, "g_k state missing");
  BT_CHECK_ARG(d->psc_coef.ptr && d->psc_tau.ptr, "PSC coefficients missing");
  BT_CHECK_ARG(d->neuron.spiking, "the fused engine needs a spiking (Heaviside) forward");
  BT_CHECK_ARG(d->n_rec >= 0 && d->n_rec <= kMaxRec, "n_rec=%d outside [0, %d]", d->n_rec, kMaxRec);
  BT_CHECK_ARG(d->n * n_rec(*d) < BT_MAX_NEURONS, "n * n_rec must be < 2^25");
  BT_CHECK_ARG(n_rec(*d) == 1 || d->mode != BT_MODE_PULL, "pull mode has no receptor channels");
  if (d->mode == BT_MODE_SCATTER) {
    BT_CHECK_ARG(d->csr_ptr && d->csr_edges && d->ring && d->work, "scatter needs CSR, ring and work");
    BT_CHECK_ARG((reinterpret_cast<uintptr_t>(d->csr_edges) & 15) == 0, "csr_edges must be 16-byte aligned");
    BT_CHECK_ARG(d->bin_lo >= 0 && d->bin_lo <= d->bin_hi && d->bin_hi < d->n_bins, "bins [%d, %d] outside [0, %d)",
                 d->bin_lo, d->bin_hi, d->n_bins);
    BT_CHECK_ARG(d->scatter_lanes == 0 || d->scatter_lanes == 1 || d->scatter_lanes == 8 || d->scatter_lanes == 32,
                 "scatter_lanes=%d (0, 1, 8 or 32)", d->scatter_lanes);
    BT_CHECK_ARG(mask_stride(d->batch) <= 8, "scatter mode supports up to 256 samples");
    BT_CHECK_ARG(d->batch * d->n * n_rec(*d) < (int64_t(1) << 31), "scatter mode needs batch * n * n_rec < 2^31");
    BT_CHECK_ARG(d->dense_rows == 0 || (d->bin_lo == d->bin_hi && d->sl_ptr && d->sl_src && d->sl_w),
                 "dense delivery needs a single delay bin and the sliced in-edge view");
    BT_CHECK_ARG(d->neuron_spt == 0 || d->neuron_spt == 1 || d->neuron_spt == 2 || d->neuron_spt == 4,
                 "neuron_spt=%d (0, 1, 2 or 4)", d->neuron_spt);
  } else if (d->mode == BT_MODE_TILE) {
    BT_CHECK_ARG(d->csr_ptr && d->csr_edges && d->ring && d->tile_off && d->tile_work,
                 "tile mode needs CSR, ring, tile offsets and tile work");
    BT_CHECK_ARG((reinterpret_cast<uintptr_t>(d->tile_work) & 63) == 0, "tile_work must be 64-byte aligned");
    BT_CHECK_ARG((reinterpret_cast<uintptr_t>(d->csr_edges) & 15) == 0, "csr_edges must be 16-byte aligned");
    BT_CHECK_ARG(d->n_bins == 1 && d->bin_lo == 0 && d->bin_hi == 0, "tile mode has no synaptic delays");
    BT_CHECK_ARG(n_rec(*d) == 1, "tile mode has no receptor channels");
    BT_CHECK_ARG(d->tile_posts > 0 && (d->tile_posts & 31) == 0, "tile_posts=%d must be a positive multiple of 32",
                 d->tile_posts);
    BT_CHECK_ARG(d->n_tiles > 0 && int64_t(d->n_tiles) * d->tile_posts >= d->n &&
                     int64_t(d->n_tiles - 1) * d->tile_posts < d->n,
                 "n_tiles=%d x tile_posts=%d does not tile n=%lld", d->n_tiles, d->tile_posts, (long long)d->n);
    BT_CHECK_ARG(d->batch <= 256 && d->batch * d->n < (int64_t(1) << 31), "tile mode: batch <= 256, batch * n < 2^31");
  } else if (d->mode == BT_MODE_CLUSTER) {
    BT_CHECK_ARG(d->cl_w && d->cl_src && d->cl_gptr, "cluster mode needs the packed in-edges cl_w / cl_src / cl_gptr");
    BT_CHECK_ARG(((reinterpret_cast<uintptr_t>(d->cl_w) | reinterpret_cast<uintptr_t>(d->cl_src)) & 15) == 0,
                 "cl_w and cl_src must be 16-byte aligned (bulk copies)");
    BT_CHECK_ARG(d->n_bins >= 1 && d->n_bins <= 32 && (d->n_bins == 1 || d->n + 32 <= (int64_t(1) << 20)),
                 "cluster mode: n_bins=%d (1..32; with delays n + 32 <= 2^20)", d->n_bins);
    BT_CHECK_ARG(d->tile_rows >= 0 && d->tile_rows % 16 == 0 && d->tile_rows < (int64_t(1) << 24),
                 "tile_rows=%lld must be a multiple of 16", (long long)d->tile_rows);
    BT_CHECK_ARG(n_rec(*d) == 1, "cluster mode has no receptor channels");
    BT_CHECK_ARG(d->tile_posts > 0 && (d->tile_posts & 31) == 0, "tile_posts=%d must be a positive multiple of 32",
                 d->tile_posts);
    BT_CHECK_ARG(d->n_tiles >= 1 && d->n_tiles <= 16 && int64_t(d->n_tiles) * d->tile_posts >= d->n &&
                     int64_t(d->n_tiles - 1) * d->tile_posts < d->n,
                 "n_tiles=%d (1..16) x tile_posts=%d does not tile n=%lld", d->n_tiles, d->tile_posts,
                 (long long)d->n);
    BT_CHECK_ARG(d->batch <= 256 && d->batch * d->n < (int64_t(1) << 31), "cluster mode: batch <= 256");
  } else if (d->mode == BT_MODE_GATHER) {
    BT_CHECK_ARG(d->csc_ptr && d->csc_src && d->csc_w, "gather needs CSC");
  } else {
    BT_CHECK_ARG(d->sl_ptr && d->sl_src && d->sl_w && d->masks, "pull needs the sliced layout and masks");
  }
  return BT_OK;
}

// The device's Div kind of divisor c (neuron.cuh make_div) is 1 or 2.
bool fast_divisor(float c, bool verified) {
  uint32_t u;
  std::memcpy(&u, &c, sizeof(u));
  const uint32_t e = u >> 23;
  return ((u & 0x7fffffu) == 0u && e >= 1u && e <= 253u) || verified;
}

// Uniform scalar parameters whose divisions all avoid the IEEE path.
bool fast_divisors(const bt_engine_desc& d, int kind) {
  const bt_neuron_desc& nd = d.neuron;
  if (!nd.uniform || !d.psc_uniform) return false;
  const float den = nd.sv[0] - nd.sv[1];  // v_threshold - v_reset, as the device computes it
  bool ok = fast_divisor(nd.sv[2], nd.fast_div & 1) && fast_divisor(den, nd.fast_div & 2) &&
            fast_divisor(d.psc_tau_s, d.psc_fast_div != 0);
  ok = ok && (kind == BT_NEURON_LIF ? fast_divisor(nd.sv[3], nd.fast_div & 4) : fast_divisor(nd.sv[9], nd.fast_div & 8));
  return ok;
}

// The arrays the scatter neuron step touches admit 16-byte accesses.
bool vec_neurons(const bt_engine_desc& d, const float* z_given) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(d.v) | reinterpret_cast<uintptr_t>(d.psc) |
                      reinterpret_cast<uintptr_t>(d.refractory) | reinterpret_cast<uintptr_t>(d.g_k) |
                      reinterpret_cast<uintptr_t>(d.ring) | reinterpret_cast<uintptr_t>(d.x) |
                      reinterpret_cast<uintptr_t>(d.spikes) | reinterpret_cast<uintptr_t>(d.v_trace) |
                      reinterpret_cast<uintptr_t>(d.psc_trace) | reinterpret_cast<uintptr_t>(d.ref_trace) |
                      reinterpret_cast<uintptr_t>(d.gk_trace) | reinterpret_cast<uintptr_t>(z_given);
  return d.n % 4 == 0 && (a & 15) == 0 && d.batch < 65536;
}

template <int KIND, bool HARD, bool USE_REF>
int run_typed(const bt_engine_desc& d, const float* z_given, cudaStream_t s) {
  const int64_t n = d.n;
  if (d.mode == BT_MODE_CLUSTER) return run_cluster(d, fast_divisors(d, KIND), s);  // no final launch
  if (d.mode == BT_MODE_TILE) {
    if (int st = run_tile(d, fast_divisors(d, KIND), s)) return st;
    k_eng_scatter_final<<<int(ceil_div(d.batch * n, 256)), 256, 0, s>>>(d);
    BT_CHECK_LAUNCH("k_eng_scatter_final");
    return BT_OK;
  }
  if (d.mode == BT_MODE_SCATTER) {
    const int S = d.neuron_spt > 0 ? d.neuron_spt : 4;
    const dim3 grid(unsigned(ceil_div(n, kEngThreads)), unsigned(ceil_div(d.batch, S)));
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int planes = d.bin_hi - d.bin_lo + 1;
    const int ms = mask_stride(d.batch);
    // Shared memory of a block: the offsets of all planes (33 KB at 128 bins) beside the
    // 33 KB of a dense step's columns; from 60 planes on more than a kernel has without
    // an attribute, from 92 on three blocks fit an SM instead of four.
    const size_t ssmem = sizeof(int32_t) * size_t(planes * kSub + 1);
    const size_t sblock = ssmem + kScatterStatic + 1024;  // (1 KB of every block is the system's)
    // one wave of resident blocks, fewer when the step cannot list that many rows
    const int64_t rows_per_block = d.scatter_lanes == 1 ? 64 : d.scatter_lanes == 8 ? kEngThreads / 8 : kEngThreads / 32;
    const int64_t wave = int64_t(sms) * std::min<int64_t>(ms <= 4 ? 4 : 3, int64_t(228 * 1024 / sblock));
    const unsigned sgrid = unsigned(std::max<int64_t>(1, std::min(wave, ceil_div(n * planes, rows_per_block))));
    // every divisor a power of two or a verified reciprocal: no IEEE division compiled in
    const bool fast = fast_divisors(d, KIND);
    auto neuron = fast ? (S == 1 ? k_eng_neuron<KIND, HARD, USE_REF, 1, true>
                          : S == 2 ? k_eng_neuron<KIND, HARD, USE_REF, 2, true> : k_eng_neuron<KIND, HARD, USE_REF, 4, true>)
                       : (S == 1 ? k_eng_neuron<KIND, HARD, USE_REF, 1, false>
                          : S == 2 ? k_eng_neuron<KIND, HARD, USE_REF, 2, false> : k_eng_neuron<KIND, HARD, USE_REF, 4, false>);
    auto pick = [&](auto g) {
      constexpr int G = decltype(g)::value;
      // MS >= ms: mask_stride gives 1, 2, 4, or 5..8 words (MS = 8)
    return ms == 1 ? k_eng_scatter<G, 1> : ms == 2 ? k_eng_scatter<G, 2> : ms <= 4 ? k_eng_scatter<G, 4>
                                                                                      : k_eng_scatter<G, 8>;
    };
    auto scatter = d.scatter_lanes == 1   ? (ms == 1 ? k_eng_scatter_flat<1> : ms == 2 ? k_eng_scatter_flat<2>
                                             : ms <= 4 ? k_eng_scatter_flat<4> : k_eng_scatter_flat<8>)
                   : d.scatter_lanes == 8 ? pick(std::integral_constant<int, 8>())
                                          : pick(std::integral_constant<int, 32>());
    const int C = n_rec(d);
    const dim3 rgrid(unsigned(ceil_div(n, kEngThreads)), unsigned(d.batch));
    // vector access to the C channels of (b, i) needs 8 / 16-byte aligned state and acc
    const bool aligned = ((reinterpret_cast<uintptr_t>(d.psc) | reinterpret_cast<uintptr_t>(d.ring)) & 15) == 0;
    auto rec = C == 4 && aligned ? k_eng_neuron_rec<KIND, HARD, USE_REF, 4>
             : C == 2 && aligned ? k_eng_neuron_rec<KIND, HARD, USE_REF, 2> : k_eng_neuron_rec<KIND, HARD, USE_REF, 0>;
    const bool vec = C == 1 && vec_neurons(d, z_given);
    const dim3 vgrid(unsigned(ceil_div(n, 4 * kVecThreads)), unsigned(d.batch));
    auto nvec = fast ? k_eng_neuron_vec<KIND, HARD, USE_REF, true> : k_eng_neuron_vec<KIND, HARD, USE_REF, false>;
    const int parts = row_parts(d, z_given, vec, sms);
    auto rows = ms == 1 ? k_eng_scatter_rows<1> : ms == 2 ? k_eng_scatter_rows<2> : ms <= 4 ? k_eng_scatter_rows<4>
                                                                                             : k_eng_scatter_rows<8>;
    const int64_t columns = d.dense_rows > 0 ? int64_t(kRowWarps) * 32 * 32 : 0;
    const size_t rsmem = sizeof(float) * size_t(kRowList + std::max(n, columns));
    // dynamic shared memory beyond what a kernel has without asking: its range's most, once
    auto allow = [&](const void* kern, size_t most) {
      if (launch_setup_known(kern, dev, most, 1)) return int(BT_OK);
      if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(most)) != cudaSuccess)
        return bt_set_error(BT_ERR_CUDA, "shared memory request of %zu bytes refused", most);
      launch_setup_add(kern, dev, most, 1);
      return int(BT_OK);
    };
    if (parts) {
      if (int st = allow(reinterpret_cast<const void*>(rows), sizeof(float) * size_t(kRowList + kRowMaxN))) return st;
    } else if (ssmem + kScatterStatic > 48 * 1024) {
      if (int st = allow(reinterpret_cast<const void*>(scatter), sizeof(int32_t) * size_t(BT_MAX_BINS * kSub + 1))) return st;
    }
    for (int64_t k = 0; k < d.n_steps; ++k) {
      const StepIdx si = step_idx(d.t0 + k, d.n_bins, d.hist_len);
      // nothing runs on after a refused launch: the state would move on without its input
      cudaError_t e = C > 1 ? launch_step(k == 0, rec, rgrid, kEngThreads, 0, s, d, k, si)
                      : vec ? launch_step(k == 0, nvec, vgrid, kVecThreads, 0, s, d, int(k), si, scatter_scratch(d, si.q_t), z_given)
                            : launch_step(k == 0, neuron, grid, kEngThreads, 0, s, d, int(k), si, scatter_scratch(d, si.q_t), z_given);
      if (e == cudaSuccess)
        e = parts ? launch_step(false, rows, dim3(unsigned(d.batch * parts)), kRowThreads, rsmem, s, d, si, parts)
                  : launch_step(false, scatter, dim3(sgrid), kEngThreads, ssmem, s, d, k, si);
      if (e != cudaSuccess) break;
    }
    BT_CHECK_LAUNCH("k_eng_neuron/k_eng_scatter");
    if (d.n_steps > 0) {
      k_eng_scatter_final<<<int(ceil_div(d.batch * n * C, 256)), 256, 0, s>>>(d);
      BT_CHECK_LAUNCH("k_eng_scatter_final");
    }
  } else if (d.mode == BT_MODE_PULL) {
    // Words of the sample mask per warp: the descriptor may ask for 2 or 4
    // (fewer warps, one vector mask load per edge); by default every warp
    // takes one 32-sample word, which gives the most warps in flight.
    const int mw = mask_stride(d.batch);
    int MWT = d.pull_words_per_warp > 0 ? d.pull_words_per_warp : 1;
    if (MWT != 1 && MWT != mw) MWT = 1;
    const int split = MWT < mw ? 1 : 0;
    const int64_t warps = ceil_div(n, 32) * (split ? mw : 1);
    const int grid = int(ceil_div(warps, kPullWarps));
    const size_t smem = sizeof(float) * kPullWarps * MWT * 32 * 32;
#define BT_PULL_LAUNCH(M)                                                                                        \
  do {                                                                                                           \
    auto kern = k_eng_pull<KIND, HARD, USE_REF, false, M>;                                                      \
    auto kfin = k_eng_pull<KIND, HARD, USE_REF, true, M>;                                                       \
    if (smem > 48 * 1024 &&                                                                                      \
        (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) != cudaSuccess ||    \
         cudaFuncSetAttribute(kfin, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) != cudaSuccess))     \
      return bt_set_error(BT_ERR_CUDA, "shared memory request of %zu bytes refused", smem);                     \
    for (int64_t k = 0; k < d.n_steps; ++k)                                                                     \
      kern<<<grid, kPullWarps * 32, smem, s>>>(d, k, split, step_idx(d.t0 + k, d.n_bins, d.hist_len));          \
    BT_CHECK_LAUNCH("k_eng_pull");                                                                               \
    kfin<<<grid, kPullWarps * 32, smem, s>>>(d, d.n_steps - 1, split,                                           \
                                             step_idx(d.t0 + d.n_steps - 1, d.n_bins, d.hist_len));              \
    BT_CHECK_LAUNCH("k_eng_pull final");                                                                         \
  } while (0)
    if (d.n_steps > 0) {
      if (MWT == 1) BT_PULL_LAUNCH(1);
      else if (MWT == 2) BT_PULL_LAUNCH(2);
      else BT_PULL_LAUNCH(4);
    }
#undef BT_PULL_LAUNCH
  } else {
    const int grid = int(ceil_div(n, 32));
    const size_t smem = sizeof(uint32_t) * size_t(d.batch);
    BT_CHECK_ARG(smem <= 48 * 1024, "batch too large for the gather engine");
    auto gather = n_rec(d) > 1 ? k_eng_gather<KIND, HARD, USE_REF, true> : k_eng_gather<KIND, HARD, USE_REF, false>;
    for (int64_t k = 0; k < d.n_steps; ++k)
      gather<<<grid, 1024, smem, s>>>(d, k, step_idx(d.t0 + k, d.n_bins, d.hist_len));
    BT_CHECK_LAUNCH("k_eng_gather");
    if (d.n_steps > 0) {
      k_eng_gather_final<<<grid, 1024, 0, s>>>(d, step_idx(d.t0 + d.n_steps - 1, d.n_bins, d.hist_len));
      BT_CHECK_LAUNCH("k_eng_gather_final");
    }
  }
  return BT_OK;
}

}  // namespace

namespace {
int engine_run(const bt_engine_desc* d, const float* z_given, void* stream) {
  if (int st = engine_check(d)) return st;
  if (d->n_steps == 0) return BT_OK;
  if (d->stats && cudaMemsetAsync(d->stats, 0, sizeof(int64_t) * 4 * size_t(d->n_steps),
                                  static_cast<cudaStream_t>(stream)) != cudaSuccess)
    return bt_set_error(BT_ERR_CUDA, "memset failed");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const bool h = d->neuron.hard_reset != 0, r = d->neuron.use_refractory != 0;
  if (d->neuron.kind == BT_NEURON_LIF) {
    if (h && r) return run_typed<BT_NEURON_LIF, true, true>(*d, z_given, s);
    if (h) return run_typed<BT_NEURON_LIF, true, false>(*d, z_given, s);
    if (r) return run_typed<BT_NEURON_LIF, false, true>(*d, z_given, s);
    return run_typed<BT_NEURON_LIF, false, false>(*d, z_given, s);
  }
  if (h && r) return run_typed<BT_NEURON_ALIF, true, true>(*d, z_given, s);
  if (h) return run_typed<BT_NEURON_ALIF, true, false>(*d, z_given, s);
  if (r) return run_typed<BT_NEURON_ALIF, false, true>(*d, z_given, s);
  return run_typed<BT_NEURON_ALIF, false, false>(*d, z_given, s);
}
}  // namespace

extern "C" int bt_engine_run(const bt_engine_desc* d, void* stream) { return engine_run(d, nullptr, stream); }

extern "C" int bt_engine_run_given(const bt_engine_desc* d, const float* spikes, void* stream) {
  if (spikes && d && (d->mode != BT_MODE_SCATTER || d->n_rec > 1))
    return bt_set_error(BT_ERR_UNSUPPORTED, "given spikes need the scatter mode without receptor channels");
  return engine_run(d, spikes, stream);
}

extern "C" int bt_engine_prime(const bt_engine_desc* d, void* stream) {
  if (int st = engine_check(d)) return st;
  if (d->mode != BT_MODE_SCATTER) return BT_OK;
  BT_CHECK_ARG(d->t0 >= d->hist_len, "t0=%lld must be >= hist_len", (long long)d->t0);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const size_t words = size_t(scatter_work_words(d->n, d->batch, d->n_bins));
  if (cudaMemsetAsync(d->work, 0, sizeof(int32_t) * words, s) != cudaSuccess ||
      cudaMemsetAsync(d->ring, 0, sizeof(float) * size_t(d->batch * d->n * n_rec(*d)), s) != cudaSuccess)
    return bt_set_error(BT_ERR_CUDA, "memset failed");
  if (d->bin_hi > 0) {
    const int64_t npad = ((d->n + 31) >> 5) * 32;
    k_prime_history<<<int(ceil_div(int64_t(d->bin_hi) * npad, 256)), 256, 0, s>>>(*d);
    BT_CHECK_LAUNCH("k_prime_history");
  }
  return BT_OK;
}

namespace {
int input_project(int64_t rows, int64_t c_in, int64_t n, const float* xin, const float* w_t, const float* bias,
                  float* out, int32_t* work, const int32_t* live_len, int64_t batch, void* stream) {
  BT_CHECK_ARG(rows >= 0 && c_in >= 0 && n >= 0, "negative size");
  if (rows == 0 || n == 0) return BT_OK;
  BT_CHECK_ARG(xin && w_t && out && work, "null pointer");
  BT_CHECK_ARG(rows * c_in < (int64_t(1) << 40), "too large");
  BT_CHECK_ARG((reinterpret_cast<uintptr_t>(work) & 7) == 0, "work must be 8-byte aligned");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  int2* pairs = reinterpret_cast<int2*>(work);
  int32_t* cnt = work + 2 * rows * c_in;
  k_row_pairs<<<int(ceil_div(rows * 32, 256)), 256, 0, s>>>(rows, c_in, xin, cnt, pairs, live_len, batch);
  BT_CHECK_LAUNCH("k_row_pairs");
  dim3 grid(unsigned(ceil_div(rows, kProjRows)), unsigned(ceil_div(n, 256 * kProjNPT)));
  BT_CHECK_ARG(grid.y < 65536 && grid.x < (1u << 31), "projection grid too large");
  k_input_project<<<grid, 256, 0, s>>>(rows, c_in, n, w_t, bias, cnt, pairs, out);
  BT_CHECK_LAUNCH("k_input_project");
  return BT_OK;
}
}  // namespace

extern "C" int bt_input_project(int64_t rows, int64_t c_in, int64_t n, const float* xin, const float* w_t,
                                const float* bias, float* out, int32_t* work, void* stream) {
  return input_project(rows, c_in, n, xin, w_t, bias, out, work, nullptr, 1, stream);
}

extern "C" int bt_input_project_live(int64_t steps, int64_t batch, int64_t c_in, int64_t n, const float* xin,
                                     const float* w_t, const float* bias, const int32_t* sample_len, float* out,
                                     int32_t* work, void* stream) {
  BT_CHECK_ARG(steps >= 0 && batch > 0, "bad steps / batch");
  return input_project(steps * batch, c_in, n, xin, w_t, bias, out, work, sample_len, batch, stream);
}

extern "C" int bt_input_grad_weight(int64_t rows, int64_t c_in, int64_t n, const float* x, const float* g,
                                    float* out, int32_t accumulate, int32_t* work, void* stream) {
  BT_CHECK_ARG(rows >= 0 && c_in >= 0 && n >= 0, "negative size");
  if (c_in == 0 || n == 0) return BT_OK;
  BT_CHECK_ARG(x && g && out && work, "null pointer");
  BT_CHECK_ARG(c_in * (rows + 1) < (int64_t(1) << 31), "c_in * rows too large");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  int32_t* lists = work;
  int32_t* counts = work + c_in * rows;
  k_channel_rows<<<int(ceil_div(c_in * 32, 256)), 256, 0, s>>>(rows, c_in, x, lists, counts);
  BT_CHECK_LAUNCH("k_channel_rows");
  const dim3 grid(unsigned(c_in), unsigned(ceil_div(n, 256 * kProjNPT)));
  BT_CHECK_ARG(grid.y < 65536, "n too large");
  k_input_grad_weight<<<grid, 256, 0, s>>>(rows, c_in, n, x, g, lists, counts, out, accumulate);
  BT_CHECK_LAUNCH("k_input_grad_weight");
  return BT_OK;
}

extern "C" int bt_bits_to_float(int64_t rows, int64_t n, const uint32_t* bits, float* out, void* stream) {
  BT_CHECK_ARG(rows >= 0 && n >= 0, "negative size");
  if (rows * n == 0) return BT_OK;
  BT_CHECK_ARG(bits && out, "null pointer");
  k_bits_to_float<<<int(ceil_div(rows * n, 256)), 256, 0, static_cast<cudaStream_t>(stream)>>>(rows, n, bits, out);
  BT_CHECK_LAUNCH("k_bits_to_float");
  return BT_OK;
}

extern "C" int bt_mask_stride(int64_t batch) { return batch > 0 ? mask_stride(batch) : 0; }

extern "C" int64_t bt_engine_work_words(int64_t n, int64_t batch, int32_t n_bins) {
  return (n > 0 && batch > 0 && n_bins >= 1 && n_bins <= BT_MAX_BINS) ? scatter_work_words(n, batch, n_bins) : 0;
}

extern "C" int bt_float_to_masks(int64_t batch, int64_t n, const float* in, uint32_t* masks, void* stream) {
  BT_CHECK_ARG(batch >= 0 && n >= 0, "negative size");
  if (batch * n == 0) return BT_OK;
  BT_CHECK_ARG(in && masks, "null pointer");
  const int64_t total = n * mask_stride(batch);
  k_float_to_masks<<<int(ceil_div(total, 256)), 256, 0, static_cast<cudaStream_t>(stream)>>>(batch, n, in, masks);
  BT_CHECK_LAUNCH("k_float_to_masks");
  return BT_OK;
}

extern "C" int bt_masks_to_float(int64_t batch, int64_t n, const uint32_t* masks, float* out, void* stream) {
  BT_CHECK_ARG(batch >= 0 && n >= 0, "negative size");
  if (batch * n == 0) return BT_OK;
  BT_CHECK_ARG(out && masks, "null pointer");
  k_masks_to_float<<<int(ceil_div(batch * n, 256)), 256, 0, static_cast<cudaStream_t>(stream)>>>(batch, n, masks, out);
  BT_CHECK_LAUNCH("k_masks_to_float");
  return BT_OK;
}

extern "C" int bt_float_to_bits(int64_t rows, int64_t n, const float* in, uint32_t* bits, void* stream) {
  BT_CHECK_ARG(rows >= 0 && n >= 0, "negative size");
  if (rows * n == 0) return BT_OK;
  BT_CHECK_ARG(bits && in, "null pointer");
  const int64_t words = (n + 31) >> 5;
  k_float_to_bits<<<int(ceil_div(rows * words * 32, 256)), 256, 0, static_cast<cudaStream_t>(stream)>>>(rows, n, in,
                                                                                                         bits);
  BT_CHECK_LAUNCH("k_float_to_bits");
  return BT_OK;
}
