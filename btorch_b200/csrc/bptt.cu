// Backward of one chunk of a recurrent run (the reverse of rnn.py:517-528 over
// time): per step t, descending,
//   dz_t       = gZ_t + W^T dpsc_t                        (k_rows_gather)
//   dI_t, dv_{t-1}, dg_k_{t-1} = neuron'(dz_t, dv_t, dg_k_t)
//   dpsc_{t-1} = dpsc_t + coef * ((-dpsc_t) / tau) + dI_t (+ the stack's gradient)
// Two launches per step: the transposed gather and k_bptt_step, which does the
// rest and hands the next step's dpsc over in both layouts.
#include <cstring>

#include "neuron_backward.cuh"

namespace bt {

// spmm.cu: out [batch][n_rows] from gT [n_cols][pitch], as a step kernel
int rows_product(bool first, int64_t batch, int64_t pitch, int64_t n_rows, const int32_t* ptr, const uint32_t* col,
                 const float* wts, const float* gT, float* out, cudaStream_t s);

struct BpttStep {
  const float *x, *psc, *v, *ref, *gk, *z;        // drive and state before the step, its spikes
  const float *gz, *g_z, *g_v, *g_gk, *g_psc;     // W^T dpsc_t; stack gradients of step t (g_psc: of step t - 1)
  float *cur_v, *cur_gk;                          // dL/d(state after the step) in, before the step out
  const float* dpsc;                              // dL/dpsc_t
  float *g_I, *next_psc, *next_T;                 // dI_t; dL/dpsc_{t-1} as [batch][n] and transposed (may be null)
};

// Block = 32 neurons x 32 samples, a thread 4 consecutive neurons of one sample
// (16-byte accesses when VEC: n a multiple of 4 and aligned arrays), all loads
// before the first store; the transposed gradient goes through a shared-memory
// tile.  One pass over 12 arrays where the step took five launches over 21
// (transpose, gather, add, neuron backward with its saved u / mask / v_charged,
// synapse, copy); u, mask and v_charged are evaluated again from the state
// before the step.
template <int KIND, bool HARD, bool USE_REF, bool FAST, bool VEC>
__global__ void __launch_bounds__(256) k_bptt_step(bt_neuron_desc nd, bt_param psc_coef, bt_param psc_tau, int64_t batch,
                                                   int64_t pitch, int64_t n, int detach_reset, BpttStep a) {
  step_begin();
  constexpr bool ALIF = KIND == BT_NEURON_ALIF;
  __shared__ float s_t[32][33];
  const int tq = int(threadIdx.x) & 7, tb = int(threadIdx.x) >> 3;
  const int64_t i0 = int64_t(blockIdx.x) * 32 + 4 * tq, b0 = int64_t(blockIdx.y) * 32, b = b0 + tb;
  const int64_t idx = b * n + i0;
  const int cnt = b < batch ? int(n - i0 < 0 ? 0 : n - i0 > 4 ? 4 : n - i0) : 0;  // neurons of this thread
  auto get = [&](const float* p, float(&q)[4]) {
    if constexpr (VEC) {
      const float4 f = (p && cnt) ? *reinterpret_cast<const float4*>(p + idx) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      q[0] = f.x, q[1] = f.y, q[2] = f.z, q[3] = f.w;
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k) q[k] = (p && k < cnt) ? p[idx + k] : 0.0f;
    }
  };
  auto put = [&](float* p, const float(&q)[4]) {
    if constexpr (VEC) {
      if (cnt) *reinterpret_cast<float4*>(p + idx) = make_float4(q[0], q[1], q[2], q[3]);
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (k < cnt) p[idx + k] = q[k];
    }
  };
  float x[4], psc[4], v[4], ref[4] = {}, gk[4] = {}, z[4], gs[4], gv[4], gg[4] = {}, dp[4], t[4], gp[4];
  get(a.x, x);
  get(a.psc, psc);
  get(a.v, v);
  if (USE_REF) get(a.ref, ref);
  get(a.z, z);
  get(a.gz, gs);
  get(a.cur_v, gv);
  get(a.dpsc, dp);
  if (ALIF) {
    get(a.gk, gk);
    get(a.cur_gk, gg);
  }
  if (a.g_z) {
    get(a.g_z, t);
#pragma unroll
    for (int k = 0; k < 4; ++k) gs[k] = add(gs[k], t[k]);
  }
  if (a.g_v) {
    get(a.g_v, t);
#pragma unroll
    for (int k = 0; k < 4; ++k) gv[k] = add(gv[k], t[k]);
  }
  if (ALIF && a.g_gk) {
    get(a.g_gk, t);
#pragma unroll
    for (int k = 0; k < 4; ++k) gg[k] = add(gg[k], t[k]);
  }
  get(a.g_psc, gp);
  NeuronParams p = load_params<KIND, USE_REF>(nd, cnt ? i0 : 0);
  float g_I[4], next[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int64_t i = k < cnt ? i0 + k : 0;
    if (!FAST && k > 0 && !nd.uniform) p = load_params<KIND, USE_REF>(nd, i);
    const float I = add(psc[k], x[k]);
    float v1 = v[k], r1 = ref[k], g1 = gk[k];
    const NeuronOut o = neuron_update<KIND, HARD, USE_REF, true, FAST>(p, I, v1, r1, g1);
    const NeuronGrad g = neuron_backward(p, nd.sg_damping, ALIF, HARD, detach_reset != 0, gs[k], gv[k], gg[k], I, v[k],
                                         gk[k], z[k], o.u, o.mask, o.v_charged);
    g_I[k] = g.x;
    gv[k] = g.v;
    gg[k] = g.gk;
    next[k] = add(psc_decay(psc_coef, psc_tau, i, dp[k]), g.x);
    if (a.g_psc) next[k] = add(next[k], gp[k]);
    s_t[4 * tq + k][tb] = k < cnt ? next[k] : 0.0f;
  }
  put(a.g_I, g_I);
  put(a.cur_v, gv);
  if (ALIF) put(a.cur_gk, gg);
  put(a.next_psc, next);
  if (!a.next_T) return;
  __syncthreads();
  const int tx = int(threadIdx.x) & 31, ty = int(threadIdx.x) >> 5;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int64_t row = int64_t(blockIdx.x) * 32 + ty + 8 * k, c = b0 + tx;
    if (row < n && c < pitch) a.next_T[row * pitch + c] = s_t[ty + 8 * k][tx];
  }
}

// dpsc of the chunk's last step: the later chunk's gradient plus the stack's, in both layouts.
__global__ void __launch_bounds__(256) k_bptt_begin(int64_t batch, int64_t pitch, int64_t n, const float* __restrict__ cur,
                                                    const float* __restrict__ g_psc, float* __restrict__ out,
                                                    float* __restrict__ outT) {
  __shared__ float s_t[32][33];
  const int tx = int(threadIdx.x) & 31, ty = int(threadIdx.x) >> 5;
  const int64_t i = int64_t(blockIdx.x) * 32 + tx, b0 = int64_t(blockIdx.y) * 32;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int64_t b = b0 + ty + 8 * k, idx = b * n + i;
    float g = 0.0f;
    if (i < n && b < batch) {
      g = cur[idx];
      if (g_psc) g = add(g, g_psc[idx]);
      out[idx] = g;
    }
    s_t[tx][ty + 8 * k] = g;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int64_t row = int64_t(blockIdx.x) * 32 + ty + 8 * k, c = b0 + tx;
    if (row < n && c < pitch) outT[row * pitch + c] = s_t[ty + 8 * k][tx];
  }
}

}  // namespace bt

using namespace bt;

namespace {

// The device's Div kind of divisor c is 1 or 2 (as engine.cu's fast_divisors,
// without the synapse's, which k_bptt_step divides by psc_decay).
bool fast_neuron(const bt_neuron_desc& nd) {
  if (!nd.uniform) return false;
  auto ok = [](float c, bool verified) {
    uint32_t u;
    std::memcpy(&u, &c, sizeof(u));
    const uint32_t e = u >> 23;
    return ((u & 0x7fffffu) == 0u && e >= 1u && e <= 253u) || verified;
  };
  return ok(nd.sv[2], nd.fast_div & 1) && ok(nd.sv[0] - nd.sv[1], nd.fast_div & 2) &&
         (nd.kind == BT_NEURON_LIF ? ok(nd.sv[3], nd.fast_div & 4) : ok(nd.sv[9], nd.fast_div & 8));
}

using StepKernel = void (*)(bt_neuron_desc, bt_param, bt_param, int64_t, int64_t, int64_t, int, BpttStep);

template <int KIND, bool FAST, bool VEC>
StepKernel pick(bool h, bool r) {
  return h ? (r ? k_bptt_step<KIND, true, true, FAST, VEC> : k_bptt_step<KIND, true, false, FAST, VEC>)
           : (r ? k_bptt_step<KIND, false, true, FAST, VEC> : k_bptt_step<KIND, false, false, FAST, VEC>);
}

template <int KIND>
StepKernel pick(bool fast, bool vec, bool h, bool r) {
  if (fast) return vec ? pick<KIND, true, true>(h, r) : pick<KIND, true, false>(h, r);
  return vec ? pick<KIND, false, true>(h, r) : pick<KIND, false, false>(h, r);
}

}  // namespace

extern "C" int bt_bptt_backward(const bt_bptt_desc* d, void* stream) {
  if (!d) return bt_set_error(BT_ERR_INVALID, "null descriptor");
  if (int st = bt_check_neuron_desc(&d->neuron)) return st;
  const bt_neuron_desc& nd = d->neuron;
  const int64_t B = d->batch, n = d->n, T = d->n_steps;
  BT_CHECK_ARG(B >= 0 && n >= 0 && T >= 0, "negative size");
  if (B * n == 0 || T == 0) return BT_OK;
  BT_CHECK_ARG(B * n < (int64_t(1) << 40) && B < (int64_t(1) << 16), "too large");
  BT_CHECK_ARG(nd.spiking, "the fused backward needs a spiking (Heaviside) forward");
  BT_CHECK_ARG(d->csr_ptr && d->x && d->v && d->psc && d->z && d->cur_psc && d->cur_v && d->G_psc && d->G_I && d->gz &&
                   d->gT, "null pointer");
  BT_CHECK_ARG(!nd.use_refractory || d->ref, "refractory state missing");
  BT_CHECK_ARG(nd.kind != BT_NEURON_ALIF || (d->gk && d->cur_gk), "g_k state missing");
  BT_CHECK_ARG(d->psc_coef.ptr && d->psc_tau.ptr, "PSC coefficients missing");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int64_t pitch = ceil_div(B, 4) * 4, per = B * n;
  const dim3 grid(unsigned(ceil_div(n, 32)), unsigned(ceil_div(pitch, 32)));
  const bool fast = fast_neuron(nd), h = nd.hard_reset != 0, r = nd.use_refractory != 0;
  uintptr_t all = 0;  // 16-byte accesses: every array and row aligned
  for (const void* p : {(const void*)d->x, (const void*)d->z, (const void*)d->v, (const void*)d->psc, (const void*)d->ref,
                        (const void*)d->gk, (const void*)d->g_z, (const void*)d->g_v, (const void*)d->g_psc,
                        (const void*)d->g_gk, (const void*)d->cur_psc, (const void*)d->cur_v, (const void*)d->cur_gk,
                        (const void*)d->G_psc, (const void*)d->G_I, (const void*)d->gz})
    all |= reinterpret_cast<uintptr_t>(p);
  const bool vec = n % 4 == 0 && (all & 15) == 0;
  const StepKernel kern = nd.kind == BT_NEURON_LIF ? pick<BT_NEURON_LIF>(fast, vec, h, r) : pick<BT_NEURON_ALIF>(fast, vec, h, r);
  auto row = [&](const float* p, int64_t t) { return p ? p + t * per : nullptr; };
  k_bptt_begin<<<grid, 256, 0, s>>>(B, pitch, n, d->cur_psc, row(d->g_psc, T - 1), d->G_psc + (T - 1) * per, d->gT);
  BT_CHECK_LAUNCH("k_bptt_begin");
  for (int64_t t = T - 1; t >= 0; --t) {
    if (int st = rows_product(false, B, pitch, n, d->csr_ptr, d->csr_dst, d->csr_w, d->gT, d->gz, s)) return st;
    BpttStep a;
    a.x = d->x + t * per;
    a.psc = d->psc + t * per;
    a.v = d->v + t * per;
    a.ref = r ? d->ref + t * per : nullptr;
    a.gk = row(d->gk, t);
    a.z = d->z + t * per;
    a.gz = d->gz;
    a.g_z = row(d->g_z, t);
    a.g_v = row(d->g_v, t);
    a.g_gk = row(d->g_gk, t);
    a.g_psc = t > 0 ? row(d->g_psc, t - 1) : nullptr;
    a.cur_v = d->cur_v;
    a.cur_gk = d->cur_gk;
    a.dpsc = d->G_psc + t * per;
    a.g_I = d->G_I + t * per;
    a.next_psc = t > 0 ? d->G_psc + (t - 1) * per : d->cur_psc;
    a.next_T = t > 0 ? d->gT : nullptr;
    if (launch_step(false, kern, grid, 256, 0, s, nd, d->psc_coef, d->psc_tau, B, pitch, n, int(d->detach_reset), a) != cudaSuccess)
      break;
  }
  BT_CHECK_LAUNCH("k_bptt_step");
  return BT_OK;
}
