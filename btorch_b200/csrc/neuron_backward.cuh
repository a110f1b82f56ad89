// Reverse-mode derivative of one neuron step, following the autograd graph the
// reference builds from its eager ops (lif.py:144-187, alif.py:193-249).  The
// fire step's surrogate is the sigmoid one: damping * 4 * s(k a u) * (1 - s(k a u)).
#pragma once

#include "neuron.cuh"

namespace bt {

struct NeuronGrad {
  float x, v, gk;  // gradients of the input current, v and g_k before the step
};

// gs, gv2, ggk2: gradients of the step's spike, v and g_k; x, v, gk: its inputs;
// s, u, mask, v1: its spike, surrogate argument, refractory mask and v after charge.
__device__ __forceinline__ NeuronGrad neuron_backward(const NeuronParams& p, float sg_damping, bool alif, bool hard_reset,
                                                      bool detach_reset, float gs, float gv2, float ggk2, float x,
                                                      float v, float gk, float s, float u, float mask, float v1) {
  const float vth = p.vth, vr = p.vr, cm = p.cm, dt = p.dt;
  const float den = vth - vr;
  // reset:  hard v2 = v1 - (v1 - vr) * s ;  soft v2 = v1 - (vth - vr) * s
  float gv1, gs_reset;
  if (hard_reset) {
    gv1 = gv2 - gv2 * s;
    gs_reset = -gv2 * (v1 - vr);
  } else {
    gv1 = gv2;
    gs_reset = -gv2 * den;
  }
  if (alif) gs_reset += ggk2 * p.dgk;  // gk2 = gk1 + dg_k * s
  if (!detach_reset) gs += gs_reset;
  // fire:  s = H(u) * mask with the surrogate derivative at u;  u = (v1 - vth) / den
  const float sig = sigmoidf_dev(p.sg_alpha * u);
  const float gu = (gs * mask) * (sg_damping * 4.0f * sig * (1.0f - sig));
  gv1 += gu / den;
  NeuronGrad o;
  if (!alif) {
    // charge: v1 = v + dt * ((-(v - vr)) / tau + I / cm)
    const float gD = dt * gv1;
    o.x = gD / cm;
    o.v = gv1 - gD / p.tau;
    o.gk = 0.0f;
    return o;
  }
  // charge: v1 = v + C(lin) * D,  D = (ngl (v - El) + (-gk)(v - Ek) + I) / cm,  lin = (ngl - gk) / cm
  const float ngl = p.ngl, Ek = p.Ek;
  const float lin = (ngl - gk) / cm;
  const float em1 = expm1f(dt * lin);
  const float C = em1 / lin;
  const float D = (ngl * (v - p.El) + (-gk) * (v - Ek) + x) / cm;
  const float gC = gv1 * D, gD = gv1 * C;
  o.x = gD / cm;
  o.v = gv1 + gD * lin;
  // dC/dlin = (dt e^{dt lin} lin - expm1(dt lin)) / lin^2 ; dlin/dgk = -1/cm ; dD/dgk = -(v - Ek)/cm
  const float dCdl = (dt * (em1 + 1.0f) * lin - em1) / (lin * lin);
  const float g_gk_charge = -(gC * dCdl) / cm - gD * (v - Ek) / cm;
  // adaptation: gk1 = gk + coef_gk * ((-gk) / tau_adapt)
  const float dgk1 = 1.0f - p.cgk / p.tau_a;
  o.gk = ggk2 * dgk1 + g_gk_charge;
  return o;
}

}  // namespace bt
