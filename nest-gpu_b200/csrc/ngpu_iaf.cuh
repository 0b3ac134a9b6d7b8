// Device code of the iaf_psc_exp step shared by the per-batch kernels (ngpu_kernels.cu) and the
// persistent step loop (ngpu_persist.cu).
#pragma once
#include "ngpu_types.h"

namespace ngpu {

// ---------------------------------------------------------------------------
// iaf_psc_exp exact propagator (src/iaf_psc_exp.cu:85-110)
// ---------------------------------------------------------------------------
__device__ __forceinline__ float iget(const IafArgs &A, int j, int i) {
  const float *p = A.parr[j];
  return p ? __ldg(p + i) : A.pval[j];
}

// State and derived parameters of one iaf_psc_exp neuron.
struct IafRegs {
  float Iex, Iin, V, refr;
  float I_e, P20, P21ex, P21in, P22, P11ex, P11in, theta, V_reset, refr_steps;
};

__device__ __forceinline__ void iaf_load(const IafArgs &A, int i, IafRegs &q) {
  const size_t n = A.n;
  q.Iex = A.var[i];
  q.Iin = A.var[n + i];
  q.V = A.var[2 * n + i];
  q.refr = A.var[3 * n + i];
  q.I_e = iget(A, IP_I_e, i);
  q.P20 = iget(A, IP_P20, i);
  q.P21ex = iget(A, IP_P21ex, i);
  q.P21in = iget(A, IP_P21in, i);
  q.P22 = iget(A, IP_P22, i);
  q.P11ex = iget(A, IP_P11ex, i);
  q.P11in = iget(A, IP_P11in, i);
  q.theta = iget(A, IP_Theta_rel, i);
  q.V_reset = iget(A, IP_V_reset_rel, i);
  q.refr_steps = iget(A, IP_refr_steps, i);
}

__device__ __forceinline__ void iaf_store(const IafArgs &A, int i, const IafRegs &q) {
  const size_t n = A.n;
  A.var[i] = q.Iex;
  A.var[n + i] = q.Iin;
  A.var[2 * n + i] = q.V;
  A.var[3 * n + i] = q.refr;
}

// One time step up to the threshold; true if the neuron spikes (and is reset).
__device__ __forceinline__ bool iaf_step(IafRegs &q) {
  if (q.refr > 0.0f) {
    q.refr = __fsub_rn(q.refr, 1.0f);
  } else {
    q.V = __fmaf_rn(q.I_e, q.P20, __fmaf_rn(q.Iin, q.P21in, __fmaf_rn(q.Iex, q.P21ex, __fmul_rn(q.V, q.P22))));
  }
  q.Iex = __fmul_rn(q.Iex, q.P11ex);
  q.Iin = __fmul_rn(q.Iin, q.P11in);
  if (!(q.V >= q.theta)) return false;
  q.V = q.V_reset;
  q.refr = q.refr_steps;
  return true;
}

// The step's input, at its end.
__device__ __forceinline__ void iaf_fold(IafRegs &q, const double *in) {
  if (in[0] != 0.0) q.Iex = (float)__fma_rn(in[0], 1.0, (double)q.Iex);
  if (in[1] != 0.0) q.Iin = (float)__fma_rn(in[1], 1.0, (double)q.Iin);
}

}  // namespace ngpu
