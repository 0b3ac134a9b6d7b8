// Spike-timing-dependent plasticity on the delivery CSR.
//
// Networks with plastic edges (synapse group > 0) advance one time step per batch, and
// each step T runs, around the step's delivery and update kernels:
//   before:  stamp reset at the 16-bit wrap points (src/nestgpu.cu:490-498,
//            src/rev_spike.cu:93-118), by the delivery kernel (reset_stamps);
//   after:   forward pass over the spikes arriving in T: each plastic edge records T as
//            its last arrival and is depressed against its target's last spike
//            (src/get_spike.cu:85-95); then the reverse pass: the plastic in-edges of
//            every node that spiked in T are potentiated against their last arrival
//            (src/rev_spike.cu:46-92).
// The delivery of T has already used the weights of the end of step T-1, as the
// reference's CollectSpike does before its update.  The weight rule is SynapseUpdate
// (src/syn_model.cu:43-56): STDPUpdate (src/stdp.cu:36-64) in FP64, or the linear test
// model (src/test_syn_model.cu:35-40).
#include <cuda_runtime.h>

#include <algorithm>

#include "ngpu_aeif.cuh"
#include "ngpu_types.h"

namespace ngpu {

constexpr int MAX_SYN_DT = 16384;   // src/syn_model.h:33

__device__ __forceinline__ float synapse_update(int type, const float *par, float w, float Dt) {
  if (type == SYN_TEST) return __fadd_rn(w, __fmaf_rn(par[0], Dt, par[1]));
  const double tau_plus = par[0], tau_minus = par[1], lambda = par[2], alpha = par[3];
  const double mu_plus = par[4], mu_minus = par[5], Wmax = par[6];
  const double wd = w;
  double w1;
  if (Dt >= 0.0f) {
    const double fact = lambda * exp(-(double)Dt / tau_plus);
    w1 = wd + fact * Wmax * pow(1.0 - wd / Wmax, mu_plus);
  } else {
    const double fact = -alpha * lambda * exp((double)Dt / tau_minus);
    w1 = wd + fact * Wmax * pow(wd / Wmax, mu_minus);
  }
  w1 = w1 > 0.0 ? w1 : 0.0;
  w1 = w1 < Wmax ? w1 : Wmax;
  return (float)w1;
}

__device__ __forceinline__ long long step_tidx(const Clock *clk, int k0) {
  return clk->tidx_base + clk->it0 + k0 + 1;
}

// One plastic edge, as one 16-byte load.
__device__ __forceinline__ PlasticEdge ldg_plastic(const PlasticEdge *p) {
  static_assert(sizeof(PlasticEdge) == 16, "PlasticEdge is one 16-byte word");
  const uint4 v = __ldg(reinterpret_cast<const uint4 *>(p));
  PlasticEdge e;
  e.pos = (unsigned long long)v.x | ((unsigned long long)v.y << 32);
  e.target = (int)v.z;
  e.group = (int)v.w;
  return e;
}

// Both passes are latency chains (ring or spike flag -> segment -> edge -> weight, then FP64
// exp and pow) over a few thousand edges, so what counts is how many edges run side by side:
// a warp per (spike, delay group) here, the warps of a block over the in-edges of its spiking
// targets below.  4000 neurons, 100 in-edges each, 24 spikes a step: with one thread per spike
// and one per target, each walking its edges, 24 and 137 us; now the two, the delivery and the
// update together take 16.9 us a step (173 before).
__global__ void __launch_bounds__(256) stdp_forward_kernel(const StdpArgs A, const Clock *clk, int k0) {
  pdl_enter();
  const int dd = blockIdx.x;
  const long long T = step_tidx(clk, k0);
  const long long te = T - 1 - (A.dmin + dd);   // the delay group's emission step
  if (te < 1) return;
  const int rs = (int)(te % A.R);
  int cnt = A.ring_cnt[rs];
  cnt = cnt < A.cap ? cnt : A.cap;
  const unsigned short t16 = (unsigned short)(T & 0xffff);
  const int lane = threadIdx.x & 31, nw = (int)(gridDim.y * (blockDim.x >> 5));
  for (int j = (int)(blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5)); j < cnt; j += nw) {
    const int src = A.ring[(size_t)rs * A.cap + j].x;
    const size_t key = (size_t)src * A.dspan + dd;
    const int p1 = __ldg(A.pl_off + key + 1);
    for (int p = __ldg(A.pl_off + key) + lane; p < p1; p += 32) {
      const PlasticEdge e = ldg_plastic(A.pl + p);
      A.stamp[p] = t16;
      const int last = A.last_tidx[e.target];
      if (last < 0) continue;   // the target has not spiked yet
      const long long Dt_int = T - last;
      if (Dt_int > 0 && Dt_int < MAX_SYN_DT) {
        const int g = e.group - 1;
        float &w = A.edge[e.pos].w;
        w = synapse_update(A.syn_type[g], A.syn_par + g * SYN_NPAR, w, -A.dt * (float)Dt_int);
      }
    }
  }
}

// A block serves 32 targets with plastic in-edges; its eight warps share the 32-edge chunks of
// those that spiked in step T.
constexpr int REV_TARGETS = 32;

__global__ void __launch_bounds__(256) stdp_reverse_kernel(const StdpArgs A, const Clock *clk, int k0) {
  pdl_enter();
  const long long T = step_tidx(clk, k0);
  const unsigned short t16 = (unsigned short)(T & 0xffff);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (long long r0 = (long long)blockIdx.x * REV_TARGETS; r0 < A.n_rev_nodes; r0 += (long long)gridDim.x * REV_TARGETS) {
    const int r = (int)r0 + lane;
    int q0 = 0, q1 = 0;
    bool spiked = false;
    if (r < A.n_rev_nodes) {
      q0 = __ldg(A.rev_off + r);
      q1 = __ldg(A.rev_off + r + 1);
      spiked = (long long)A.last_tidx[__ldg(A.rev_node + r)] == T;
    }
    int chunk = 0;             // chunks of the block's spiking targets so far
    for (unsigned mask = __ballot_sync(0xffffffffu, spiked); mask; mask &= mask - 1) {
      const int f = __ffs(mask) - 1;
      const int a = __shfl_sync(0xffffffffu, q0, f), b = __shfl_sync(0xffffffffu, q1, f);
      const int nc = (b - a + 31) >> 5;
      for (int c = ((warp - chunk) % nw + nw) % nw; c < nc; c += nw) {
        const int q = a + 32 * c + lane;
        if (q >= b) continue;
        const int p = __ldg(A.rev_id + q);
        const unsigned short Dt_int = (unsigned short)(t16 - A.stamp[p]);
        if (Dt_int < MAX_SYN_DT) {
          const PlasticEdge e = ldg_plastic(A.pl + p);
          const int g = e.group - 1;
          float &w = A.edge[e.pos].w;
          w = synapse_update(A.syn_type[g], A.syn_par + g * SYN_NPAR, w, A.dt * (float)Dt_int);
        }
      }
      chunk += nc;
    }
  }
}

// Spikes whose dendritic delay ends in step T reach their neuron's synapses: the reverse
// ring slot of T gives last_rev = T (set at the start of step T in the reference,
// src/spike_buffer.cu:314-316; only the plasticity passes after the update read it), and the
// slot is emptied for T + rev_R.
__global__ void rev_arrival_kernel(int *rev_ring, int *rev_cnt, int rev_R, int rev_cap, int *last_rev,
                                   const Clock *clk, int k0) {
  pdl_enter();
  const long long T = step_tidx(clk, k0);
  const int rs = (int)(T % rev_R);
  int cnt = rev_cnt[rs];
  cnt = cnt < rev_cap ? cnt : rev_cap;
  for (int j = threadIdx.x; j < cnt; j += blockDim.x) last_rev[rev_ring[(size_t)rs * rev_cap + j]] = (int)T;
  __syncthreads();
  if (threadIdx.x == 0) rev_cnt[rs] = 0;
}

int launch_rev_arrivals(int *rev_ring, int *rev_cnt, int rev_R, int rev_cap, int *last_rev, const Clock *clk,
                        int k0, cudaStream_t st) {
  launch_k(rev_arrival_kernel, dim3(1), dim3(256), 0, st, rev_ring, rev_cnt, rev_R, rev_cap, last_rev, clk, k0);
  return 1;
}

int launch_stdp_forward(const StdpArgs &A, const Clock *clk, int k0, cudaStream_t st) {
  // up to eight blocks (64 warps) per delay group while the grid stays below four blocks per SM
  const int y = std::max(1, std::min(8, 592 / A.dspan));
  launch_k(stdp_forward_kernel, dim3(A.dspan, y), dim3(256), 0, st, A, clk, k0);
  return 1;
}

int launch_stdp_reverse(const StdpArgs &A, const Clock *clk, int k0, cudaStream_t st) {
  const int nb = (A.n_rev_nodes + REV_TARGETS - 1) / REV_TARGETS;
  launch_k(stdp_reverse_kernel, dim3(std::max(1, std::min(nb, 148 * 32))), dim3(256), 0, st, A, clk, k0);
  return 1;
}

}  // namespace ngpu
