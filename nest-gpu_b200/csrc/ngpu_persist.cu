// Persistent step loop of iaf_psc_exp networks.
#include <algorithm>

#include "ngpu_aeif.cuh"
#include "ngpu_iaf.cuh"
#include "ngpu_types.h"

namespace ngpu {

// ---------------------------------------------------------------------------
// Persistent step loop for networks whose neurons are all iaf_psc_exp: one cooperative launch
// (one block per SM, all co-resident) advances K steps with one grid barrier per step.
//
// A block has two kinds of warps.  Step s of its neuron warps (one neuron per thread, state and
// parameters in registers): update; add the edges of the block's own spikes that arrive in step
// s + 1 (total delay one step); arrive at the grid barrier; while the others arrive, file the
// spikes in the ring, add their edges that arrive in step s + 2, draw the Poisson input; wait;
// fold the input of step s.  Its delivery warps meanwhile add the block's share of all other
// edges that arrive in step s + 1: spikes of steps <= s - 2, which were filed before barrier
// s - 1, a warp or, where segments are short, eight lanes per (spike, delay) segment, spread over all
// blocks.  They have from barrier s - 1
// until the block arrives at barrier s + 1, so their chain of four dependent loads stays off the
// critical path, which is: fold, update, the own spikes' first edges, the fence behind their
// reductions, and the barrier's round trip through L2.
// Arrivals of four steps are open at a time: accumulator slots s mod 4.  Before the first step
// what arrives in it (and from the step before, in the next one) is delivered from the ring, and
// nothing is delivered beyond the last step: between launches the state is that of the per-batch
// kernels, and the two can take turns.
//
// Layered microcircuit, us per step, against two launches per step (delivery, update) in a CUDA
// graph: at a tenth of its populations (7,700 neurons, 14k events a step) 15.7 -> 3.6, at full size
// (77,169 neurons, 96k events) 19.3 -> 4.7.  Of a step of 3.35 / 4.4 us the last block to arrive
// takes 2.6 / 3.8 us from barrier to barrier (two thirds of it its own spikes' edges and the
// release); an empty grid barrier of 148 blocks takes 1.34 us.
// ---------------------------------------------------------------------------
constexpr int PERS_NEURON = 576;      // neuron threads: 85,248 neurons on 148 SMs
constexpr int PERS_DELIVER = 192;     // delivery threads
constexpr int PERS_THREADS = PERS_NEURON + PERS_DELIVER;   // 80 registers a thread
constexpr int PERS_MAX_SPAN = PERS_DELIVER;   // delay groups at most (one count per delivery thread)
constexpr int PERS_SLOTS = 4;
// named barriers of a block: neuron warps; delivery warps; and, by step parity, "the deliveries
// for step s are done" (delivery warps arrive) and "barrier s has completed" (neuron warps arrive)
enum { NB_NEURON = 1, NB_DELIVER = 2, NB_DONE = 3, NB_NEXT = 5 };

__device__ __forceinline__ void nb_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void nb_arrive(int id, int n) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory");
}

// Waits until `count` has reached `target` (both wrap), at most about a second; then a block
// records a timeout in the status word and the kernel ends.  The polls are relaxed loads, with one
// acquire at the end: each acquire empties the SM's L1.
__device__ __forceinline__ bool grid_wait(unsigned *count, unsigned target, unsigned *status) {
  for (long long polls = 0; polls < (1LL << 21); polls++) {
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
    if ((int)(v - target) >= 0) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
      return true;
    }
  }
  atomicOr(status, ST_BARRIER_TIMEOUT);
  return false;
}
// By one thread, after a block-level barrier that all threads whose writes it covers passed.
__device__ __forceinline__ void grid_arrive(unsigned *count) {
  asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
}

// The blocks wait for one another before the first of them changes anything: while another kernel
// holds some of the GPU the launch has blocks that cannot start, and the barriers of the others
// would run out in the middle of the steps.  Whoever waits too long (2^17 polls, 18 ms) closes
// the gate; then no block goes on, the clock stays where it is and the engine runs the steps per
// batch.  One compare-and-swap decides, so all blocks see the same.
__device__ __forceinline__ void gate_enter(GridBarrier *bar, unsigned nblocks) {
  if (atomicAdd(&bar->gate, 1u) + 1u == nblocks) atomicCAS(&bar->state, (unsigned)GATE_WAIT, (unsigned)GATE_OPEN);
}
__device__ __forceinline__ bool gate_wait(GridBarrier *bar) {
  for (int polls = 0; polls < (1 << 17); polls++) {
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(&bar->state) : "memory");
    if (v != GATE_WAIT) return v == GATE_OPEN;
  }
  return atomicCAS(&bar->state, (unsigned)GATE_WAIT, (unsigned)GATE_CLOSED) == GATE_OPEN;
}

// A segment's edges by LANES lanes: e, e + stride, ..., four of them LANES apart at a time, in flight
// together before their reductions.  (Eight cost registers, and the kernel spills as it is.)
template <int LANES>
__device__ __forceinline__ void deliver_segment(const EdgeW *edge, double *acc, long long e0, int len, float height, int e,
                                                int stride) {
  const uint2 *p = reinterpret_cast<const uint2 *>(edge) + e0;
  for (; e < len; e += stride) {
    uint2 ew[4];
#pragma unroll
    for (int u = 0; u < 4; u++)
      if (e + LANES * u < len) ew[u] = __ldg(p + e + LANES * u);
#pragma unroll
    for (int u = 0; u < 4; u++)
      if (e + LANES * u < len) atomicAdd(&acc[ew[u].x], (double)__fmul_rn(height, __uint_as_float(ew[u].y)));
  }
}

// A neuron's Poisson input: none; one generator that is on during the whole launch, into receptor
// 0 or 1, drawn from shared memory; anything else, edge by edge.
enum PersPin { PIN_NONE = -2, PIN_LIST = -1, PIN_PORT0 = 0 };

struct PersShared {
  float par[IP_NPAR][PERS_NEURON];
  U4 word[PERS_NEURON];                 // Philox block of the Poisson edge for the current four steps
  unsigned key_lo[PERS_NEURON], key_hi[PERS_NEURON];
  float lam[PERS_NEURON], emlam[PERS_NEURON], weight[PERS_NEURON];
  long long e0[PERS_NEURON];            // the neuron's edges: start, and the numbers of those with a
  int2 len[PERS_NEURON];                // total delay of one and two steps
  int group[PERS_NEURON], idx[PERS_NEURON];   // the neuron's group (-1: none) and index in it
  int pin[PERS_NEURON];                 // its Poisson input (PersPin)
  int own[PERS_NEURON];                 // threads whose neuron spiked in the step
  unsigned long long nev;               // synaptic events delivered by the block
  int pref[PERS_MAX_SPAN + 1];
  int ns[2], ok[2];                     // by step parity
};

__device__ __forceinline__ int slot_back(int rs, int d, int R) { return rs >= d ? rs - d : rs - d + R; }

// LANES per segment of the delivery warps, by the mean segment's length (PERS_SHORT)
template <int LANES>
__global__ void __launch_bounds__(PERS_THREADS, 1) persistent_iaf_kernel(
    const DeliverArgs D, const IafArgs *tab, const int *first, int ngroups, const SpikeOut so, const Clock *clk, int K,
    GridBarrier *bar, uint64_t seed, int extra, int gate_extra) {
  extern __shared__ __align__(16) unsigned char pers_smem[];
  PersShared &S = *reinterpret_cast<PersShared *>(pers_smem);
  int *s_pref = S.pref, *s_ns = S.ns, *s_ok = S.ok;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int G = gridDim.x;
  const unsigned per_bar = (unsigned)(G + extra);   // extra, gate_extra > 0 only in the tests of the failure paths
  if (tid == 0) gate_enter(bar, (unsigned)(G + gate_extra));
  const long long t1 = clk->tidx_base + clk->it0 + 1;   // time index of the first step
  int rs = (int)(t1 % D.R);             // ring slot of the step
  int as = (int)(t1 % PERS_SLOTS);      // accumulator slot of the step
  // delay groups: total delay d + 1 steps, d = dmin + group; d = 0 and 1 are the spiking block's
  const int g0 = D.dmin == 0 ? 0 : -1;                                     // group with d = 0
  const int g1 = D.dmin <= 1 && 1 - D.dmin < D.dspan ? 1 - D.dmin : -1;    // group with d = 1
  const int gd = min(D.dspan, max(0, 2 - D.dmin));                         // first of the others

  // counts of the groups dd0 .. dspan-1 as seen from the step with time index te0 and ring slot
  // rs0 (emission steps te0 - dmin - dd), thread j of the caller's range; then one warp's scan
  auto load_counts = [&](int j, long long te0, int rs0, int dd0) {
    if (j < D.dspan - dd0) {
      const int d = D.dmin + dd0 + j;
      s_pref[j + 1] = te0 - d >= 1 ? min(__ldcg(D.ring_cnt + slot_back(rs0, d, D.R)), D.cap) : 0;
    }
  };
  auto scan_counts = [&](int np) {
    int carry = 0;
    if (lane == 0) s_pref[0] = 0;
    for (int b = 0; b < np; b += 32) {
      int v = b + lane < np ? s_pref[b + lane + 1] : 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += x;
      }
      if (b + lane < np) s_pref[b + lane + 1] = carry + v;
      carry += __shfl_sync(0xffffffffu, v, 31);
    }
  };
  const int sub = lane & (LANES - 1);
  auto deliver_entry = [&](int sl, int j, int dd, double *acc) {
    const int2 sp = __ldcg(D.ring + (size_t)sl * D.cap + j);
    const size_t key = (size_t)sp.x * D.dspan + dd;
    const long long e0 = __ldg(D.ev_off + key), e1 = __ldg(D.ev_off + key + 1);
    deliver_segment<LANES>(D.edge, acc, e0, (int)(e1 - e0), __int_as_float(sp.y), sub, 4 * LANES);
    if (sub == 0) atomicAdd(&S.nev, (unsigned long long)(e1 - e0));
  };
  // this block's share of those groups' segments, thread t of nt; consecutive ones go to
  // different blocks
  auto deliver_items = [&](int t, int nt, int rs0, int dd0, double *acc) {
    const int np = D.dspan - dd0, total = s_pref[np];
    for (int item = t / LANES * G + blockIdx.x; item < total; item += nt / LANES * G) {
      int a = 0, b = np;                // pair with s_pref[p] <= item < s_pref[p+1]
      while (b - a > 1) {
        const int mid = (a + b) >> 1;
        if (s_pref[mid] <= item) a = mid; else b = mid;
      }
      deliver_entry(slot_back(rs0, D.dmin + dd0 + a, D.R), item - s_pref[a], dd0 + a, acc);
    }
  };

  // what arrives in the first step; what the step before would have added for the next one
  {
    const int rs0 = slot_back(rs, 1, D.R);
    load_counts(tid, t1 - 1, rs0, 0);
    if (tid == 0) {
      S.nev = 0;
      s_ns[0] = s_ns[1] = 0;
      s_ok[0] = gate_wait(bar) ? 1 : 0;
      if (s_ok[0] && blockIdx.x == 0) D.ring_cnt[rs] = 0;   // holds no spike of the last dmax + 1 steps
    }
    __syncthreads();
    if (!s_ok[0]) return;
    if (warp == 0) scan_counts(D.dspan);
    __syncthreads();
    deliver_items(tid, PERS_THREADS, rs0, 0, D.acc + (size_t)as * D.slot_stride);
    if (g1 >= 0 && K > 1 && t1 - 1 >= 1) {
      const int c = min(__ldcg(D.ring_cnt + rs0), D.cap);
      for (int j = tid / LANES * G + blockIdx.x; j < c; j += PERS_THREADS / LANES * G)
        deliver_entry(rs0, j, g1, D.acc + (size_t)((as + 1) % PERS_SLOTS) * D.slot_stride);
    }
    __syncthreads();
    if (tid == 0) {
      grid_arrive(&bar->count);
      s_ok[0] = grid_wait(&bar->count, per_bar, so.status) ? 1 : 0;
    }
    __syncthreads();
    if (!s_ok[0]) return;
  }
  unsigned target = per_bar;

  if (tid >= PERS_NEURON) {
    // ---- delivery warps
    const int dt = tid - PERS_NEURON, dw = dt >> 5;
    nb_arrive(NB_DONE, PERS_THREADS);            // nothing is outstanding for the first step
    for (int k = 0; k < K - 1; k++) {
      as = (as + 1) % PERS_SLOTS;
      load_counts(dt, t1 + k, rs, gd);
      nb_sync(NB_DELIVER, PERS_DELIVER);
      if (dw == 0) scan_counts(D.dspan - gd);
      nb_sync(NB_DELIVER, PERS_DELIVER);
      deliver_items(dt, PERS_DELIVER, rs, gd, D.acc + (size_t)as * D.slot_stride);
      nb_arrive(NB_DONE + ((k + 1) & 1), PERS_THREADS);
      nb_sync(NB_NEXT + (k & 1), PERS_THREADS);
      if (!s_ok[k & 1]) break;
      rs = rs + 1 < D.R ? rs + 1 : 0;
    }
  } else {
    // ---- neuron warps
    // two warps share an own spike's segments; warp 0, which polls, delivers last
    const int rwarp = PERS_NEURON / 32 - 1 - warp, half = lane + 128 * (rwarp & 1);
    float Iex = 0.0f, Iin = 0.0f, V = 0.0f, refr = 0.0f;
    double *acc_i = nullptr;              // this neuron's entry of slot 0, receptor 0 (null: no neuron)
    int n = 0;                            // receptor 1 is n entries on
    {
      const int total_n = first[ngroups];
      const int npb = (total_n + G - 1) / G;
      const int gi = blockIdx.x * npb + tid;
      S.group[tid] = -1;
      if (tid < npb && gi < total_n) {
        int lo = 0, hi = ngroups;   // group with first[g] <= gi < first[g+1]
        while (hi - lo > 1) {
          const int mid = (lo + hi) >> 1;
          if (first[mid] <= gi) lo = mid; else hi = mid;
        }
        const IafArgs &A = tab[lo];
        const int i = gi - first[lo], node = A.i0 + i;
        S.group[tid] = lo;
        S.idx[tid] = i;
        n = A.n;
        acc_i = A.in.acc + i;
        IafRegs q;
        iaf_load(A, i, q);
        Iex = q.Iex;
        Iin = q.Iin;
        V = q.V;
        refr = q.refr;
        S.par[IP_I_e][tid] = q.I_e;
        S.par[IP_P20][tid] = q.P20;
        S.par[IP_P21ex][tid] = q.P21ex;
        S.par[IP_P21in][tid] = q.P21in;
        S.par[IP_P22][tid] = q.P22;
        S.par[IP_P11ex][tid] = q.P11ex;
        S.par[IP_P11in][tid] = q.P11in;
        S.par[IP_Theta_rel][tid] = q.theta;
        S.par[IP_V_reset_rel][tid] = q.V_reset;
        S.par[IP_refr_steps][tid] = q.refr_steps;
        const long long *off = D.ev_off + (size_t)node * D.dspan;
        int2 len = make_int2(0, 0);
        S.e0[tid] = __ldg(off);
        if (g0 >= 0) len.x = (int)(__ldg(off + 1) - __ldg(off));
        if (g1 >= 0) len.y = (int)(__ldg(off + g1 + 1) - __ldg(off + g1));
        S.len[tid] = len;
        S.pin[tid] = PIN_NONE;
        if (A.in.pin_off) {
          const int pe0 = __ldg(A.in.pin_off + i), npe = __ldg(A.in.pin_off + i + 1) - pe0;
          if (npe > 0) S.pin[tid] = PIN_LIST;
          if (npe == 1) {
            const PoissonIn pe = ldg_pin(A.in.pin + pe0);
            const GenPar gp = ldg_gen(A.in.gen + pe.gen);
            const float lam = __fmul_rn(A.in.lam_scale, gp.rate);
            const Clock cl = *clk;
            const double ta = step_at(cl, 0, 0, D.dt).tnow - (double)gp.origin - (double)pe.delay,
                         tb = step_at(cl, K - 1, 0, D.dt).tnow - (double)gp.origin - (double)pe.delay;
            if (ta >= (double)gp.start && tb <= (double)gp.stop && lam > 0.0f && lam <= 10.0f)
              S.pin[tid] = PIN_PORT0 + pe.port;
            S.lam[tid] = lam;
            S.emlam[tid] = exp_m(-lam);
            S.weight[tid] = pe.weight;
            const uint64_t key = pin_key(pe);
            S.key_lo[tid] = (unsigned)key;
            S.key_hi[tid] = (unsigned)(key >> 32);
          }
        }
      }
    }
    const bool rec = acc_i && tab[S.group[tid]].rec.first != nullptr;
    for (int k = 0; k < K; k++) {
      const bool last = k == K - 1;
      const int par = k & 1;
      const int as1 = (as + 1) % PERS_SLOTS, rs1 = rs + 1 < D.R ? rs + 1 : 0;
      bool spike = false;
      if (acc_i) {
        IafRegs q;
        q.Iex = Iex;
        q.Iin = Iin;
        q.V = V;
        q.refr = refr;
        q.I_e = S.par[IP_I_e][tid];
        q.P20 = S.par[IP_P20][tid];
        q.P21ex = S.par[IP_P21ex][tid];
        q.P21in = S.par[IP_P21in][tid];
        q.P22 = S.par[IP_P22][tid];
        q.P11ex = S.par[IP_P11ex][tid];
        q.P11in = S.par[IP_P11in][tid];
        q.theta = S.par[IP_Theta_rel][tid];
        q.V_reset = S.par[IP_V_reset_rel][tid];
        q.refr_steps = S.par[IP_refr_steps][tid];
        spike = iaf_step(q);
        Iex = q.Iex;
        Iin = q.Iin;
        V = q.V;
        refr = q.refr;
        if (spike) {
          const int node = tab[S.group[tid]].i0 + S.idx[tid];
          so.last_tidx[node] = (int)(t1 + k);
          so.last_height[node] = 1.0f;
          S.own[atomicAdd(&s_ns[par], 1)] = tid;
        }
        if (rec) {
          const float yr[4] = {Iex, Iin, V, refr};
          const IafArgs &A = tab[S.group[tid]];
          const int i = S.idx[tid];
          write_records<4>(A.rec, so, A.i0 + i, i, yr, 4, refr, clk->it0 + k - clk->rec_it0, t1 + k);
        }
      }
      nb_sync(NB_NEURON, PERS_NEURON);
      const int ns = s_ns[par];
      if (tid == 0) {
        s_ns[par ^ 1] = 0;
        if (blockIdx.x == 0) D.ring_cnt[rs1] = 0;
      }
      if (!last)
        for (int j = rwarp >> 1; j < ns; j += PERS_NEURON / 64) {
          const int o = S.own[j], len = S.len[o].x;
          deliver_segment<32>(D.edge, D.acc + (size_t)as1 * D.slot_stride, S.e0[o], len, 1.0f, half, 256);
          if (half == 0) atomicAdd(&S.nev, (unsigned long long)len);
        }
      nb_sync(NB_DONE + par, PERS_THREADS);
      target += per_bar;
      if (tid == 0) grid_arrive(&bar->count);
      if (spike) {
        atomicAdd(so.n_spikes, 1ULL);
        const IafArgs &A = tab[S.group[tid]];
        const int i = S.idx[tid], node = A.i0 + i;
        file_spike(so, A.srec, i, step_at(*clk, k, 0, D.dt).tnow);
        if (so.has_out[node]) {
          const int pos = atomicAdd(&so.ring_cnt[rs], 1);
          if (pos < so.cap) so.ring[(size_t)rs * so.cap + pos] = make_int2(node, __float_as_int(1.0f));
          else atomicOr(so.status, ST_RING_OVERFLOW);
        }
      }
      if (k + 2 < K)
        for (int j = rwarp >> 1; j < ns; j += PERS_NEURON / 64) {
          const int o = S.own[j];
          const int2 len = S.len[o];
          deliver_segment<32>(D.edge, D.acc + (size_t)((as + 2) % PERS_SLOTS) * D.slot_stride, S.e0[o] + len.x, len.y, 1.0f,
                          half, 256);
          if (half == 0) atomicAdd(&S.nev, (unsigned long long)len.y);
        }
      double in[2] = {0.0, 0.0};
      const int pin = acc_i ? S.pin[tid] : PIN_NONE;
      if (pin >= PIN_PORT0) {
        const int w = (int)(t1 + k) & 3;
        if (k == 0 || w == 0)
          S.word[tid] = poisson_block(seed, ((uint64_t)S.key_hi[tid] << 32) | S.key_lo[tid], t1 + k, 0);
        const int c = poisson_small(S.lam[tid], S.emlam[tid], u01((&S.word[tid].x)[w]));
        if (c > 0) add_to_port<2>(in, pin - PIN_PORT0, (double)__fmul_rn(S.weight[tid], (float)c));
      } else if (pin == PIN_LIST) {
        const IafArgs &A = tab[S.group[tid]];
        const StepT t = step_at(*clk, k, 0, D.dt);
        for (int e = A.in.pin_off[S.idx[tid]]; e < A.in.pin_off[S.idx[tid] + 1]; e++) {
          const PoissonIn p = A.in.pin[e];
          poisson_add<2>(in, A.in, p, A.in.gen[p.gen], t.tidx, t.tnow);
        }
      }
      if (tid == 0) s_ok[par] = grid_wait(&bar->count, target, so.status) ? 1 : 0;
      nb_sync(NB_NEURON, PERS_NEURON);
      if (!last) nb_arrive(NB_NEXT + par, PERS_THREADS);
      if (!s_ok[par]) break;
      if (acc_i) {
        double *p = acc_i + (size_t)as * D.slot_stride;
        const double a0 = __ldcg(p), a1 = __ldcg(p + n);
        if (a0 != 0.0) p[0] = 0.0;
        if (a1 != 0.0) p[n] = 0.0;
        in[0] = a0 + in[0];
        in[1] = a1 + in[1];
        if (in[0] != 0.0) Iex = (float)__fma_rn(in[0], 1.0, (double)Iex);
        if (in[1] != 0.0) Iin = (float)__fma_rn(in[1], 1.0, (double)Iin);
      }
      as = as1;
      rs = rs1;
    }
    if (acc_i) {
      float *var = tab[S.group[tid]].var + S.idx[tid];
      var[0] = Iex;
      var[(size_t)n] = Iin;
      var[2 * (size_t)n] = V;
      var[3 * (size_t)n] = refr;
    }
  }
  __syncthreads();
  if (tid == 0 && S.nev) atomicAdd(D.n_events, S.nev);
}

// The clock after a launch: advanced, or the steps noted for the host where the gate was closed.
__global__ void persistent_advance_kernel(Clock *clk, int K, const GridBarrier *bar, long long *skipped) {
  if (bar->state == GATE_OPEN) clk->it0 += K;
  else *skipped += K;
}

// Edges of total delay one and two steps (the first `groups` delay groups of every node).
__global__ void first_edges_kernel(const long long *ev_off, int n_nodes, int dspan, int groups, unsigned long long *sum) {
  unsigned long long s = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_nodes; i += gridDim.x * blockDim.x) {
    const long long *off = ev_off + (size_t)i * dspan;
    s += (unsigned long long)(off[groups] - off[0]);
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0 && s) atomicAdd(sum, s);
}

// `d_sum`: a zeroed counter on the device.  -1: it could not run.
long long persistent_own_edges(const long long *ev_off, int n_nodes, int dspan, unsigned long long *d_sum) {
  first_edges_kernel<<<std::min((n_nodes + 255) / 256, 592), 256>>>(ev_off, n_nodes, dspan, std::min(dspan, 2), d_sum);
  unsigned long long h = 0;
  if (cudaGetLastError() != cudaSuccess) return -1;
  if (cudaMemcpy(&h, d_sum, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
  return (long long)h;
}

// Blocks of the persistent loop for a network of `n_iaf` iaf_psc_exp neurons and `dspan` delay
// groups on this GPU (one neuron per neuron thread, one co-resident block per SM), 0 if it does
// not fit.
int persistent_blocks(long long n_iaf, int dspan) {
  int dev = 0, n_sm = 0, per_sm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev);
  if (dspan > PERS_MAX_SPAN || n_iaf > (long long)n_sm * PERS_NEURON) return 0;
  for (auto *kernel : {persistent_iaf_kernel<8>, persistent_iaf_kernel<32>}) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(PersShared)) != cudaSuccess)
      return 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, PERS_THREADS, sizeof(PersShared));
    if (per_sm < 1) return 0;
  }
  return n_sm;
}

// A warp of the delivery warps serves one segment, or four short ones side by side: what a segment
// costs there is its chain of four dependent loads, whatever its length.  us per step, a warp / eight lanes a segment, 70,000
// neurons of 29 delay groups and 550 spikes a step: 7 edges a segment 23.0 / 10.2, 34 edges 26.3 /
// 13.4; 40,000 neurons, 315 spikes, 50 edges 16.0 / 9.6; 20,000 of 10 groups, 160 spikes, 60 edges
// 3.9 / 3.8, but 100 edges 4.2 / 5.0, and the layered microcircuit (130 edges) 3.6 / 7.8 at a tenth of
// its size, 4.6 / 10.5 at full size.
constexpr double PERS_SHORT = 64.0;

// Cooperative launch of the persistent loop over `steps` steps, then the clock; the number of
// launches, or -1 where the cooperative launch is refused.
int launch_persistent_iaf(const DeliverArgs &D, const IafArgs *tab, const int *first, int ngroups, const SpikeOut &so,
                          Clock *clk, int steps, GridBarrier *bar, long long *skipped, uint64_t seed, int nblocks,
                          int barrier_extra, int gate_extra, double mean_segment, cudaStream_t st) {
  void *kernel = mean_segment <= PERS_SHORT ? (void *)persistent_iaf_kernel<8> : (void *)persistent_iaf_kernel<32>;
  DeliverArgs d = D;
  const IafArgs *t = tab;
  const int *f = first;
  int ng = ngroups;
  SpikeOut s = so;
  const Clock *c = clk;
  int k = steps;
  GridBarrier *b = bar;
  uint64_t sd = seed;
  int x = barrier_extra, gx = gate_extra;
  void *args[] = {&d, &t, &f, &ng, &s, &c, &k, &b, &sd, &x, &gx};
  if (cudaLaunchCooperativeKernel(kernel, dim3(nblocks), dim3(PERS_THREADS), args, sizeof(PersShared), st) != cudaSuccess)
    return -1;
  persistent_advance_kernel<<<1, 1, 0, st>>>(clk, steps, bar, skipped);
  return 2;
}

}  // namespace ngpu
