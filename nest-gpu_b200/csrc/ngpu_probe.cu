// Measured denominator for the delivery kernel's roofline: the rate of FP64 reductions
// (red.global.add.f64) to uniformly random addresses of a buffer, the access pattern of the
// delivery's accumulator updates (random targets inside one accumulator slot).  No
// counterpart in the reference.
#include <cuda_runtime.h>

#include <stdexcept>
#include <string>

#include "ngpu_math.cuh"

namespace ngpu {

__global__ void random_reduction_kernel(double *buf, unsigned long long n_elem, long long ops_per_thread,
                                        unsigned seed) {
  const unsigned long long tid = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
  unsigned x = (unsigned)(tid * 2654435761ULL) ^ seed;
  for (long long k = 0; k < ops_per_thread; k++) {
    // xorshift32: a new pseudo-random index per operation
    x ^= x << 13;
    x ^= x >> 17;
    x ^= x << 5;
    atomicAdd(&buf[x % n_elem], 1.0);
  }
}

static void probe_ok(cudaError_t e, const char *what) {
  if (e != cudaSuccess) throw std::runtime_error(std::string("CUDA error in ") + what + ": " + cudaGetErrorString(e));
}

// Reductions per second (1e9) over a buffer of `bytes` bytes, `n_ops` reductions in total
// (after one untimed launch of the same size).
double measure_random_reduction_rate(size_t bytes, long long n_ops) {
  const unsigned long long n_elem = bytes / sizeof(double);
  if (n_elem < 1 || n_ops < 1) throw std::runtime_error("reduction probe: empty buffer or no operations");
  int dev = 0, n_sm = 0;
  probe_ok(cudaGetDevice(&dev), "device");
  probe_ok(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev), "attribute");
  const int threads = 256, blocks = n_sm * 8;
  const long long per = (n_ops + (long long)threads * blocks - 1) / ((long long)threads * blocks);
  double *buf = nullptr;
  probe_ok(cudaMalloc(&buf, n_elem * sizeof(double)), "cudaMalloc");
  cudaEvent_t a, b;
  cudaEventCreate(&a);
  cudaEventCreate(&b);
  float ms = 0.0f;
  cudaError_t err = cudaMemset(buf, 0, n_elem * sizeof(double));
  if (err == cudaSuccess) {
    random_reduction_kernel<<<blocks, threads>>>(buf, n_elem, per, 12345u);
    cudaEventRecord(a);
    random_reduction_kernel<<<blocks, threads>>>(buf, n_elem, per, 67890u);
    cudaEventRecord(b);
    err = cudaEventSynchronize(b);
    if (err == cudaSuccess) err = cudaEventElapsedTime(&ms, a, b);
  }
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  cudaFree(buf);
  probe_ok(err, "reduction probe");
  return (double)per * threads * blocks / (ms * 1e-3) / 1e9;
}

// ---------------------------------------------------------------------------
// The branch-free reciprocal and quotient of ngpu_math.cuh against the compiler's correctly
// rounded ones: every float from 1/16 up to 2^126, and every quotient that log_m forms.
// ---------------------------------------------------------------------------
constexpr unsigned RCP_FIRST = 0x3d800000u, RCP_END = 0x7e800000u;   // 1/16, 2^126
constexpr unsigned LOG_FIRST = 0x3f3504f0u, LOG_LAST = 0x3fb504f8u;  // sqrt(1/2) .. sqrt(2)

// n[0]: inputs on which they differ; n[1]: inputs compared
__global__ void check_rounded_kernel(unsigned long long *n_out) {
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  const unsigned long long i0 = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
  unsigned long long n = 0, seen = 0;
  for (unsigned long long b = RCP_FIRST + i0; b < RCP_END; b += stride, seen++) {
    const float x = __uint_as_float((unsigned)b);
    n += __float_as_uint(rcp_m(x)) != __float_as_uint(__frcp_rn(x));
  }
  for (unsigned long long b = LOG_FIRST + i0; b <= LOG_LAST; b += stride, seen++) {
    const float m = __uint_as_float((unsigned)b), num = __fsub_rn(m, 1.0f), den = __fadd_rn(m, 1.0f);
    n += __float_as_uint(div_m(num, den)) != __float_as_uint(__fdiv_rn(num, den));
  }
  if (n) atomicAdd(n_out, n);
  atomicAdd(n_out + 1, seen);
}

// Number of inputs on which they differ (-1: not all of them were compared).
long long check_rounded_ops() {
  unsigned long long *d = nullptr, h[2] = {0, 0};
  if (cudaMalloc(&d, sizeof(h)) != cudaSuccess) return -1;
  bool ok = cudaMemset(d, 0, sizeof(h)) == cudaSuccess;
  check_rounded_kernel<<<148 * 8, 256>>>(d);
  ok = cudaGetLastError() == cudaSuccess && ok;
  ok = cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost) == cudaSuccess && ok;
  cudaFree(d);
  const unsigned long long want = (unsigned long long)(RCP_END - RCP_FIRST) + (LOG_LAST - LOG_FIRST + 1);
  return ok && h[1] == want ? (long long)h[0] : -1;
}

}  // namespace ngpu
