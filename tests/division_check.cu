// Compares the device functions div_by and Divisor::quot (csrc/step_kernels.cuh)
// with the hardware's correctly rounded division, for tests/test_gpu_division.py.
#include "step_kernels.cuh"

using qg::div_by;
using qg::Divisor;

namespace {
__device__ unsigned long long mix(unsigned long long z) {
  z += 0x9e3779b97f4a7c15ull;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}
// a double of random sign and mantissa with a biased exponent in [e0, e1]
__device__ double draw(unsigned long long r, int e0, int e1) {
  const unsigned long long e = (unsigned long long)(e0 + (int)((r >> 52) % (unsigned)(e1 - e0 + 1)));
  return __longlong_as_double((long long)((mix(r) & 0x800fffffffffffffull) | e << 52));
}
__device__ bool same(double x, double y) {
  return __double_as_longlong(x) == __double_as_longlong(y) || (x != x && y != y);
}
__global__ void k_random(unsigned long long seed, long long n, int e0, int e1, unsigned long long* bad) {
  unsigned long long b = 0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const double a = draw(mix(seed + 2 * i), e0, e1), d = draw(mix(seed + 2 * i + 1), e0, e1);
    b += !same(div_by(a, d, __drcp_rn(d)), __ddiv_rn(a, d));
  }
  if (b) atomicAdd(bad, b);
}
__global__ void k_list(int n, const double* a, const double* d, const double* r, double* q, double* exact) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  q[i] = div_by(a[i], d[i], r[i]);
  exact[i] = __ddiv_rn(a[i], d[i]);
}
__global__ void k_quot(int n, const double* a, Divisor d, double* q, double* exact) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  q[i] = d.quot(a[i]);
  exact[i] = __ddiv_rn(a[i], d.d);
}
}  // namespace

// quotients of n random operands, exponents in [e0, e1], that differ from the
// hardware's; -1 on a CUDA error
extern "C" long long division_random(unsigned long long seed, long long n, int e0, int e1) {
  unsigned long long *d = nullptr, h = 0;
  if (cudaMalloc(&d, sizeof h) != cudaSuccess || cudaMemset(d, 0, sizeof h) != cudaSuccess) return -1;
  k_random<<<152 * 8, 256>>>(seed, n, e0, e1, d);
  const bool ok = cudaGetLastError() == cudaSuccess && cudaMemcpy(&h, d, sizeof h, cudaMemcpyDeviceToHost) == cudaSuccess;
  cudaFree(d);
  return ok ? (long long)h : -1;
}
// div_by (one = 0) or Divisor(d[0]).quot (one = 1) of the n operands, and the
// hardware's quotients; device arrays
extern "C" int division_list(int n, int one, const double* a, const double* d, const double* r, double* q, double* exact) {
  if (one) {
    double x = 0.0;
    if (cudaMemcpy(&x, d, sizeof x, cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
    k_quot<<<(n + 255) / 256, 256>>>(n, a, Divisor(x), q, exact);
  } else {
    k_list<<<(n + 255) / 256, 256>>>(n, a, d, r, q, exact);
  }
  return cudaGetLastError() != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess;
}
