// rcp_positive of qas_device.cuh on the device, bit for bit against 1.0/x: the largest and the smallest
// significands and those around a half at every exponent of its range, and the error of its seed, of which the
// derivation uses no more than 2^-14.  Prints both, exits 1 where either fails.
#include <cmath>
#include <cstdio>

#include "qas_device.cuh"

using namespace qas;

constexpr int E_LO = 1023 - 999, E_N = 1999, NEAR = 512;

// significand s of a set: k from the top, from the bottom, around 1.5, and spread over the binade
__device__ double point(int e, int set, unsigned long long k)
{
  const unsigned long long top = (1ull << 52) - 1, m = set == 0 ? top - k : set == 1 ? k : set == 2 ? (top >> 1) - NEAR / 2 + k
                                                                       : (k * 0x9E3779B97F4A7C15ull) >> 12;
  return __longlong_as_double((long long)(((unsigned long long)e << 52) | m));
}

__global__ void k_points(unsigned long long *bad)
{
  const long long n = (long long)E_N * 4 * NEAR;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
    const double x = point(E_LO + (int)(t / (4 * NEAR)), (int)(t / NEAR % 4), t % NEAR);
    if (__double_as_longlong(rcp_positive(x)) != __double_as_longlong(1.0 / x)) atomicAdd(bad, 1ull);
  }
}

// largest |1 - x*seed| over 2^28 significands of [1, 2), by the bits of the (positive) error
__global__ void k_seed(unsigned long long *worst)
{
  double w = 0.0;
  for (unsigned long long t = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; t < 1ull << 28;
       t += (unsigned long long)gridDim.x * blockDim.x) {
    const double x = __longlong_as_double((long long)((1023ull << 52) | (t << 24) | (t * 0x9E3779B97F4A7C15ull >> 40)));
    w = fmax(w, fabs(fma(-x, rcp_seed(x), 1.0)));
  }
  atomicMax(worst, (unsigned long long)__double_as_longlong(w));
}

int main()
{
  unsigned long long *d, h[2] = {0, 0};
  if (cudaMalloc(&d, sizeof(h)) != cudaSuccess || cudaMemset(d, 0, sizeof(h)) != cudaSuccess) return 2;
  k_points<<<1184, 256>>>(&d[0]);
  k_seed<<<1184, 256>>>(&d[1]);
  if (cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
  cudaFree(d);
  double seed;
  memcpy(&seed, &h[1], sizeof(seed));
  printf("%llu differing, seed error 2^%.2f\n", h[0], log2(seed));
  return h[0] || !(seed < ldexp(1.0, -14)) ? 1 : 0;
}
