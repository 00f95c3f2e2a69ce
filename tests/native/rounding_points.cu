// The short division forms of qas_device.cuh against the compiler's IEEE divisions, bit for bit, on
// the device: rcp_normal(x) == 1.0/x and div24(x) == x/24.  Prints the number of differing inputs
// per set and exits 1 if there are any.
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "qas_device.cuh"

using namespace qas;

__device__ unsigned long long mix(unsigned long long x)
{
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}
__device__ double from_bits(unsigned long long sign, unsigned long long e, unsigned long long m)
{
  return __longlong_as_double((long long)((sign << 63) | (e << 52) | (m & 0xFFFFFFFFFFFFFull)));
}
__device__ bool same(double a, double b)
{
  return __double_as_longlong(a) == __double_as_longlong(b) || (a != a && b != b);
}

// significands: random, near 1, near 2 (all ones and below), few bits set; exponents of the form's range
__global__ void k_rcp(unsigned long long n, unsigned long long seed, unsigned long long *bad)
{
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n;
       i += (unsigned long long)gridDim.x * blockDim.x) {
    const unsigned long long r = mix(i + seed), q = mix(r);
    unsigned long long m = r;
    switch (q & 7) {
      case 0: m = (q >> 8) & 1023; break;
      case 1: m = ~((q >> 8) & 1023); break;
      case 2: m = ~0ull; break;
      case 3: m = 1ull << ((q >> 8) % 52); break;
      case 4: m = ~(1ull << ((q >> 8) % 52)); break;
      default: break;
    }
    const double x = from_bits((q >> 3) & 1, 1023 - 999 + (q >> 20) % 1999, m);
    if (!same(rcp_normal(x), 1.0 / x)) atomicAdd(bad, 1ull);
  }
}
// every exponent, zeros, subnormals, infinities and NaN among them; multiples of 24 and of 12
__global__ void k_div24(unsigned long long n, unsigned long long seed, unsigned long long *bad)
{
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n;
       i += (unsigned long long)gridDim.x * blockDim.x) {
    const unsigned long long r = mix(i + seed), q = mix(r);
    double x;
    switch (q & 7) {
      case 0: x = (double)(long long)(r >> 16) * 24.0; break;
      case 1: x = (double)(long long)(r >> 16) * 12.0; break;
      case 2: x = from_bits((q >> 3) & 1, (q >> 20) % 8, r >> ((q >> 32) % 52)); break;
      case 3: x = from_bits((q >> 3) & 1, 100 + (q >> 20) % 60, r); break;
      case 4: x = from_bits((q >> 3) & 1, 2040 + (q >> 20) % 8, r & ((q >> 31) & 1 ? ~0ull : 0ull)); break;
      default: x = from_bits((q >> 3) & 1, (q >> 20) % 2048, r); break;
    }
    if (!same(div24(x), x / 24.0)) atomicAdd(bad, 1ull);
  }
}

int main(int argc, char **argv)
{
  const unsigned long long n = argc > 1 ? strtoull(argv[1], nullptr, 10) : 1ull << 28;
  unsigned long long *bad, h[2] = {0, 0};
  if (cudaMalloc(&bad, sizeof(h)) != cudaSuccess || cudaMemset(bad, 0, sizeof(h)) != cudaSuccess) return 2;
  k_rcp<<<1184, 256>>>(n, 1, &bad[0]);
  k_div24<<<1184, 256>>>(n, 2, &bad[1]);
  if (cudaMemcpy(h, bad, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
  printf("rcp_normal %llu div24 %llu differing of %llu\n", h[0], h[1], n);
  cudaFree(bad);
  return h[0] || h[1] ? 1 : 0;
}
