// The exact shortcuts of mom5_gb300/csrc/fp64_bodies.cuh -- half, double, quarter and
// the product by a mask of 0 or 1 -- against the multiplication instruction, bit for bit
// (NaN payloads aside): every exponent field with mixed, all-zero and all-one
// significands and both signs, every subnormal magnitude around a tie, and random bit
// patterns.  Prints "ok <cases>" and exits 0, else the first mismatches and exits 1.
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include "fp64_bodies.cuh"

using namespace mom5::fp64;

__device__ unsigned long long cases, bad;

__device__ uint64_t mix(uint64_t z) {  // splitmix64's output function
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
  return z ^ (z >> 31);
}
__device__ void check(const char* what, double x, double got, double want) {
  atomicAdd(&cases, 1ULL);
  if (__double_as_longlong(got) == __double_as_longlong(want) || (got != got && want != want)) return;
  if (atomicAdd(&bad, 1ULL) < 8)
    printf("%s of %llx: %llx, not %llx\n", what, __double_as_longlong(x), __double_as_longlong(got),
           __double_as_longlong(want));
}

__global__ void k_check(double half, double two, double quarter, double one, double zero) {
  const uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x, r = mix(t + 1);
  const uint64_t kind = t >> 17, n = t & 0x1ffff;
  uint64_t b;
  if (kind == 0) {  // 2048 exponent fields x 64 significands
    const uint64_t s = n & 63, f = n >> 6;
    const uint64_t m = s == 0 ? 0 : s == 1 ? 0xfffffffffffffULL : s < 16 ? s - 1 : s < 32 ? 0xfffffffffffffULL - (s - 16) : r >> 12;
    b = (r << 63) | (f << 52) | (m & 0xfffffffffffffULL);
  } else if (kind == 1) {  // magnitudes next to 0, 2^-1023 and 2^-1022, both signs
    const uint64_t base = n & 1 ? 0 : n & 2 ? 1ULL << 51 : 1ULL << 52;
    b = ((n & 4) << 61) | (base + (n >> 3) - (base ? 8192 : 0));
  } else {
    b = r;
  }
  const double x = __longlong_as_double((long long)b);
  check("half", x, half_exact(x), half * x);
  check("twice", x, twice(x), two * x);
  check("quarter", x, quarter_exact(x), quarter * x);
  check("x*1", x, mask_sel(x, 1.0), x * one);
  check("x*0", x, mask_sel(x, 0.0), x * zero);
  check("x*-0", x, mask_sel(x, -0.0), x * -zero);
}

int main() {
  k_check<<<(1u << 20) / 128, 128>>>(0.5, 2.0, 0.25, 1.0, 0.0);
  unsigned long long n = 0, nb = 0;
  if (cudaDeviceSynchronize() != cudaSuccess || cudaMemcpyFromSymbol(&n, cases, sizeof(n)) != cudaSuccess ||
      cudaMemcpyFromSymbol(&nb, bad, sizeof(nb)) != cudaSuccess) {
    printf("CUDA error\n");
    return 2;
  }
  if (nb) {
    printf("%llu of %llu cases differ\n", nb, n);
    return 1;
  }
  printf("ok %llu\n", n);
  return 0;
}
