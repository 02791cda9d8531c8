// The FP64 division (mom5_gb300/csrc/fp64_div.cuh) where its argument has no slack.
//
// 1. Every pattern of a divisor's 24 leading bits, with the bits below all zero, all
//    one and mixed, and with every reciprocal within the stated 2^-23 of the true one
//    (not only the one this chip's rcp.approx gives): dividends one and two units below
//    and above the divisor, equal to it, all ones, 1 and mixed.  rcp.approx itself is
//    checked against 2^-23 over the same patterns.
// 2. The edges of the exponent range the integer path takes, for dividend and divisor,
//    where the quotient overflows or goes subnormal.
//
// Every quotient must equal the division instruction's, bit for bit (NaN payloads
// aside).  Prints "ok <cases>" and exits 0, else the first mismatches and exits 1.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <stdio.h>

#include "fp64_div.cuh"

using namespace mom5::fp64;

struct Bad {
  double a, b, got, want;
  float y;
};

__device__ unsigned long long cases, bad, rcp_bad;
__device__ Bad first_bad[8];

__device__ uint64_t mix(uint64_t z) {  // splitmix64's output function
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
  return z ^ (z >> 31);
}
__device__ void check(double a, double b, float y, double got) {
  const double want = a / b;
  if (__double_as_longlong(got) == __double_as_longlong(want) || (got != got && want != want)) return;
  const unsigned long long n = atomicAdd(&bad, 1ULL);
  if (n < 8) first_bad[n] = {a, b, got, want, y};
}

__global__ void k_significands() {
  const uint64_t lead = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;  // 23 fraction bits
  if (lead >= 1u << 23) return;
  const float xt = __uint_as_float(0x3f800000u | (unsigned)lead);
  const double r = 1.0 / (double)xt;
  float hw;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(hw) : "f"(xt));
  if (fabs((double)hw - r) > 0x1p-23) atomicAdd(&rcp_bad, 1ULL);
  unsigned long long done = 0;
  const unsigned near = __float_as_uint((float)r);
  for (int low = 0; low < 3; ++low) {
    const uint64_t rnd = mix(lead * 3 + low + 1);
    const uint64_t tail = low == 0 ? 0 : low == 1 ? 0x1fffffffULL : rnd & 0x1fffffffULL;
    const uint64_t bb = 0x3ff0000000000000ULL | (lead << 29) | tail;
    const double b = __longlong_as_double((long long)bb);
    const uint64_t frac = 0x000fffffffffffffULL, one = 0x3ff0000000000000ULL;
    const uint64_t as[] = {bb, bb - 1, bb - 2, bb + 1, bb + 2, one | frac, one, one | (mix(rnd) & frac)};
    for (int d = -8; d <= 8; ++d) {
      const float y = __uint_as_float(near + (unsigned)d);
      if (fabs((double)y - r) > 0x1p-23) continue;
      const Divisor dv = divisor_with(b, y);
      for (int q = 0; q < 8; ++q) {
        const double a = __longlong_as_double((long long)as[q]);
        check(a, b, y, div_by(a, b, dv));
        ++done;
      }
    }
  }
  atomicAdd(&cases, done);
}

// exponent fields at the edges, significands mixed, all zero and all one
__global__ void k_exponents() {
  const unsigned e[] = {0x000, 0x001, 0x1fe, 0x1ff, 0x200, 0x201, 0x202, 0x203, 0x3fe, 0x3ff,
                        0x400, 0x5fd, 0x5fe, 0x5ff, 0x600, 0x601, 0x7fe, 0x7ff};
  const unsigned ne = sizeof(e) / sizeof(e[0]), t = blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned kind = t >> 10;
  if (kind >= ne * ne) return;
  const uint64_t ra = mix(2 * t + 1), rb = mix(2 * t + 2);
  auto value = [](unsigned field, uint64_t r) {
    uint64_t m = r & 0x800fffffffffffffULL;
    if ((r >> 60 & 3) == 0) m &= 0x8000000000000000ULL;
    if ((r >> 60 & 3) == 1) m |= 0x000fffffffffffffULL;
    return __longlong_as_double((long long)(m | (uint64_t)field << 52));
  };
  const double a = value(e[kind / ne], ra), b = value(e[kind % ne], rb);
  check(a, b, 0.0f, div_seeded(a, b));
  double yh, yl;
  recip_pair(b, yh, yl);
  check(a, b, 0.0f, div_pair(a, b, yh, yl));
  atomicAdd(&cases, 2ULL);
}

int main() {
  k_significands<<<(1u << 23) / 128, 128>>>();
  k_exponents<<<18 * 18 * 1024 / 128, 128>>>();
  unsigned long long n = 0, nb = 0, nr = 0;
  Bad f[8];
  if (cudaDeviceSynchronize() != cudaSuccess || cudaMemcpyFromSymbol(&n, cases, sizeof(n)) != cudaSuccess ||
      cudaMemcpyFromSymbol(&nb, bad, sizeof(nb)) != cudaSuccess ||
      cudaMemcpyFromSymbol(&nr, rcp_bad, sizeof(nr)) != cudaSuccess ||
      cudaMemcpyFromSymbol(f, first_bad, sizeof(f)) != cudaSuccess) {
    printf("CUDA error\n");
    return 2;
  }
  for (unsigned long long i = 0; i < nb && i < 8; ++i)
    printf("%a / %a = %a, not %a (reciprocal %a)\n", f[i].a, f[i].b, f[i].got, f[i].want, (double)f[i].y);
  if (nr) printf("rcp.approx further than 2^-23 from the reciprocal in %llu patterns\n", nr);
  if (nb || nr) {
    printf("%llu of %llu cases differ\n", nb, n);
    return 1;
  }
  printf("ok %llu\n", n);
  return 0;
}
