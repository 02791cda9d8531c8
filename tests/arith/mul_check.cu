// Exactness check of the FP64 product on the integer pipe
// (mom5_gb300/csrc/fp64_mul.cuh): for every case the bit pattern must equal the
// multiplication instruction's and the host's (NaN payloads aside), in each of the
// four forms (with and without a path of its own for a zero first or second
// operand).  Cases: uniformly random bit patterns (every exponent, subnormals, Inf,
// NaN), moderate exponents, significands with few bits (exact products and ties),
// zeros, and the edges of the exponent range the integer path takes, where the
// product overflows or goes subnormal.  Prints "ok <cases>" and exits 0, else lists
// the first mismatches and exits 1.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include <vector>

#include "fp64_mul.cuh"

__global__ void k_mul(const double* a, const double* b, double* p, long n) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  p[i] = mom5::fp64::mul_int<false, false>(a[i], b[i]);
  p[n + i] = mom5::fp64::mul_int<true, false>(a[i], b[i]);
  p[2 * n + i] = mom5::fp64::mul_int<false, true>(a[i], b[i]);
  p[3 * n + i] = mom5::fp64::mul_int<true, true>(a[i], b[i]);
  p[4 * n + i] = a[i] * b[i];
}

static uint64_t s_state = 0x243f6a8885a308d3ULL;
static uint64_t next_u64() {  // splitmix64
  uint64_t z = (s_state += 0x9e3779b97f4a7c15ULL);
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
  return z ^ (z >> 31);
}
static double from_bits(uint64_t u) {
  double d;
  memcpy(&d, &u, 8);
  return d;
}
static uint64_t bits(double d) {
  uint64_t u;
  memcpy(&u, &d, 8);
  return u;
}
// a value of exponent field e with the lowest `cut` significand bits zero
static double value(unsigned e, int cut) {
  uint64_t m = next_u64() & 0x800fffffffffffffULL;
  m &= ~((1ULL << cut) - 1) | 0x8000000000000000ULL;
  return from_bits(m | ((uint64_t)(e & 0x7ff) << 52));
}

int main() {
  std::vector<double> A, B;
  auto add = [&](double a, double b) {
    A.push_back(a);
    B.push_back(b);
  };
  for (int i = 0; i < 1 << 20; ++i) add(from_bits(next_u64()), from_bits(next_u64()));
  for (int i = 0; i < 1 << 20; ++i) add(value(963 + next_u64() % 121, 0), value(963 + next_u64() % 121, 0));
  for (int i = 0; i < 1 << 20; ++i)  // 53 to 54 bits in the product: exact or a tie
    add(value(1013 + next_u64() % 20, 20 + next_u64() % 10), value(1013 + next_u64() % 20, 22 + next_u64() % 10));
  const unsigned edge[] = {0x000, 0x001, 0x1ff, 0x200, 0x201, 0x3fe, 0x5fc, 0x5fd, 0x5fe, 0x5ff, 0x600, 0x7fe, 0x7ff};
  for (unsigned ea : edge)
    for (unsigned eb : edge)
      for (int i = 0; i < 2048; ++i) add(value(ea, i % 53), value(eb, (i / 53) % 53));
  const double special[] = {0.0, -0.0, 1.0, -1.0, INFINITY, -INFINITY, NAN, 5e-324, 0x1p-511, 0x1p512, 1e-30};
  for (double x : special)
    for (int i = 0; i < 1 << 12; ++i) {
      add(x, i & 1 ? value(next_u64() % 2048, 0) : special[next_u64() % 11]);
      add(value(next_u64() % 2048, 0), x);
    }
  const long n = (long)A.size();
  double *a, *b, *p;
  cudaMalloc(&a, n * 8);
  cudaMalloc(&b, n * 8);
  cudaMalloc(&p, 5 * n * 8);
  cudaMemcpy(a, A.data(), n * 8, cudaMemcpyHostToDevice);
  cudaMemcpy(b, B.data(), n * 8, cudaMemcpyHostToDevice);
  k_mul<<<(unsigned)((n + 255) / 256), 256>>>(a, b, p, n);
  std::vector<double> P(5 * n);
  if (cudaMemcpy(P.data(), p, 5 * n * 8, cudaMemcpyDeviceToHost) != cudaSuccess) {
    printf("CUDA error\n");
    return 1;
  }
  long bad = 0;
  for (long i = 0; i < n; ++i) {
    volatile double host = A[i] * B[i];
    for (int f = 0; f < 5; ++f) {
      const double x = P[f * n + i];
      if (bits(x) == bits(host) || (isnan(x) && isnan(host))) continue;
      if (bad++ < 10) printf("form %d: %a * %a = %a, not %a\n", f, A[i], B[i], x, (double)host);
    }
  }
  if (bad) return 1;
  printf("ok %ld\n", n);
  return 0;
}
