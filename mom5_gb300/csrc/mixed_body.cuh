// Arithmetic and indexing of the precision-form MDFL tile (mixed_stream.cuh).
#pragma once
#include <math.h>

#include "internal.h"

namespace mom5 {
namespace mixed {

#define DEVI __device__ __forceinline__


constexpr int ZW = 32;       // tile width incl. the 2-cell halo on each side (one warp)
constexpr int TI = ZW - 4;   // interior width

DEVI long I2(const Geo& g, int i, int j) { return (long)j * g.nxd + i; }
DEVI long I3(const Geo& g, int i, int j, int k) { return (long)k * g.n2 + (long)j * g.nxd + i; }
DEVI long IM(const Geo& g, int i, int j, int k) { return ((long)k * (g.nj + 4) + (j + 1)) * (g.ni + 4) + (i + 1); }

// FP64 -> FP32 by truncation of the significand, with integer operations.
DEVI float d2f(double x) {
  unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  unsigned sign = hi & 0x80000000u, mag = hi & 0x7fffffffu;
  if (mag < (897u << 20)) return __uint_as_float(sign);
  if (mag >= (1151u << 20)) return __uint_as_float(sign | 0x7f800000u);
  return __uint_as_float(sign | ((mag - (896u << 20)) << 3) | (lo >> 29));
}
// FP64 -> FP32 rounded to nearest (ties away from zero): half an FP32 ulp added
// to the bit pattern, then truncated.
DEVI float d2f_rn(double x) { return d2f(__longlong_as_double(__double_as_longlong(x) + (1LL << 28))); }
// FP32 -> FP64, exact, with integer operations (subnormal floats read as zero).
DEVI double f2d(float f) {
  unsigned b = __float_as_uint(f);
  unsigned sign = b & 0x80000000u, mag = b & 0x7fffffffu;
  if (mag < 0x00800000u) return __hiloint2double((int)sign, 0);
  return __hiloint2double((int)(sign | ((mag >> 3) + (896u << 20))), (int)(mag << 29));
}

// The FP32 arithmetic of the precision form.  Every product and sum is rounded
// on its own (__fmul_rn / __fadd_rn / __fsub_rn are never contracted into a
// multiply-add), so the result of a formula does not depend on how the compiler
// schedules the kernel around it: every launch shape gives the same bits.
DEVI float fm(float a, float b) { return __fmul_rn(a, b); }
DEVI float fa(float a, float b) { return __fadd_rn(a, b); }
DEVI float fs(float a, float b) { return __fsub_rn(a, b); }

// a / b as a times the hardware reciprocal (at most two ulps, as __fdividef, whose
// bits it gives for normal b: no divisor here is subnormal, 1e-30 + x with x of
// FP32 spacing included; |b| above 2^126 gives 0, as there)
DEVI float rcp(float b) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(b));
  return r;
}
DEVI float fdiv(float a, float b) { return fm(a, rcp(b)); }

// d0, d1 and the limiter slope (1-cfl)/(1e-30+cfl) of a Courant number
DEVI void cfl_terms(float cfl, float& d0, float& d1, float& c) {
  const float sixth = 1.0f / 6.0f;
  d0 = fm(fm(fs(2.0f, cfl), fs(1.0f, cfl)), sixth);
  d1 = fm(fs(1.0f, fm(cfl, cfl)), sixth);
  c = fdiv(fs(1.0f, cfl), fa(1.0e-30f, cfl));
}
// vertical face terms of a column: mass flux dat*w, cfl = |w*dt/rho_dzt|
DEVI void z_terms(float wk, float wkm1, float rdz, float dat, float dt, float& mf, float& d0, float& d1, float& c,
                  float& dtr, float& wd) {
  float rr = 1.0f / rdz;
  mf = fm(dat, wk);
  cfl_terms(fabsf(fm(fm(wk, dt), rr)), d0, d1, c);
  dtr = fm(dt, rr);
  wd = fs(wkm1, wk);
}
// horizontal face terms: mass flux len*u, cfl = |u*dt*2/((rdz + rdz_nb)*dist)|
DEVI void h_terms(float u, float len, float rdz, float rdz_nb, float dist, float dt, float& mf, float& d0, float& d1,
                  float& c) {
  mf = fm(len, u);
  float den = fm(fa(rdz, rdz_nb), dist);
  cfl_terms(fabsf(fdiv(fm(fm(u, dt), 2.0f), den)), d0, d1, c);
}
// x-cell terms: dtime*datr/rho_dzt where wet, and the x divergence dyte*uh - dyte(i-1)*uh(i-1)
DEVI float x_coef(bool wet, float dt, float datr, float rdz) { return wet ? fm(dt, datr) / rdz : 0.0f; }
DEVI float x_div(float dyte, float uh, float dyte_w, float uh_w) { return fs(fm(dyte, uh), fm(dyte_w, uh_w)); }

// image of a tile position under the single-domain halo rules; false when it lies
// outside a non-cyclic boundary (the reference's halo holds zero there)
DEVI bool image(const Geo& g, int& i, int& j) {
  if (i < 1 || i > g.ni) {
    if (!g.cx) return false;
    i = ((i - 1) % g.ni + g.ni) % g.ni + 1;
  }
  if (j < 1 || j > g.nj) {
    if (!g.cy) return false;
    j = ((j - 1) % g.nj + g.nj) % g.nj + 1;
  }
  return true;
}

DEVI bool mask_at(const Geo& g, const uint8_t* m2, int i, int j, int k) {
  if (i < -1 || i > g.ni + 2 || j < -1 || j > g.nj + 2) return false;
  return m2[IM(g, i, j, k)] != 0;
}

// Stream-ordered 8-byte copy global -> shared (cp.async, L1-allocating); src_size 0
// fills the destination with zeros and reads nothing.
DEVI void cp_async8(void* dst, const void* src, int src_size) {
  unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src), "r"(src_size) : "memory");
}
DEVI void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
DEVI void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

}  // namespace mixed
}  // namespace mom5
