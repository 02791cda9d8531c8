// Correctly rounded FP64 division without FP64 instructions, and the exact
// shortcut of the limiters' 1e-30 + x.  GB300 issues FP64 at 1/64 of the FP32
// rate, so the exact schemes are bound by their FP64 instruction count; a
// quotient here is a long division on the integer pipe, and a lane outside its
// range takes the division instruction, so every function returns exactly the
// IEEE result.
#pragma once
#include <math.h>

namespace mom5 {
namespace fp64 {

#define DEVI __device__ __forceinline__

// Bit pattern of a double and back through an opaque move.  With a plain bit
// cast the compiler rewrites some integer tests as FP64 instructions (a masked
// sign bit becomes an FP64 absolute value); through the move they stay on the
// integer pipe.
DEVI long long bits_of(double x) {
  long long b;
  asm("mov.b64 %0, %1;" : "=l"(b) : "d"(x));
  return b;
}
DEVI double double_of(long long b) {
  double x;
  asm("mov.b64 %0, %1;" : "=d"(x) : "l"(b));
  return x;
}

// f() for the lanes with `rare` set, in a loop that runs once: the assembler turns
// a branch around a few instructions into predicated ones, and an FP64
// instruction takes its 19.4 cycles of the pipe with every lane switched off too
// (measured: a product on the integer pipe whose fallback was a branch left the
// FP64 pipe's instruction count as it was).
template <class F>
DEVI void rare_lanes(bool rare, F&& f) {
  const unsigned act = __activemask();
  for (unsigned m = __ballot_sync(act, rare); m; m &= ~act)
    if (rare) f();
}

// Quotients by long division on the integer pipe.  GB300 issues one FP64 warp
// instruction per 19.4 SM cycles (measured; the number of active lanes does not
// matter), an integer one per 0.3 to 0.5 (the 64-bit product and the high half
// of a product per 1.1), so a division in integers leaves the FP64 pipe to the
// additions and products: 26 SM cycles per warp and none of them on the FP64
// pipe, against 76 for the Markstein correction of an FP32 reciprocal with its
// FP64 proof (4 FP64 instructions) and 140 for the division instruction.  The
// advection step of 10 tracers on 360x270x50 cells went from 7.34 to 5.42 ms
// with it, that of 2 tracers on 120x80x30 from 0.143 to 0.102 ms.
//
// With significands A, B in [2^52, 2^53) three digits of 18 bits give
// Q = floor(A 2^54 / B), in (2^53, 2^55).  A digit is the high half of the
// remainder's top bits times Y, a 24-bit reciprocal of B rounded down, so it is
// never above the true digit and at most one below it: Y is rcp.approx of B's
// 24 leading bits (within 2^-23 of the reciprocal on [1, 2), that is two units
// of 2^-24, and at most two more too large for the bits cut from B) less four
// units, hence below 2^24 2^52/B by at most 2^-20.4 of it, and a digit is below
// 2^19.  Every remainder is then in [0, 2B), so arithmetic modulo 2^64 is
// exact, and the last one says whether one more belongs to Q.  The reciprocal is held
// to [1/2, 1 - 2^-24], where the true one lies too (but for B = 2^52, whose 1 loses
// one unit): outside it the 24 bits would not start at the same place, and next to
// both ends the error of rcp.approx reaches outside.  A quotient of two 53-bit
// significands is never the midpoint of two doubles, so Q's bits below the result's
// last one round it correctly without a sticky bit.
//
// Dividends of an exponent within 2^-509 .. 2^512 over divisors within
// 2^-511 .. 2^512 take this path, and a zero dividend with such a divisor; any other
// lane takes the division instruction, so every function returns exactly the IEEE
// result.
//
// Shifts are written as products where that lets the multiply-add pipe do them:
// with the products of the schemes on the integer pipe too, the adder and logic
// pipe is what bounds the rest.
struct Divisor {
  unsigned ex, nlo, nhi, y;  // sign and exponent of b (its high word less the significand's); -B modulo 2^64; 24-bit reciprocal
};
// The divisor b given rcp.approx of its 24 leading bits.
DEVI Divisor divisor_with(double b, float y) {
  const unsigned hi = (unsigned)__double2hiint(b), lo = (unsigned)__double2loint(b);
  const unsigned m = (hi & 0xfffffu) | 0x100000u;
  const unsigned yb = min(max(__float_as_uint(y), 0x3f000000u), 0x3f7fffffu);
  const unsigned long long nb = 0ULL - (((unsigned long long)m << 32) | lo);
  return {hi - m, (unsigned)nb, (unsigned)(nb >> 32), ((yb & 0x7fffffu) | 0x800000u) - 4u};
}
DEVI Divisor divisor_of(double b) {
  const unsigned hi = (unsigned)__double2hiint(b), lo = (unsigned)__double2loint(b);
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float((__funnelshift_l(lo, hi, 3) & 0x7fffffu) | 0x3f800000u)));
  return divisor_with(b, y);
}
// The next 18-bit digit of r / B; r becomes the remainder.
DEVI unsigned div_digit(unsigned long long& r, const Divisor& d) {
  const unsigned q = __umulhi((unsigned)(r >> 26), d.y), rh = (unsigned)(r >> 32);
  r = (unsigned long long)(unsigned)r * (1u << 18) + (unsigned long long)q * d.nlo;
  r += (unsigned long long)(q * d.nhi + rh * (1u << 18)) << 32;
  return q;
}
DEVI double div_by(double a, double b, const Divisor& d) {
  const unsigned ah = (unsigned)__double2hiint(a), al = (unsigned)__double2loint(a);
  const unsigned am = (ah & 0xfffffu) | 0x100000u;
  unsigned long long r = ((unsigned long long)am << 32) | al;
  const unsigned q1 = div_digit(r, d), q2 = div_digit(r, d), q3 = div_digit(r, d);
  const unsigned long long q = (unsigned long long)q2 * (1u << 18) + q3;
  unsigned ql, qh;
  // r + (-B) carries out of 64 bits where r >= B
  asm("{\n .reg .u32 t;\n add.cc.u32 t, %2, %4;\n addc.cc.u32 t, %3, %5;\n addc.cc.u32 %0, %6, 0;\n addc.u32 %1, %7, 0;\n}"
      : "=r"(ql), "=r"(qh)
      : "r"((unsigned)r), "r"((unsigned)(r >> 32)), "r"(d.nlo), "r"(d.nhi), "r"((unsigned)q),
        "r"((unsigned)(q >> 32) + q1 * 16u));
  // one or two bits lie below the result's last: Q 2^31 or 2^30 plus half of 2^32, over 2^32
  const unsigned top = qh >> 22, m = 0x80000000u >> top;
  const unsigned long long w0 = (unsigned long long)ql * m + 0x80000000u;
  const unsigned long long w = (unsigned long long)qh * m + (w0 >> 32);
  // the signs' sum and the exponents' difference; w's leading bit adds one to the field
  unsigned lo = (unsigned)w, hi = (unsigned)(w >> 32) + (ah - am - d.ex) + 0x3fd00000u + top * 0x100000u;
  const unsigned eb = (d.ex + 0x100000u) * 2u - 0x40000000u;
  const bool bn = (int)eb >= 0, zero = ((ah << 1) | al) == 0;
  const bool ok = bn && (zero || ah * 2u - 0x40400000u < 0x7fc00000u);
  if (zero) lo = 0, hi = (ah ^ d.ex) & 0x80000000u;
  double x = __hiloint2double((int)hi, (int)lo);
  rare_lanes(!ok, [&] { x = a / b; });
  return x;
}

// a / b for a divisor used once.
DEVI double div_seeded(double a, double b) { return div_by(a, b, divisor_of(b)); }

// A divisor shared by many quotients, kept in two doubles' bits: yh holds its
// reciprocal, yl the negated significand.
DEVI void recip_pair(double b, double& yh, double& yl) {
  const Divisor d = divisor_of(b);
  yh = __hiloint2double((int)d.ex, (int)d.y);
  yl = __hiloint2double((int)d.nhi, (int)d.nlo);
}
DEVI double div_pair(double a, double b, double yh, double yl) {
  return div_by(a, b, {(unsigned)__double2hiint(yh), (unsigned)__double2loint(yl), (unsigned)__double2hiint(yl),
                       (unsigned)__double2loint(yh)});
}

// RN(1e-30 + x) without an FP64 addition where that is exact by inspection:
// +-0 gives the constant 1e-30, and for |x| >= 2^-45 (biased exponent >= 978)
// the sum rounds back to x (1e-30 is below half an ulp of x, also of the
// binade under x when x is a negative power of two).  Tiny non-zero x, Inf and
// NaN take the addition.
DEVI double add_1em30(double x) {
  long long b = bits_of(x);
  unsigned e = (unsigned)((unsigned long long)b >> 52) & 0x7ffu;
  bool zero = (b << 1) == 0;
  bool keep = e >= 978u && e <= 2046u;
  double r = zero ? 1.0e-30 : x;
  rare_lanes(!(zero || keep), [&] { r = 1.0e-30 + x; });
  return r;
}

}  // namespace fp64
}  // namespace mom5
