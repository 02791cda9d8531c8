// FP64 products on the integer pipe.  GB300 issues one FP64 warp instruction per
// 19.4 SM cycles, and the exact schemes keep that pipe 83 to 90% busy while two
// thirds of the issue slots are idle.  A product here takes about 40 integer
// instructions (18 SM cycles when nothing else runs), beside the FP64 pipe: 8 of
// them next to 8 FP64 multiplications take 172 SM cycles, those 8 alone 165
// (measured, 20 warps per SM).  Sums stay where they are: their integer form, with
// its alignment and normalisation shifts, takes twice the instructions.
#pragma once
#include "fp64_div.cuh"

namespace mom5 {
namespace fp64 {

// a * b, the IEEE result.  Significands A, B in [2^52, 2^53): the top 85 of the 117
// bits of A * (B 2^11) are formed, 52 or 53 of them above bit 32, and rounded with
// the 32 below.  A remainder of exactly half (a tie, or the rare product with more
// bits below those), an a of an exponent outside 2^-511 .. 2^510, a b of one outside
// 2^-511 .. 2^512, Inf and NaN take the multiplication instruction.  So do zeros,
// unless ZA or ZB says that a or b is zero often enough to be given its own path.
// Shifts are written as products, which the multiply-add pipe does; the sum of the
// high words less the significands carries both the sign and the exponent.
template <bool ZA = false, bool ZB = false>
DEVI double mul_int(double a, double b) {
  const unsigned ah = (unsigned)__double2hiint(a), al = (unsigned)__double2loint(a);
  const unsigned bh = (unsigned)__double2hiint(b), bl = (unsigned)__double2loint(b);
  const unsigned a1 = (ah & 0xfffffu) | 0x100000u, bm = (bh & 0xfffffu) | 0x100000u;
  const unsigned long long bw = (unsigned long long)bl * 2048u;
  const unsigned b0 = (unsigned)bw, b1 = bm * 2048u + (unsigned)(bw >> 32);
  const unsigned long long p1 = (unsigned long long)al * b1 + __umulhi(al, b0);
  const unsigned long long p2 = (unsigned long long)a1 * b0 + (unsigned)p1;
  const unsigned long long q = (unsigned long long)a1 * b1 + (p1 >> 32) + (p2 >> 32);
  const unsigned qh = (unsigned)(q >> 32), s2 = 2u - (qh >> 20);  // 52 bits: one more from below
  const unsigned long long w0 = (unsigned long long)(unsigned)p2 * s2 + 0x80000000u;
  const unsigned long long w = (unsigned long long)(unsigned)q * s2 + (w0 >> 32);
  unsigned lo = (unsigned)w;
  unsigned hi = qh * s2 + (unsigned)(w >> 32) + (ah - a1) + (bh - bm) + (qh & 0x100000u) - 0x3fe00000u;
  // exponent fields in 0x200 .. 0x5fd and 0x200 .. 0x5ff
  const unsigned ra = ah * 2u - 0x40000000u, rb = bh * 2u - 0x40000000u;
  bool oka = ra < 0x7fc00000u, okb = (int)rb >= 0, tie = (unsigned)w0 == 0, zero = false;
  if (ZA) {
    const bool z = ((ah << 1) | al) == 0;
    oka = oka || z;
    zero = z;
  }
  if (ZB) {
    const bool z = ((bh << 1) | bl) == 0;
    okb = okb || z;
    zero = zero || z;
  }
  if ((ZA || ZB) && zero) lo = 0, hi = (ah ^ bh) & 0x80000000u, tie = false;
  double x = __hiloint2double((int)hi, (int)lo);
  rare_lanes(!(oka && okb && !tie), [&] { x = a * b; });
  return x;
}

}  // namespace fp64
}  // namespace mom5
