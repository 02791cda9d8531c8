// MDPPM (advect_tracer_mdppm, ocean_tracer_advect.F90:5990-6507): direction-split
// piecewise-parabolic advection, z then x then y, with the edge limiter chosen
// per tracer (ppm_hlimiter: 1 Colella-Woodward 1984 :6510-6538, 2 improved full
// constraint :6555-6580, 3 Suresh-Huynh 1997 :6601-6660; the reference applies
// it in all three directions).  FP64 in the reference's operation order; built
// with --fmad=false.
//
// A pass runs along lines of cells, one thread per position of a segment, stage by
// stage with a barrier between stages (tile_line).  Values outside the compute
// domain come from the halo of width 4 by the single-PE rules (periodic image, else
// 0) in the horizontal passes, as tracer_mdppm and tmask_mdppm hold them
// (mdppm_init :1702-1735), and from the nearest level, masked, in the vertical.
//
// Every pass is bound by the FP64 pipe, so what need not run there does not:
// products by powers of two, signs, masks, minima and maxima are integer
// operations, other products run on the integer pipe (mul_int), the one-sided
// differences of a cell serve its extrema too, and 6*S is formed once per cell.
// A masked or one-sided form is selected where the reference multiplies by masks
// (0 or 1: tracer_advect_init refuses others).
// 180x135x50 cells, 2 tracers: 1.88 -> 0.62 ms a step.
#pragma once

#include "fp64_bodies.cuh"
#include "fp64_select.cuh"
#include "internal.h"

namespace mom5 {
namespace ppm {

#define DEVI __device__ __forceinline__

constexpr double kR12 = 1.0 / 12.0, kSixth = 1.0 / 6.0, kTwoThirds = 2.0 / 3.0, kFourThirds = 4.0 / 3.0;

// a > b ? a : b and a < b ? a : b, compared on the integer pipe
DEVI double mx(double a, double b) { return sel::gt_max(a, b); }
DEVI double mn(double a, double b) { return sel::lt_min(a, b); }

using fp64::bits_of;
using fp64::double_of;
using fp64::half_exact;
using fp64::mul_int;
using fp64::neg_if;
using fp64::rare_lanes;
using fp64::twice;

DEVI bool negative(double x) { return bits_of(x) < 0; }
DEVI double magnitude(double x) { return double_of(bits_of(x) & 0x7fffffffffffffffLL); }

// Slope of a cell (:6064-6099): the two one-sided third-order estimates count half
// each where the cells two away are wet (m2, p2), or one of them whole, or neither;
// zero unless the cell and its neighbours are wet (inner).  S6m, S6, S6p: six times
// the cell and its neighbours; dm, dp: Si - Sim1 and Sip1 - Si, whose larger and
// smaller give the distances to the neighbours' extrema.
DEVI double slope(double Sim2, double Sim1, double Sip1, double Sip2, double S6m, double S6, double S6p, double dm,
                    double dp, bool m2, bool inner, bool p2) {
  const double da3m = mul_int<false, true>(kR12, twice(Sim2) - twice(S6m) + S6 + twice(twice(Sip1)));
  const double da3p =
      mul_int<false, true>(kR12, neg_if(twice(twice(Sim1)), true) - S6 + twice(S6p) - twice(Sip2));
  double a = m2 && p2 ? half_exact(da3m) + half_exact(da3p) : p2 ? da3p : da3m;
  rare_lanes(!m2 && !p2, [&] { a = 0.5 * (Sip1 - Sim1); });
  const double dMx = mx(mx(dp, neg_if(dm, true)), 0.0), dMn = mx(mx(neg_if(dp, true), dm), 0.0);
  const double d = mn(magnitude(a), twice(mn(dMx, dMn)));
  return inner ? neg_if(d, negative(a)) : 0.0;
}

DEVI void limit(int lim, double Si, double da, double d1m, double d1p, double d1mm, double d1pp, double& aL,
                double& aR) {
  if (lim == 1) {
    if (!sel::gt0((aR - Si) * (Si - aL))) {
      aL = Si;
      aR = Si;
    }
    double da2 = aR - aL, da4 = 0.5 * (aR + aL);
    double da3m = 6. * da2 * (Si - da4), da3p = da2 * da2;
    if (sel::ord0(da3m) > sel::ord0(da3p)) aL = 3. * Si - 2. * aR;
    if (sel::ord0(da3m) < sel::ord0(-da3p)) aR = 3. * Si - 2. * aL;
  } else if (lim == 2) {
    const double ada = magnitude(da);
    const bool neg = negative(da);
    aL = Si - neg_if(mn(ada, magnitude(aL - Si)), neg);
    aR = Si + neg_if(mn(ada, magnitude(aR - Si)), neg);
  } else {
    double Sim1 = Si - d1m, Sip1 = Si + d1p;
    double z = d1m - d1mm, w = d1p - d1m;
    double x = 4. * w - z, y = 4. * z - w;
    double dM4m = mx(0., mn(mn(mn(x, y), z), w)) + mn(0., mx(mx(mx(x, y), z), w));
    z = d1pp - d1p;
    x = 4. * w - z;
    y = 4. * z - w;
    double dM4p = mx(0., mn(mn(mn(x, y), z), w)) + mn(0., mx(mx(mx(x, y), z), w));
    double qAV = 0.5 * (Si + Sip1);
    x = d1p;
    y = 3. * d1m;
    double qMP = Si + mx(0., mn(x, y)) + mn(0., mx(x, y));
    double qUL = Si + y;
    double qLC = (Si + 0.5 * d1m) + kFourThirds * dM4m;
    double qMD = qAV - 0.5 * dM4p;
    double qMin = mx(mn(mn(qMD, Si), Sip1), mn(mn(Si, qUL), qLC));
    double qMax = mn(mx(mx(qMD, Si), Sip1), mx(mx(Si, qUL), qLC));
    if (sel::ord0((aR - Si) * (aR - qMP)) > sel::ord0(1.e-10)) aR = mn(mx(aR, qMin), qMax);
    qAV = 0.5 * (Si + Sim1);
    x = -d1m;
    y = -3. * d1p;
    qMP = Si + mx(0., mn(x, y)) + mn(0., mx(x, y));
    qUL = Si + y;
    qLC = (Si - 0.5 * d1p) + kFourThirds * dM4p;
    qMD = qAV - 0.5 * dM4m;
    qMin = mx(mn(mn(qMD, Si), Sim1), mn(mn(Si, qUL), qLC));
    qMax = mn(mx(mx(qMD, Si), Sim1), mx(mx(Si, qUL), qLC));
    if (sel::ord0((aL - Si) * (aL - qMP)) > sel::ord0(1.e-10)) aL = mn(mx(aL, qMin), qMax);
  }
}

// Flux through a face of mass flux mf from the cell it leaves, whose edge towards the
// face is E0, the other E1 and curvature E6, at Courant number cfl >= 0 (:6128-6145,
// :6293-6305, :6470-6482; against the flow the reference writes the same operations
// with their signs changed).
DEVI double upwind_flux(double mf, double cfl, double E0, double E1, double E6) {
  const double c = 1. - mul_int<false, true>(kTwoThirds, cfl);
  const double r = (E1 - E0) + mul_int<false, true>(c, E6);
  return mul_int<false, true>(mf, E0 + mul_int<true, true>(half_exact(cfl), r));
}

// The line's positions p0 .. p0+L-1 (lane = the line's slot): slopes, limited edge
// values, fluxes and updates; cells p0+4 .. p0+L-5 are updated (the first and last
// four positions only supply their neighbours).  S(pos), M(pos) give the tracer of
// and whether a cell is wet at any position in [-3, n+4]; face(pos, left, right) returns the flux through
// the wet face between cells pos and pos+1, left and right being their edge data;
// upd(pos, S, wet, Fw, Fe) applies the update of cell pos.  CLAMP: the slopes beyond
// the line's ends are those of its end cells.
struct Edges {
  double L, R, six;
};
template <int L, int BI>
struct LineSmem {
  double s[L][BI], q[L][BI], da[L][BI], l[L][BI], r[L][BI], f[L][BI];
  bool wet[L][BI];
};
template <int L, int BI, bool CLAMP, class FS, class FM, class FF, class FU>
DEVI void tile_line(int n, int lim, int p0, int t, int lane, bool lane_ok, LineSmem<L, BI>& sm, FS S, FM M, FF face,
                    FU upd) {
  const int p = p0 + t;
  double sv = 0.0;
  bool wet = false;
  if (lane_ok && p >= -3 && p <= n + 4) {
    sv = S(p);
    wet = M(p);
  }
  sm.s[t][lane] = sv;
  sm.wet[t][lane] = wet;
  const double s6 = mul_int<false, true>(6.0, sv);
  sm.q[t][lane] = s6;
  __syncthreads();
  // slope and one-sided differences of positions -1 .. n+2
  double da = 0.0, d1m = 0.0, d1p = 0.0, d1mm = 0.0, d1pp = 0.0;
  if (lane_ok && t >= 2 && t <= L - 3 && p >= -1 && p <= n + 2) {
    const double Sim2 = sm.s[t - 2][lane], Sim1 = sm.s[t - 1][lane], Sip1 = sm.s[t + 1][lane], Sip2 = sm.s[t + 2][lane];
    const bool m2 = sm.wet[t - 2][lane], m1 = sm.wet[t - 1][lane], p1 = sm.wet[t + 1][lane], p2 = sm.wet[t + 2][lane];
    const double dm = sv - Sim1, dp = Sip1 - sv;
    da = slope(Sim2, Sim1, Sip1, Sip2, sm.q[t - 1][lane], s6, sm.q[t + 1][lane], dm, dp, m2, m1 && wet && p1, p2);
    d1m = m1 ? dm : 0.0;
    d1p = p1 ? dp : 0.0;
    if (lim == 3) {
      d1mm = m1 && m2 ? Sim1 - Sim2 : 0.0;
      d1pp = p1 && p2 ? Sip2 - Sip1 : 0.0;
    }
  }
  sm.da[t][lane] = da;
  __syncthreads();
  // limited edge values and curvature of cells 0 .. n+1
  Edges e = {0.0, 0.0, 0.0};
  if (lane_ok && t >= 3 && t <= L - 4 && p >= 0 && p <= n + 1) {
    const double dl = CLAMP && p == 1 ? da : sm.da[t - 1][lane], dr = CLAMP && p == n ? da : sm.da[t + 1][lane];
    const double Sim1 = sv - d1m, Sip1 = sv + d1p;
    e.L = half_exact(Sim1 + sv) + mul_int<false, true>(kSixth, dl - da);
    e.R = half_exact(sv + Sip1) + mul_int<false, true>(kSixth, da - dr);
    limit(lim, sv, da, d1m, d1p, d1mm, d1pp, e.L, e.R);
    e.six = s6 - mul_int<false, true>(3., e.R + e.L);
  }
  sm.l[t][lane] = e.L;
  sm.r[t][lane] = e.R;
  sm.q[t][lane] = e.six;  // the slopes have read 6*S
  __syncthreads();
  // flux through face p (between positions p and p+1), faces 0 .. n
  double f = 0.0;
  if (lane_ok && t >= 3 && t <= L - 5 && p >= 0 && p <= n && wet && sm.wet[t + 1][lane])
    f = face(p, e, Edges{sm.l[t + 1][lane], sm.r[t + 1][lane], sm.q[t + 1][lane]});
  sm.f[t][lane] = f;
  __syncthreads();
  // update of cells 1 .. n
  if (lane_ok && t >= 4 && t <= L - 5 && p >= 1 && p <= n) upd(p, sv, wet, sm.f[t - 1][lane], f);
}

}  // namespace ppm
}  // namespace mom5
