// Tile of the precision form: fluxes and limiters in FP32, tracer state in FP64.
//
// A tile of 28 columns by ZR-4 rows does the z, x and y passes of
// advect_tracer_mdfl_sweby (ocean_tracer_advect.F90:3806-4066) in one go,
// marching down k, its 2-cell halo recomputed instead of exchanged: the z pass
// on the 32 x ZR positions, the x pass on ZR rows of 28 columns, the y pass on
// the interior.  Face terms (mass flux, Courant number, d0, d1, the limiter
// slope) are formed once per level and shared by every tracer.
//
// The increment T_mdfl - T is carried as the sum of the three flux-divergence
// increments; the divergence corrections the reference adds per pass and
// removes at the end cancel exactly and are applied only to the intermediate
// values the next pass limits on.  The state update
// T(taup1) = (rho_dzt(taum1)*T + dtime*th)*rho_dztr (ocean_tracer.F90:2341-2350)
// is evaluated as T + [(rho_dzt(taum1)*rho_dztr - 1)*T + rho_dzt(tau)*rho_dztr*dT]
// with one FP64 add per tracer-cell.  FP64<->FP32 conversions are integer
// operations: on GB300 a conversion issues at the FP64 rate.
//
// What bounds it is the issue of instructions and their latency at 20 to 32 warps
// per SM (DRAM 30% busy), so the tile is laid out for few of them:
//   * two tracers per 64-bit register pair, one packed FP32 instruction for both;
//   * one position per thread, the column's levels carried in registers; level
//     k+3 of each tracer and the next level's fields come by cp.async into the
//     thread's own shared-memory slots, from its own cell or that cell's periodic
//     image, so a position in the halo needs no code of its own and any row length
//     will do (a TMA box wants rows of whole 16 bytes);
//   * a face's cells read from shared memory at offsets chosen once per face from
//     the sign of its flow, instead of selecting among values per tracer;
//   * no branch in the loops over tracers, so their instructions interleave.
// 1440x1080x50 cells, 10 tracers: 7.10 ms; a tile staged by TMA, one tracer at a
// time, took 11.1 (2822 instructions per warp and level against 1364).
#pragma once
#include "mixed_body.cuh"

namespace mom5 {
namespace mixed {

// Two tracers' FP32 values in one 64-bit register pair.  GB300 multiplies or adds
// both in one instruction (mul/add/fma.rn.f32x2), each half rounded on its own.
typedef unsigned long long f2;
DEVI f2 pk(float a, float b) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
DEVI float lo(f2 v) { return __uint_as_float((unsigned)v); }
DEVI float hi(f2 v) { return __uint_as_float((unsigned)(v >> 32)); }
DEVI f2 dup(float a) { return pk(a, a); }
DEVI f2 mul2(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
DEVI f2 fma2(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
DEVI f2 add2(f2 a, f2 b) { return fma2(a, 0x3f8000003f800000ULL, b); }
DEVI f2 sub2(f2 a, f2 b) { return fma2(b, 0xbf800000bf800000ULL, a); }
// The sum of a product m and b.  The assembler contracts mul.rn.f32x2 followed by
// add.rn.f32x2 (or by an fma with the constant factor 1) into one fused
// multiply-add, also under -fmad=false (measured: the fused result's bits).  With
// a factor 1 that it cannot see -- one, from the kernel's arguments -- the sum stays
// a rounding of its own: the product by 1 is exact.
DEVI f2 addm2(f2 m, f2 b, f2 one) { return fma2(m, one, b); }
DEVI f2 sel2(bool p, f2 a, f2 b) { return p ? a : b; }

// The terms of a face that every tracer shares: mass flux, limiter coefficients,
// 1e-30 with the flow's sign, whether the flux is kept (wet face, mass flux not zero)
struct Face {
  float mf, d0, d1, c, tiny;
  bool pos, keep;
  DEVI void close(bool wet) {
    pos = mf > 0.0f;
    tiny = pos ? 1.0e-30f : -1.0e-30f;
    keep = wet && mf != 0.0f;
  }
};
// Flux of a face for two tracers (ocean_tracer_advect.F90:3860-3890), given the
// cells the flow comes from (up), goes to (dn) and the one behind up (w; up itself
// where that one is dry).  Where the reference writes the difference of the two
// cells one way for both flows, differences, divisor and limited step change sign
// together here, which changes no bit of their ratio or of the flux.
DEVI f2 face_flux2(const Face& f, f2 one, f2 w, f2 up, f2 dn) {
  const f2 rj = sub2(dn, up), num = sub2(up, w), den = add2(rj, dup(f.tiny));
  const f2 theta = mul2(num, pk(rcp(lo(den)), rcp(hi(den))));
  const f2 lin = addm2(mul2(dup(f.d1), theta), dup(f.d0), one), ct = mul2(dup(f.c), theta);
  const f2 psi = pk(fmaxf(0.0f, fminf(fminf(1.0f, lo(lin)), lo(ct))), fmaxf(0.0f, fminf(fminf(1.0f, hi(lin)), hi(ct))));
  return sel2(f.keep, mul2(dup(f.mf), addm2(mul2(psi, rj), up, one)), 0ULL);
}

enum { S_RDZ = 0, S_RDZE, S_RDZN, S_UH, S_UHW, S_VH, S_W, S_RDZR, S_RDZM1, S_FIELDS };

// Shared memory of a block: per position, each tracer's next level and the
// level's fields as they arrive (FP64, the thread's own slots), the tracers after
// the z and then the x pass and their y fluxes for the neighbours to read.
template <int NP, int ZR>
struct StreamSmem {
  static constexpr int N = ZR * 32;
  double t[2 * NP][N];
  double f[S_FIELDS][N];
  f2 tzx[NP][N + 96];  // [c + 32]: after z (read by the row's neighbours), then after x (by the rows above and below)
  f2 fy[NP][N + 32];   // [c + 32]: y fluxes
  uint8_t wet[N + 96];
  // the flux through the top face, where the registers of a thread do not hold it too
  static constexpr bool kFtp = ZR >= 24 && NP > 2;
  f2 ftp[kFtp ? NP : 1][kFtp ? N : 1];
};

// One tile (tile_x, tile_y) of the domain, levels k0 .. k1-1, of 2*NP or 2*NP-1 tracers.
template <int NP, int ZR>
DEVI void stream_tile(const MixArgs& a, int n0, int tile_x, int tile_y, int k0, int k1, StreamSmem<NP, ZR>& s) {
  constexpr int TJ = ZR - 4;
  constexpr bool FS = StreamSmem<NP, ZR>::kFtp;
  const Geo& g = a.g;
  const int zi = threadIdx.x & 31, zj = threadIdx.x >> 5, c = threadIdx.x;
  const int i0 = 1 + tile_x * TI, j0 = 1 + tile_y * TJ;
  const float dt = a.dtime;
  const bool odd = a.ntr < 2 * NP;  // the last pair holds one tracer, twice
  const int last = odd ? 2 * NP - 2 : 2 * NP - 1;
  const int pi = i0 - 2 + zi, pj = j0 - 2 + zj;
  int i = pi, j = pj;
  const bool in = image(g, i, j);
  const long o = in ? I2(g, i, j) : 0;
  const bool interior = zj >= 2 && zj <= ZR - 3 && zi >= 2 && zi <= 29 && pi <= g.ni && pj <= g.nj;
  const int nkm1 = g.nk - 1;
  const int fill = in ? 8 : 0;  // positions outside a wall read zeros

  auto fetch_t = [&](int k) {
    const double* T = a.T + ((long)k * g.n2 + o);
#pragma unroll
    for (int n = 0; n < 2 * NP; ++n) {
      if (n < 2 * NP - 1 || !odd) cp_async8(&s.t[n][c], T, fill);
      T += g.n3;
    }
  };
  auto fetch_f = [&](int k) {
    const long p = (long)k * g.n2 + o;
    cp_async8(&s.f[S_RDZ][c], a.rdz + p, fill);
    cp_async8(&s.f[S_RDZE][c], a.rdz + p + (in ? 1 : 0), fill);
    cp_async8(&s.f[S_RDZN][c], a.rdz + p + (in ? g.nxd : 0), fill);
    cp_async8(&s.f[S_UH][c], a.uh + p, fill);
    cp_async8(&s.f[S_UHW][c], a.uh + p - (in ? 1 : 0), fill);
    cp_async8(&s.f[S_VH][c], a.vh + p, fill);
    cp_async8(&s.f[S_W][c], a.w + p + g.n2, fill);
    if (a.fused) {
      cp_async8(&s.f[S_RDZR][c], a.rdzr + p, fill);
      cp_async8(&s.f[S_RDZM1][c], a.rdz_m1 + p, fill);
    }
  };

  // a segment below the surface first forms the flux through its top face: the
  // z pass of the level above, nothing else of it
  const int ks = k0 > 0 ? k0 - 1 : 0;
  const int ksm = ks > 0 ? ks - 1 : 0;
  const int ks1 = ks + 1 < g.nk ? ks + 1 : nkm1, ks2 = ks + 2 < g.nk ? ks + 2 : nkm1;
  fetch_t(ks2);
  fetch_f(ks);
  cp_async_commit();
  // 2-D metrics of this position, once per tile
  float m_dat = 0.f, m_datr = 0.f, m_dyte = 0.f, m_dyte_w = 0.f, m_dxte = 0.f, m_dxtn = 0.f, m_dytn = 0.f;
  if (in) {
    m_dat = d2f(a.dat[o]);
    m_datr = d2f(a.datr[o]);
    m_dyte = d2f(a.dyte[o]);
    m_dyte_w = d2f(a.dyte[o - 1]);
    m_dxte = d2f(a.dxte[o]);
    m_dxtn = d2f(a.dxtn[o]);
    m_dytn = d2f(a.dytn[o]);
  }
  // wet bits of levels k-1, k, k+1, k+2 (level 0 for the one above the surface)
  unsigned mb = (mask_at(g, a.mask2, pi, pj, ksm) ? 1u : 0u) | (mask_at(g, a.mask2, pi, pj, ks) ? 2u : 0u) |
                (mask_at(g, a.mask2, pi, pj, ks1) ? 4u : 0u) | (mask_at(g, a.mask2, pi, pj, ks2) ? 8u : 0u);
  // carried down the column: T(k-1), T(k), T(k+1) and the flux through the top face
  f2 tm[NP], tk[NP], tk1[NP], tk2[NP], ftp[FS ? 1 : NP];
#pragma unroll
  for (int q = 0; q < NP; ++q) {
    float v[2] = {0.f, 0.f}, v1[2] = {0.f, 0.f}, vm[2] = {0.f, 0.f};
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if (in) {
        const int n = 2 * q + h < last ? 2 * q + h : last;
        const double* T = a.T + (long)n * g.n3 + o;
        vm[h] = d2f(T[(long)ksm * g.n2]);
        v[h] = d2f(T[(long)ks * g.n2]);
        v1[h] = d2f(T[(long)ks1 * g.n2]);
      }
    tm[q] = pk(vm[0], vm[1]);
    tk[q] = pk(v[0], v[1]);
    tk1[q] = pk(v1[0], v1[1]);
    if constexpr (FS) s.ftp[q][c] = 0ULL;
    else ftp[q] = 0ULL;
  }
  float wk_prev = 0.f;
  const f2 one = dup(a.one);

  for (int k = ks; k < k1; ++k) {
    const int kp3 = k + 3 < g.nk ? k + 3 : nkm1;
    const bool more = k + 1 < k1;
    const bool m_next = more && mask_at(g, a.mask2, pi, pj, kp3);
    cp_async_wait_all();
    // ---- face terms of this position ----
    const bool wet = in && (mb & 2u);
    const float rdz_c = d2f(s.f[S_RDZ][c]);
    Face fz;
    float zdtr, zwd;
    const float wk = d2f(s.f[S_W][c]);
    z_terms(wk, wk_prev, rdz_c, m_dat, dt, fz.mf, fz.d0, fz.d1, fz.c, zdtr, zwd);
    wk_prev = wk;
    fz.close(wet && (mb & 4u));
    const bool run = k >= k0;  // false: only the z fluxes are wanted
    // ---- z pass of every tracer: the flow through the bottom face comes from
    // level k+1 where it is positive, else from level k ----
    const bool wback = (mb & (fz.pos ? 8u : 1u)) != 0;
    f2 fzx[NP];
#pragma unroll
    for (int q = 0; q < NP; ++q) {
      tk2[q] = pk(d2f(s.t[2 * q][c]), d2f(s.t[2 * q + 1 < 2 * NP - 1 ? 2 * q + 1 : last][c]));
      const f2 up = sel2(fz.pos, tk1[q], tk[q]), dn = sel2(fz.pos, tk[q], tk1[q]);
      const f2 fb = face_flux2(fz, one, sel2(wback, sel2(fz.pos, tk2[q], tm[q]), up), up, dn);
      f2 ft;
      if constexpr (FS) ft = s.ftp[q][c];
      else ft = ftp[q];
      const f2 adiv = mul2(dup(m_datr), sub2(fb, ft));
      fzx[q] = mul2(dup(zdtr), adiv);
      s.tzx[q][c + 32] = addm2(mul2(dup(zdtr), addm2(mul2(tk[q], dup(zwd)), adiv, one)), tk[q], one);
      if constexpr (FS) s.ftp[q][c] = fb;
      else ftp[q] = fb;
    }
    // every lane has read its own slots, and the row's z results are visible to it
    __syncwarp();
    if (more) fetch_t(kp3);
    if (run) {
      const unsigned full = 0xffffffffu;
      const unsigned wt = wet ? 1u : 0u;
      const unsigned wA = __shfl_up_sync(full, wt, 1), wC = __shfl_down_sync(full, wt, 1);
      const unsigned wD = __shfl_down_sync(full, wt, 2);
      Face fx, fyf;
      const float uh_c = d2f(s.f[S_UH][c]);
      h_terms(uh_c, m_dyte, rdz_c, d2f(s.f[S_RDZE][c]), m_dxte, dt, fx.mf, fx.d0, fx.d1, fx.c);
      fx.close(zi >= 1 && zi <= 29 && wet && wC);
      const float xcoef = x_coef(wet, dt, m_datr, rdz_c);
      const float xdiv = x_div(m_dyte, uh_c, m_dyte_w, d2f(s.f[S_UHW][c]));
      h_terms(d2f(s.f[S_VH][c]), m_dxtn, rdz_c, d2f(s.f[S_RDZN][c]), m_dytn, dt, fyf.mf, fyf.d0, fyf.d1, fyf.c);
      float uq = 0.f, ur = 0.f;
      if (a.fused) {
        const double r = s.f[S_RDZR][c];
        uq = d2f(fma(s.f[S_RDZM1][c], r, -1.0));
        ur = wet ? d2f(s.f[S_RDZ][c] * r) : 0.0f;
      } else {
        ur = wet ? rdz_c / dt : 0.0f;
      }
      s.wet[c + 32] = wet;
      __syncwarp();
      if (more) fetch_f(k + 1);
      cp_async_commit();
      // ---- x pass of every tracer: cells zi-1 .. zi+2 around face zi ----
      {
        const int eu = c + 32 + (fx.pos ? 0 : 1), ed = c + 32 + (fx.pos ? 1 : 0);
        const int ew = (fx.pos ? wA : wD) ? c + 32 + (fx.pos ? -1 : 2) : eu;
#pragma unroll
        for (int q = 0; q < NP; ++q) {
          const f2 f = face_flux2(fx, one, s.tzx[q][ew], s.tzx[q][eu], s.tzx[q][ed]);
          const f2 tz = s.tzx[q][c + 32];
          const f2 fw = pk(__shfl_up_sync(full, lo(f), 1), __shfl_up_sync(full, hi(f), 1));
          const f2 fi = mul2(dup(xcoef), sub2(fw, f));
          fzx[q] = addm2(fzx[q], fi, one);
          __syncwarp();  // the row has read its neighbours
          s.tzx[q][c + 32] = add2(tz, addm2(mul2(dup(xcoef), mul2(tk[q], dup(xdiv))), fi, one));
        }
      }
      __syncthreads();
      // the FP64 T(k) of the first outputs
      constexpr int kRing = 2 * NP < 4 ? 2 * NP : 4;
      double t64[kRing];
      const long p = I3(g, pi, pj, k);
#pragma unroll
      for (int q = 0; q < kRing; ++q)
        t64[q] = (a.fused && interior && q <= last) ? a.T[(long)q * g.n3 + p] : 0.0;
      // ---- y fluxes of every tracer (face zj, between rows zj and zj+1) ----
      {
        const bool yface = zj >= 1 && zj <= ZR - 3 && zi >= 2 && zi <= 29;
        fyf.close(yface && wet && s.wet[c + 64]);
        const int eu = c + (fyf.pos ? 32 : 64), ed = c + (fyf.pos ? 64 : 32), eb = c + (fyf.pos ? 0 : 96);
        const int ew = s.wet[eb] ? eb : eu;
#pragma unroll
        for (int q = 0; q < NP; ++q)
          s.fy[q][c + 32] = face_flux2(fyf, one, s.tzx[q][ew], s.tzx[q][eu], s.tzx[q][ed]);
      }
      __syncthreads();
      // ---- outputs of the interior cells ----
      if (interior && (wet || a.fused)) {
        if (a.fused) {
          const int hx = (g.cx && pi == g.ni) ? 0 : (g.cx && pi == 1) ? g.ni + 1 : -1;
          const int hy = (g.cy && pj == g.nj) ? 0 : (g.cy && pj == 1) ? g.nj + 1 : -1;
          const bool edge = hx >= 0 || hy >= 0;
          double* out = a.out + (long)n0 * g.n3;
#pragma unroll
          for (int q = 0; q < NP; ++q) {
            const f2 dT = addm2(mul2(dup(xcoef), sub2(s.fy[q][c], s.fy[q][c + 32])), fzx[q], one);
            const f2 inc = addm2(mul2(dup(uq), tk[q]), mul2(dup(ur), dT), one);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int n = 2 * q + h;
              if (n == 2 * NP - 1 && odd) break;
              const double tn = t64[n % kRing] + f2d(h ? hi(inc) : lo(inc));
              out[p] = tn;
              if (edge) {  // halo update of T(taup1) in cyclic directions (ocean_model.F90:1903-1911)
                if (hx >= 0) out[I3(g, hx, pj, k)] = tn;
                if (hy >= 0) out[I3(g, pi, hy, k)] = tn;
                if (hx >= 0 && hy >= 0) out[I3(g, hx, hy, k)] = tn;
              }
              if (n + kRing < 2 * NP) {
                if (n + kRing < 2 * NP - 1 || !odd) t64[n % kRing] = a.T[(long)(n + kRing) * g.n3 + p];
              }
              out += g.n3;
            }
          }
        } else {
#pragma unroll
          for (int q = 0; q < NP; ++q) {
            const f2 dT = addm2(mul2(dup(xcoef), sub2(s.fy[q][c], s.fy[q][c + 32])), fzx[q], one);
            const f2 inc = mul2(dup(ur), dT);
            double* out = a.out + (long)(2 * q) * g.n3;
            out[p] = out[p] + f2d(lo(inc));
            if (2 * q + 1 < 2 * NP - 1 || !odd) out[p + g.n3] = out[p + g.n3] + f2d(hi(inc));
          }
        }
      }
    } else {
      if (more) fetch_f(k + 1);  // the z terms have read this thread's slots before the barrier above
      cp_async_commit();
    }
#pragma unroll
    for (int q = 0; q < NP; ++q) {
      tm[q] = tk[q];
      tk[q] = tk1[q];
      tk1[q] = tk2[q];
    }
    mb = (mb >> 1) | (m_next ? 8u : 0u);
  }
  cp_async_wait_all();
  __syncthreads();
}

}  // namespace mixed
}  // namespace mom5
