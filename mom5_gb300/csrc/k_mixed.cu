// Precision form: the barotropic subcycle kernels, and the arguments and launches
// of the advection (mixed_stream.cuh, k_mixed_stream.cu).
#include "internal.h"
#include "bt_fast_body.cuh"

namespace mom5 {

__global__ void __launch_bounds__(128) k_btf_prep(BtArgs a) { btfast::prep_body(a, blockIdx.x); }
// The subcycle kernels are launched as programmatic dependents (launch_pdl).
__global__ void __launch_bounds__(128) k_btf_pred(BtArgs a, int so, int sn, int reuse) {
  pdl_wait();
  pdl_trigger();
  btfast::pred_body(a, so, sn, reuse, blockIdx.x);
}
template <bool EARLY>
__global__ void __launch_bounds__(128) k_btf_mom(BtArgs a, int so, int sn, double wgt) {
  btfast::mom_body<EARLY>(a, so, sn, wgt, blockIdx.x);
}
__global__ void __launch_bounds__(128) k_btf_corr(BtArgs a, int so, int sn) {
  pdl_wait();
  pdl_trigger();
  btfast::corr_body(a, so, sn, blockIdx.x);
}
template <bool EARLY>
__global__ void __launch_bounds__(128) k_btf_corr_pred(BtArgs a, int so, int sn) {
  btfast::corr_pred_body<EARLY>(a, so, sn, blockIdx.x);
}

void launch_btf_prep(const BtArgs& a, cudaStream_t s) {
  k_btf_prep<<<bt_grid(a.g, 128), 128, 0, s>>>(a);
}

// One launch per subcycle (mom5gpu_set_barotropic_fusion mode 1): 32 x 8 tiles of
// 352 threads, one point per thread in each phase (the 34 x 10 surface-pressure
// ring is the largest).  Measured per precision-form step: 0.66 ms against 0.72
// ms for form 0 on 360x300 (80 subcycles), where the launches set the time, but
// 7.2 ms against 4.6 ms on 1440x1080 (60 subcycles), which form 0's streaming
// launches keep near the memory bound.  On 360x300 the 64 x 8 (256 threads,
// several points per thread), 32 x 16, 128 x 4 and 64 x 16 tiles were slower
// than 32 x 8.
constexpr int kBtfTX = 32, kBtfTY = 8, kBtfThreads = 352;
__global__ void __launch_bounds__(kBtfThreads) k_btf_fused(BtArgs a, int so, int sn, int reuse, double wgt) {
  pdl_wait();
  pdl_trigger();
  btfast::fused_body<kBtfTX, kBtfTY>(a, so, sn, reuse, wgt, blockIdx.x, blockIdx.y);
}

// Subcycle itime of nts.  Form 0: the predictor (a launch of its own only in the
// first subcycle), the momentum step, and the corrector, which in every
// subcycle but the last also forms the next subcycle's predictor; 1 + 2*nts
// launches per step.  Form 1: one launch per subcycle.  Returns the launches.
BtResident btf_resident() {
  auto pair = [](auto* mom, auto* corr) { return bt_resident_columns((const void*)mom, (const void*)corr, 128); };
  return {pair(k_btf_mom<true>, k_btf_corr_pred<true>), pair(k_btf_mom<false>, k_btf_corr_pred<false>)};
}

int launch_btf_subcycle(const BtArgs& a, int itime, int nts, bool fused, cudaStream_t s) {
  const int so = itime % 2, sn = (itime + 1) % 2;
  const double wgt = (double)(nts - itime + 1);
  if (fused) {
    dim3 gf((a.g.ni + 2 + kBtfTX - 1) / kBtfTX, (a.g.nj + 2 + kBtfTY - 1) / kBtfTY);
    launch_pdl(k_btf_fused, gf, dim3(kBtfThreads), s, a, so, sn, (int)(itime > 1), wgt);
    return 1;
  }
  const dim3 b(btf_threads(a.g)), g2 = bt_grid(a.g, b.x);
  const bool early = a.early;
  if (itime == 1) launch_pdl(k_btf_pred, g2, b, s, a, so, sn, 0);
  launch_pdl(early ? k_btf_mom<true> : k_btf_mom<false>, g2, b, s, a, so, sn, wgt);
  if (itime < nts) launch_pdl(early ? k_btf_corr_pred<true> : k_btf_corr_pred<false>, g2, b, s, a, so, sn);
  else launch_pdl(k_btf_corr, g2, b, s, a, so, sn);
  return itime == 1 ? 3 : 2;
}

int make_mix_args(mom5gpu_domain* d, int taum1, int tau, int taup1, double dtime, MixArgs* ap) {
  MixArgs& a = *ap;
  a.g = d->geo;
  a.ntr = d->dims.num_prog_tracers;
  a.dtime = (float)dtime;
  a.mask2 = d->mask2;
  a.dat = fptr(d, MOM5GPU_DAT, 0, 0);
  a.datr = fptr(d, MOM5GPU_DATR, 0, 0);
  a.dxte = fptr(d, MOM5GPU_DXTE, 0, 0);
  a.dyte = fptr(d, MOM5GPU_DYTE, 0, 0);
  a.dxtn = fptr(d, MOM5GPU_DXTN, 0, 0);
  a.dytn = fptr(d, MOM5GPU_DYTN, 0, 0);
  a.uh = fptr(d, MOM5GPU_UHRHO_ET, 0, 0);
  a.vh = fptr(d, MOM5GPU_VHRHO_NT, 0, 0);
  a.w = fptr(d, MOM5GPU_WRHO_BT, 0, 0);
  a.rdz = fptr(d, MOM5GPU_RHO_DZT, 0, tau);
  a.rdz_m1 = fptr(d, MOM5GPU_RHO_DZT, 0, taum1);
  a.rdzr = fptr(d, MOM5GPU_RHO_DZTR, 0, 0);
  a.fused = 1;
  a.T = a.ntr > 0 ? fptr(d, MOM5GPU_TRACER, 1, taum1) : nullptr;
  a.out = a.ntr > 0 ? fptr(d, MOM5GPU_TRACER, 1, taup1) : nullptr;
  if (!a.dat || !a.datr || !a.dxte || !a.dyte || !a.dxtn || !a.dytn || !a.uh || !a.vh || !a.w || !a.rdz || !a.rdz_m1 ||
      !a.rdzr || !d->mask2 || !a.T || !a.out)
    return fail(d, MOM5GPU_ESTATE, "precision form: a required field was never set");
  return MOM5GPU_OK;
}

int launch_mdfl_mixed(mom5gpu_domain* d, int n_first, int ntr, int taum1, int tau, int taup1, double dtime,
                      bool fused_update) {
  ClockScope clk(d, SEC_MDFL_MIXED);
  const Geo& g = d->geo;
  MixArgs a;
  a.g = g;
  a.dtime = (float)dtime;
  a.mask2 = d->mask2;
  a.dat = fptr(d, MOM5GPU_DAT, 0, 0);
  a.datr = fptr(d, MOM5GPU_DATR, 0, 0);
  a.dxte = fptr(d, MOM5GPU_DXTE, 0, 0);
  a.dyte = fptr(d, MOM5GPU_DYTE, 0, 0);
  a.dxtn = fptr(d, MOM5GPU_DXTN, 0, 0);
  a.dytn = fptr(d, MOM5GPU_DYTN, 0, 0);
  a.uh = fptr(d, MOM5GPU_UHRHO_ET, 0, 0);
  a.vh = fptr(d, MOM5GPU_VHRHO_NT, 0, 0);
  a.w = fptr(d, MOM5GPU_WRHO_BT, 0, 0);
  a.rdz = fptr(d, MOM5GPU_RHO_DZT, 0, tau);
  a.rdz_m1 = fptr(d, MOM5GPU_RHO_DZT, 0, taum1);
  a.rdzr = fptr(d, MOM5GPU_RHO_DZTR, 0, 0);
  a.fused = fused_update ? 1 : 0;
  if (!a.dat || !a.datr || !a.dxte || !a.dyte || !a.dxtn || !a.dytn || !a.uh || !a.vh || !a.w || !a.rdz || !a.rdz_m1 ||
      !a.rdzr || !d->mask2)
    return fail(d, MOM5GPU_ESTATE, "precision form: a required field was never set");
  int rc = MOM5GPU_OK;
  for (int c0 = 0; c0 < ntr && rc == MOM5GPU_OK; c0 += 10) {
    int cn = ntr - c0 < 10 ? ntr - c0 : 10;
    a.ntr = cn;
    a.T = fptr(d, MOM5GPU_TRACER, n_first + c0, taum1);
    if (fused_update) {
      a.out = fptr(d, MOM5GPU_TRACER, 1, taup1);  // indexed with the absolute tracer number
    } else {
      a.out = fptr(d, MOM5GPU_TH_TENDENCY, n_first + c0, 0);
    }
    if (!a.T || !a.out) return fail(d, MOM5GPU_ENOMEM, "precision form: tracer storage");
    rc = launch_mixed_stream(d, a, fused_update ? n_first - 1 + c0 : 0);
  }
  if (rc) return rc;
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? MOM5GPU_OK : cuda_fail(d, e, "precision form launch");
}

}  // namespace mom5
