// Precision-form barotropic subcycles over a batch's work list.
#include "internal.h"
#include "bt_fast_body.cuh"

namespace mom5 {

namespace {

DEVI int find_entry_m(const int* prefix, int count, int b) {
  int lo = 0, hi = count;
  while (hi - lo > 1) {
    int mid = (lo + hi) >> 1;
    if (prefix[mid] <= b) lo = mid;
    else hi = mid;
  }
  return lo;
}

// precision-form barotropic subcycle over a work list of (domain, 2-D block) items
#define BTF_ENTRY                                    \
  int e = find_entry_m(w.pb2, w.count, blockIdx.x);  \
  const BtArgs& a = d[w.entries[e]];                 \
  const int bx = blockIdx.x - w.pb2[e];

__global__ void __launch_bounds__(128) kb_btf_prep(const BtArgs* d, BatchWork w) {
  BTF_ENTRY
  btfast::prep_body(a, bx);
}
__global__ void __launch_bounds__(128) kb_btf_pred(const BtArgs* d, BatchWork w, int so, int sn, int reuse) {
  pdl_wait();
  pdl_trigger();
  BTF_ENTRY
  btfast::pred_body(a, so, sn, reuse, bx);
}
template <bool EARLY>
__global__ void __launch_bounds__(128) kb_btf_mom(const BtArgs* d, BatchWork w, int so, int sn, double wgt) {
  BTF_ENTRY
  btfast::mom_body<EARLY>(a, so, sn, wgt, bx);
}
__global__ void __launch_bounds__(128) kb_btf_corr(const BtArgs* d, BatchWork w, int so, int sn) {
  pdl_wait();
  pdl_trigger();
  BTF_ENTRY
  btfast::corr_body(a, so, sn, bx);
}
template <bool EARLY>
__global__ void __launch_bounds__(128) kb_btf_corr_pred(const BtArgs* d, BatchWork w, int so, int sn) {
  BTF_ENTRY
  btfast::corr_pred_body<EARLY>(a, so, sn, bx);
}

}  // namespace

void launch_batch_btf_prep(const BtArgs* bt, const BatchWork& w, cudaStream_t s) {
  if (w.tb2 > 0) kb_btf_prep<<<w.tb2, 128, 0, s>>>(bt, w);
}

// subcycle itime of nts, as the one-domain form 0: the predictor launched only in
// the first subcycle, the corrector forming the next subcycle's predictor in all
// but the last; returns the launches
BtResident batch_btf_resident() {
  auto pair = [](auto* mom, auto* corr) { return bt_resident_columns((const void*)mom, (const void*)corr, 128); };
  return {pair(kb_btf_mom<true>, kb_btf_corr_pred<true>), pair(kb_btf_mom<false>, kb_btf_corr_pred<false>)};
}

int launch_batch_btf_subcycle(const BtArgs* bt, const BatchWork& w, int itime, int nts, cudaStream_t s) {
  if (w.tb2 <= 0) return 0;
  const int so = itime % 2, sn = (itime + 1) % 2;
  const double wgt = (double)(nts - itime + 1);
  const dim3 g2(w.tb2), b(128);
  const bool early = w.early;
  if (itime == 1) launch_pdl(kb_btf_pred, g2, b, s, bt, w, so, sn, 0);
  launch_pdl(early ? kb_btf_mom<true> : kb_btf_mom<false>, g2, b, s, bt, w, so, sn, wgt);
  if (itime < nts) launch_pdl(early ? kb_btf_corr_pred<true> : kb_btf_corr_pred<false>, g2, b, s, bt, w, so, sn);
  else launch_pdl(kb_btf_corr, g2, b, s, bt, w, so, sn);
  return itime == 1 ? 3 : 2;
}

}  // namespace mom5
