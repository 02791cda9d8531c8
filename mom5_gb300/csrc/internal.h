// Internal declarations shared by the C-ABI layer and the kernel files.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <string>
#include <vector>

#include "../../include/mom5gpu.h"

namespace mom5 {

// Geometry passed by value to every kernel.
struct Geo {
  int ni, nj, nk;   // compute domain
  int nxd, nyd;     // data domain (halo 1)
  int cx, cy;       // cyclic flags
  long n2;          // nxd*nyd
  long n3;          // n2*nk
};

// Field shape classes.
enum Shape { S2D = 0, S3D = 1, S3DW = 2 };

struct FieldInfo {
  int id;
  Shape shape;
  bool per_tracer;
  bool per_level;
};

const FieldInfo* field_info(int id);

// Per-tracer scheme selection (field_table).
struct TracerScheme {
  int horz = MOM5GPU_ADVECT_MDFL_SWEBY;
  int vert = MOM5GPU_ADVECT_MDFL_SWEBY;
  double min_limit = -1.0e10;
  double max_limit = 1.0e10;
  int ppm_limiter = 2;  // ppm_hlimiter (ocean_tpm_util.F90:87): 1 cw84, 2 ifc, 3 sh
  int psom_limit = 0;   // psom_limit (ocean_tpm_util.F90:86)
};

// Quicker weights on the device (quicker_init, ocean_tracer_advect.F90:1442-1586).
struct QuickerWeights {
  double* quick_x = nullptr;  // 2 * n2
  double* quick_y = nullptr;  // 2 * n2
  double* curv_xp = nullptr;  // 3 * n2
  double* curv_xn = nullptr;
  double* curv_yp = nullptr;
  double* curv_yn = nullptr;
  double* quick_z = nullptr;  // 2 * nk
  double* curv_zp = nullptr;  // 3 * nk
  double* curv_zn = nullptr;
};

}  // namespace mom5

struct mom5gpu_domain {
  mom5gpu_dims dims;
  mom5gpu_options opt;
  mom5::Geo geo;
  cudaStream_t own_stream = nullptr;
  cudaStream_t stream = nullptr;
  std::string err;
  size_t bytes = 0;
  // one allocation per field id; nullptr until first set/used
  std::vector<double*> field;  // indexed by field id
  std::vector<mom5::TracerScheme> scheme;
  std::vector<std::string> tracer_name, tracer_file;  // T_prog(n)%name, %restart_file
  // host copies needed at init time
  std::vector<double> dzt_h, zw_h;
  std::vector<int> kmt_h;
  // derived device data
  uint8_t* mask2 = nullptr;  // tmask with a 2-cell halo (tmask_mdfl / tmask_quick), (ni+4)(nj+4)nk
  mom5::QuickerWeights qw;
  double* cori1 = nullptr;
  double* cori2 = nullptr;
  bool advect_ready = false;
  bool baro_ready = false;
  int nts = 0;
  double dtuv = 0.0, dtbt = 0.0;
  // scratch
  double* mdfl_a = nullptr;  // tracer_mdfl after the z pass, ntr * n3
  double* mdfl_b = nullptr;  // after the x pass, ntr * n3
  size_t mdfl_cap = 0;       // tracers that fit
  float* mixed_scr = nullptr;  // precision-form scratch
  size_t mixed_cap = 0;
  double* bt = nullptr;        // barotropic scratch
  int* kmt_d = nullptr;        // device copy of kmt (uploaded on first use)
  double* psom_scr = nullptr;  // PSOM mass and x/y/z face fluxes, 4 x n3; cells beside the segments
  long itt0 = 0;               // Time%itt0 (orders the PSOM sweeps)
  double* red = nullptr;       // reduction scratch (device)
  double* red_h = nullptr;     // pinned host result
  int* flag = nullptr;         // device flag word
  // profiling
  bool timing = false;
  struct Clock {
    int section;
    cudaEvent_t a, b;
  };
  std::vector<Clock> clocks;           // recorded, not yet resolved
  std::vector<cudaEvent_t> event_pool;
  double clock_ms[8] = {0};
  long clock_calls[8] = {0};
  long launches = 0;
  // autotuned launch shapes (0 = built-in heuristic)
  int tune_mixed_rows = 32;  // precision-form tile height incl. halo: 16 or 24, else by the number of tracers
  int tune_mixed_pf = 0;     // precision form: accepted and reported, every value runs the one staging there is
  int* wait_err = nullptr;   // set when a bounded device wait gave up: bit 1 a grid barrier
  unsigned* bt_sync = nullptr;  // arrival counter of the cooperative barotropic subcycle's grid barriers
  int tune_y_tj = 0;         // FP64 y-pass rows per thread
  bool bt_early = true;      // the barotropic subcycles load early (BtResident), set by barotropic_init
  int bt_fused = 0;          // exact B-grid subcycles: 0 two launches each, 1 one launch each,
                             // 2 all in one cooperative launch
  int coop_blocks = 0;       // resident blocks per SM of the cooperative subcycle kernel (0: not queried, -1: none)
  int coop_sms = 0;          // SMs of the device
  // CUDA graphs of the barotropic subcycle loop, one per set of kernel arguments
  // (the bytes of the BtArgs it was captured with: time levels rotate), at most
  // kBtGraphs, the oldest replaced first
  struct BtGraph {
    cudaGraphExec_t exec = nullptr;
    std::vector<unsigned char> key;
  };
  std::vector<BtGraph> bt_graphs;
  // domain decomposition (decomp.cu): sides facing a neighbouring subdomain
  // (bits 1 west, 2 east, 4 south, 8 north) and the MDFL halo strips
  int nbr = 0;
  double* hz = nullptr;  // tracer_mdfl after z, columns -1, 0, ni+1, ni+2: ntr*nk*nj*4
  double* hx = nullptr;  // after x, rows -1, 0, nj+1, nj+2: ntr*nk*4*ni
};

namespace mom5 {

// error helpers (capi.cu)
int fail(mom5gpu_domain* d, int code, const char* fmt, ...);
int cuda_fail(mom5gpu_domain* d, cudaError_t e, const char* where);
double* fptr(mom5gpu_domain* d, int id, int n, int level);  // nullptr if absent
double* fptr_if_set(mom5gpu_domain* d, int id, int n, int level);  // nullptr if never allocated
size_t field_count(const Geo& g, Shape s);

// profiling sections
enum Section { SEC_MDFL = 0, SEC_MDFL_MIXED, SEC_UPDATE, SEC_BAROTROPIC, SEC_UPWIND, SEC_QUICKER, SEC_BATCH, SEC_N };
// RAII: events around a section when timing is on
struct ClockScope {
  mom5gpu_domain* d;
  int sec;
  cudaEvent_t a = nullptr;
  ClockScope(mom5gpu_domain* d_, int s);
  ~ClockScope();
};
inline void count_launches(mom5gpu_domain* d, long n) { d->launches += n; }

// Arguments of the FP64 MDFL passes (k_fp64.cu).
struct MdflArgs {
  Geo g;
  int ntr;
  double dtime;
  const uint8_t* mask2;  // tmask_mdfl
  const double *dat, *datr, *dxte, *dyte, *dxtn, *dytn;
  const double *uh, *vh, *w;  // uhrho_et, vhrho_nt, wrho_bt (0:nk)
  const double* rdz;          // rho_dzt(tau)
  const double* T;            // tracer 0 at taum1; tracer n at T + n*tstride
  long tstride;
  double* tz;                 // after z, tracer n at tz + n*g.n3
  double* tx;                 // after x
  double* th;                 // th_tendency of tracer 0, tracer n at th + n*g.n3
  int tj = 0;                 // y-pass rows per thread (0 = choose from the domain size)
  int th_fresh = 0;           // th is +0 at every compute cell: the y pass writes out + 0.0 instead of th + out
  // the whole step (th_fresh): the y pass also zeroes th's halo ring and writes the
  // explicit update with its periodic images; nullptr Tp1: th_tendency only
  const double *rdz_m1 = nullptr, *rdzr = nullptr;  // rho_dzt(taum1), rho_dztr
  double* Tp1 = nullptr;                            // tracer 0 at taup1, tracer n at + n*tstride
  // decomposed domains: sides whose halo comes from a neighbouring subdomain
  // (bits 1 west, 2 east, 4 south, 8 north) and the strips its exchange filled:
  // tracer_mdfl after the z pass at i = -1, 0, ni+1, ni+2 (hz[((n*nk + k)*nj + j-1)*4 + slot])
  // and after the x pass at j = -1, 0, nj+1, nj+2 (hx[((n*nk + k)*4 + slot)*ni + i-1])
  int nbr = 0;
  const double* hz = nullptr;
  const double* hx = nullptr;
};


// Arguments of the barotropic kernels (fp64_bodies.cuh) for one domain and one
// (tau, taup1) pair, and the step's other inputs and outputs.
// Largest number of tracers the FP64 MDFL kernels advect per launch set.
constexpr int kMdflChunk = 10;

struct BtArgs {
  Geo g;
  int cgrid, nts, stepB;
  int early;  // one-domain subcycles load early (BtResident)
  double dtbt, dtbt_gamma_rho0r, dtbt_rho0r, gamma;
  const double *tmask1, *umask1, *f, *dxu, *dyu, *dxur, *dyur, *dat, *datr, *dxter, *dytnr, *tmen_e, *tmen_n;
  const double *dte, *dtw, *dus, *dun, *daur;
  const double *patm, *thicku, *thicken_e, *thicken_n, *forcing_u, *forcing_v, *rho_g, *cori1, *cori2;
  double* eta_bt;  // 2 levels
  double* ubt;     // 2 levels
  double* vbt;     // 2 levels
  double* steady;
  double* ps;
  double* cf;  // coriolis_force_bt, 6 planes (component-major within AB level)
  double* ca;  // coriolis_accel_bt, 2 planes
  double *eta_bar, *udrho_u, *udrho_v;  // taup1 accumulators
  double *uhb, *vhb;  // B grid: ubt*dyu and vbt*dxu, 2 levels like ubt (reuse the C-grid Coriolis planes)
  double* btf;        // precision form, B grid: folded step coefficients (bt_fast_body.cuh), else nullptr
  double* dvs;        // divergence of the corrector's transports, reused by the next subcycle's predictor
};
// planes of barotropic scratch: 18 for the exact path (the reused divergence in
// two planes for the one-launch subcycle), 9 more for the precision form
constexpr int kBtPlanes = 18, kBtFastPlanes = 10;
struct BtExtra {
  const double *eta_bar_tau, *eta_tau, *ud_tau, *vd_tau, *pme, *river, *source, *eta_smooth;
  double *conv, *eta_u, *ps_out, *gxo, *gyo;
  int initsum_with_bar;
};

// Arguments of the precision-form kernel (mixed_body.cuh).
struct MixArgs {
  Geo g;
  int ntr;
  float dtime;
  const uint8_t* mask2;
  const double *dat, *datr, *dxte, *dyte, *dxtn, *dytn, *uh, *vh, *w;
  const double *rdz, *rdz_m1, *rdzr;  // rho_dzt(tau), rho_dzt(taum1), rho_dztr
  const double* T;                    // tracer 0 at taum1 (tracer n at + n*g.n3)
  double* out;                        // fused: T(taup1); else th_tendency (tracer n at + n*g.n3)
  int fused;
  float one = 1.0f;                   // a factor that the compiler cannot see to be 1 (mixed_stream.cuh)
};

// Arguments of the FP64 explicit update.
struct UpdArgs {
  Geo g;
  int ntr;
  long tstride;
  const double *rdz_m1, *rdzr, *Tm1, *th;
  double* Tp1;
  double dtime;
};

// argument builders (k_fp64.cu, k_mixed.cu); status codes as the C ABI
int make_mdfl_args(mom5gpu_domain* d, int n_first, int ntr, int taum1, int tau, double dtime, MdflArgs* a);
int make_upd_args(mom5gpu_domain* d, int taum1, int taup1, double dtime, UpdArgs* u);
int make_bt_args(mom5gpu_domain* d, int tau, int taup1, BtArgs* a, BtExtra* x);
int make_mix_args(mom5gpu_domain* d, int taum1, int tau, int taup1, double dtime, MixArgs* a);

// ---- FP64 kernels (k_fp64.cu) ----
// the three MDFL passes on the stream, for the tracers described by a
// (at most 8 per call); scratch a.tz/a.tx and a.mask2 are the caller's.
void run_mdfl_kernels(const MdflArgs& a, bool all, bool sweby, cudaStream_t s);
void run_mdfl_pass(const MdflArgs& a, bool all, bool sweby, int pass, cudaStream_t s);
int launch_barotropic_phase(mom5gpu_domain* d, int tau, int taup1, int phase, int itime);
void launch_halo_fill(const Geo& g, double* a, int nlev, int flags, cudaStream_t s);
void launch_zero_ring(const Geo& g, double* a, long nlev, cudaStream_t s);
int launch_mdfl(mom5gpu_domain* d, bool all, int n_first, int ntr, int taum1, int tau, double dtime,
                double sweby_limiter);
// the whole step of every tracer: th_tendency = its advection, T(taup1) by the explicit update
int launch_mdfl_step(mom5gpu_domain* d, bool all, int taum1, int tau, int taup1, double dtime);
constexpr int kSms = 152;  // SMs of the GB300, by which the launch rules share work
int y_strip_rows(long cols, long nj);
int add_step_args(mom5gpu_domain* d, int n_first, int taum1, int taup1, MdflArgs* a);
int launch_upwind_horz(mom5gpu_domain* d, int n, int taum1);
int launch_upwind_vert(mom5gpu_domain* d, int n, int taum1);
int launch_quicker_horz(mom5gpu_domain* d, int n, int taum1, int tau);
int launch_quicker_vert(mom5gpu_domain* d, int n, int taum1, int tau);
int launch_update_tracer(mom5gpu_domain* d, int n_first, int ntr, int taum1, int taup1, double dtime);
int launch_tmask_limit(mom5gpu_domain* d, int n, int tau);
int launch_tmask_limit_ts_same(mom5gpu_domain* d, int nt, int ns);
int launch_eta_tendency(mom5gpu_domain* d, int tau);
int launch_eta_update(mom5gpu_domain* d, int taum1, int taup1, double dtime);
// Programmatic dependent launch of the barotropic subcycle kernels.  A kernel
// launched by launch_pdl may be scheduled while the kernel before it in the
// stream runs its last blocks; its blocks first wait in pdl_wait()
// (griddepcontrol.wait) until that kernel has completed and its writes are
// visible, then allow the next kernel to be scheduled (pdl_trigger), so every
// kernel still reads only completed results.  Launched the ordinary way, the
// two instructions do nothing.
#ifdef __CUDACC__
// The data-domain point of this thread in a 2-D barotropic launch, its rows laid end
// to end: with blocks of one row each the last of a row is part empty, and the SMs
// that get more of the full ones set the time (270x200 columns, 80 subcycles: 1.18 ->
// 0.81 ms; 300x260: 1.40 -> 0.99).
__device__ __forceinline__ bool bt_point(const Geo& g, int block, int& i, int& j) {
  const unsigned q = (unsigned)block * blockDim.x + threadIdx.x;
  if (q >= (unsigned)g.n2) return false;
  j = (int)(q / (unsigned)g.nxd);
  i = (int)(q - (unsigned)j * (unsigned)g.nxd);
  return true;
}
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// The start of a subcycle kernel; with EARLY it stands between the loads of what the
// launch before does not write and the rest, so that their latency overlaps the end
// of that launch.  Such a load may read what the launch before that one wrote, with no
// wait of its own.  Two things make it see those writes:
//   * pdl_trigger comes after pdl_wait everywhere, so the launch before allowed this
//     one only when each of its blocks had waited for the launch before it, that is for
//     its completion and for its writes to be performed and visible;
//   * the load goes to L2, where those writes are (load_early): a line that this SM's L1
//     kept from an earlier subcycle cannot answer it, whatever the launch of a
//     dependent does with that cache.  The manual promises visibility to a launch that
//     has waited; it says nothing of one that has not.
__device__ __forceinline__ void bt_after_previous() {
  pdl_wait();
  pdl_trigger();
}
template <bool EARLY, class T>
__device__ __forceinline__ T load_early(const T* p) {
  return EARLY ? __ldcg(p) : *p;
}
// A value loaded where it is declared (EARLY) or, to hold no register until then,
// where it is used.
template <bool EARLY, class T>
struct Loaded {
  const T* p;
  T v;
  __device__ __forceinline__ explicit Loaded(const T* q) : p(q) {
    if (EARLY) v = load_early<EARLY>(q);
  }
  __device__ __forceinline__ operator T() const { return EARLY ? v : *p; }
};
#endif
template <typename... P, typename... A>
cudaError_t launch_pdl(void (*k)(P...), dim3 grid, dim3 block, cudaStream_t s, A... args) {
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = 0;
  cfg.stream = s;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k, args...);
}

// Whether a launch over so many columns takes the subcycle's products on the integer
// pipe (bt_mul).  Small launches are chains of latency, which its longer sequence
// adds to; larger ones are bound by the FP64 pipe.  On the FP64 and on the integer pipe,
// 60 subcycles, us a step: B grid 394 and 406 at 28566 columns, 490 and 438 at 34748;
// batches 349 and 360 at 12928, 424 and 412 at 21376, 440 and 430 at 38144; C grid
// 494 and 552 at 52750, 588 and 567 at 58968, 684 and 644 at 71052.
inline bool bt_int_products(bool cgrid, long columns) { return columns >= (cgrid ? 60000 : 30000); }
// Columns over which both a running launch of kernel a and a waiting one of kernel b, in
// blocks of so many threads, are resident.
long bt_resident_columns(const void* a, const void* b, int threads);
// Whether the subcycle kernels load early (bt_after_previous).  A launch's blocks come
// to the SMs as soon as the one before has started all of its own, and wait there.
// Where both launches fit the SMs together, the start of each is hidden behind the end
// of the other and early loads win.  They take registers, so this holds up to fewer
// columns for the kernels that load early (`early`) than for those that load late
// (`late`); between the two late loads win.  Past both, the waiting blocks come as the
// running ones end in either form, and early loads win again.
// 60 subcycles, us a step, early and late.  B grid, blocks of 64 (48 + 64 and 40 + 40
// registers, 9 and 12 pairs of blocks an SM): 659 and 739 at 86955 columns, 1021 and 764
// at 91134, 1024 and 843 at 111360, 1036 and 1386 at 119110, 1382 and 1465 at 226524.
// Precision form, blocks of 128 (40 + 40 and 32 + 32: 6 and 8 pairs): 455 and 495 at
// 111360, 675 and 533 at 119110, 686 and 595 at 151140, 696 and 933 at 166600, 874 and
// 972 at 286812.  The C grid's kernels lose at most 3% by early loads (785 and 769 at 95914
// columns, 834 and 808 at 111360, 882 and 911 at 127167, 904 and 1514 at 137200) and
// always load early, and so do the exact form's batches, whose two forms fit up to the
// same 4 pairs of blocks of 128 (600 and 668 at 67584 columns, 952 and 1102 at 88192,
// 2038 and 2213 at 323968).
struct BtResident {
  long early = 0, late = 0;
  bool loads_early(long columns) const { return columns <= early || columns > late; }
};
BtResident bt_resident();           // B grid, exact form (k_fp64.cu)
BtResident btf_resident();          // B grid, precision form (k_mixed.cu)
BtResident batch_btf_resident();    // batches, precision form (k_batch.cu)
// the instantiation <INT, EARLY> of an exact B-grid subcycle kernel; FP64 products only on few
// columns, where the loads are early
#define BT_VARIANT(K, columns, early) \
  (!bt_int_products(false, columns) ? K<false, true> : (early) ? K<true, true> : K<true, false>)
// Threads per block of a one-domain 2-D launch.  Exact form: 64 (60 subcycles against
// blocks of 128: 513 and 567 us a step at 52750 columns, 1132 and 1143 at 166600, 5056 and 5119 at 1003230).
// Precision form, whose kernels are half as long: 128 from 30000 columns on (338 us against
// 409 with 64 at 52750, 446 against 585 at 102960), 64 below (307 and 313 at 22444).
constexpr int kBtThreads = 64;
inline int btf_threads(const Geo& g) { return g.n2 < 30000 ? 64 : 128; }
inline dim3 bt_grid(const Geo& g, int threads) { return dim3((unsigned)((g.n2 + threads - 1) / threads)); }
// precision-form barotropic subcycle (k_mixed.cu, k_batch.cu)
void launch_btf_prep(const BtArgs& a, cudaStream_t s);
int launch_btf_subcycle(const BtArgs& a, int itime, int nts, bool fused, cudaStream_t s);
int launch_centred(mom5gpu_domain* d, int n, int tau, int order, bool horz);
int ensure_kmt_device(mom5gpu_domain* d);
int launch_mdfl_sup_b(mom5gpu_domain* d, int n, int taum1, int tau, double dtime);
int launch_mdppm(mom5gpu_domain* d, int n, int taum1, int tau, double dtime);
int launch_psom(mom5gpu_domain* d, int n, int taum1, double dtime);
int launch_quickmom3_horz(mom5gpu_domain* d, int n, int taum1, int tau);
int launch_tracer_boundary(mom5gpu_domain* d, int n);
int launch_barotropic_forcing(mom5gpu_domain* d, int tau);  // tau 0: no friction
int launch_update_ucell_thickness(mom5gpu_domain* d, int taup1, int vcoord, bool linear_fs, bool dzwu_k0);
int launch_advection_velocity(mom5gpu_domain* d, int tau);
int launch_barotropic(mom5gpu_domain* d, int tau, int taup1);
int grid_barrier_selftest(mom5gpu_domain* d, int rounds, int unreachable);
int launch_content(mom5gpu_domain* d, int n, int level, double* out_host);
int launch_content_fixed(mom5gpu_domain* d, int n, int level, long long* acc_host);
int launch_eta_integral(mom5gpu_domain* d, const double* eta, double* out_host);
int launch_check_finite(mom5gpu_domain* d, const double* a, size_t count, int* out_host);

// FP64 MDFL scratch of a domain, for ntr tracers at a time (k_fp64.cu)
int ensure_mdfl_scratch(mom5gpu_domain* d, int ntr);

// ---- batched launches (k_batch64.cu, k_batch.cu) ----
// One work list in device memory: entries[e] is the descriptor index of entry
// e; p*[e] is the first block of entry e in each pass (p*[count] = total).
struct BatchWork {
  const int* entries;
  const int *pz, *px, *py, *pb2, *pb1, *pm;
  int count;
  int tz, tx, ty, tb2, tb1, tm;      // total blocks of each pass
  int seg;                           // levels per item of the precision form
  bool early;                        // the precision form's subcycles load early (BtResident)
};
// blocks of one domain in each pass, for the work-list prefix sums; m: the
// precision form's items, tiles of tile_rows rows by segments of seg levels
struct BatchBlocks {
  int z, x, y, b2, b1, m;
};
BatchBlocks batch_blocks(const Geo& g, int TJ, int tile_rows, int seg);
// FP64: z/x/y MDFL passes, the last with the explicit update, for every entry
void launch_batch_fp64_advection(const MdflArgs* mdfl, const BatchWork& w, int ntr, bool sweby, int TJ, cudaStream_t s);
// the barotropic step (init, nts x (pred, mom, corr), post) for every entry; halo fills of
// cyclic domains are issued by the caller between the post phases
void launch_batch_barotropic_loop(const BtArgs* bt, const BtExtra* x, const BatchWork& w, int nts, int stepB, bool fast,
                                  cudaStream_t s);
// precision form: folded subcycle over the work list (k_batch.cu)
void launch_batch_btf_prep(const BtArgs* bt, const BatchWork& w, cudaStream_t s);
int launch_batch_btf_subcycle(const BtArgs* bt, const BatchWork& w, int itime, int nts, cudaStream_t s);
void launch_batch_barotropic_post(const BtArgs* bt, const BtExtra* x, const BatchWork& w, int nts, int stepB, int phase,
                                  cudaStream_t s);

// ---- precision-form advection (k_mixed_stream.cu) ----
// tile height of a tuning value (16, 24, or by the tracer count), a domain's tiles
// of that height, and the levels per segment for a launch of so many tiles
int stream_tile_rows(int tuned, int ntr, bool batch);
long stream_tiles(const Geo& g, int rows);
int stream_levels(long tiles, int nk, int ntr, int rows);
// the tracers of a (at most 10) of one domain, outputs numbered from n0
int launch_mixed_stream(mom5gpu_domain* d, const MixArgs& a, int n0);
// persistent kernel over a batch's items
int launch_batch_mixed(const MixArgs* mix, const BatchWork& w, int ntr, int tuned_rows, int blocks_per_sm, int sms,
                       int* counter, cudaStream_t s);
// Attributes of the kernels that up to ntr tracers may take, one domain or batched: they
// belong to the device, so every precision-form domain (tracer_advect_init) and batch
// sets them for its own, before any launch or capture.
int prepare_mixed(int ntr, bool batch);

// ---- precision form (k_mixed.cu) ----
int launch_mdfl_mixed(mom5gpu_domain* d, int n_first, int ntr, int taum1, int tau, int taup1, double dtime,
                      bool fused_update);
int ensure_wait_words(mom5gpu_domain* d);

}  // namespace mom5
