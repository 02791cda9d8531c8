// Precision form of MDFL Sweby: the kernels over the streaming tile
// (mixed_stream.cuh), one domain per launch or a batch's work list, and the rules
// for their launch shapes.
#include "mixed_stream.cuh"

namespace mom5 {

using namespace mixed;

namespace {

// Rows of a tile (with its halo) and blocks per SM for NP tracer pairs.  Up to two
// pairs, two blocks of 16 rows (64 registers) overlap each other's barriers:
// 720x540x50 cells, 4 tracers, 895 us against 978 to 1033 with 12, 20, 24 or 32 rows; 2
// tracers 674 against 734 to 871.  Three pairs and more do not fit twice; one block
// of 20 rows (96 registers) is the largest that spills next to nothing (8 bytes with five
// pairs, against 52 with 24 rows): 1440x1080x50, 10 tracers, 7.10 ms against 7.54 with
// 16 rows and 8.43 with 24.
constexpr int stream_rows(int np) { return np <= 2 ? 16 : 20; }
// The same for the persistent kernel, whose registers hold its work list too: a height
// that spills there pays for each spill with a trip to L2, as the tiles leave no L1
// (a step of 8 domains, precision form with 40 subcycles: 4 tracers 1.42 ms with 24
// rows, 2.00 with 16; 9 tracers 2.06 with 16, 3.03 with 20, 3.21 with 24; 6 tracers 1.65
// with 20, 1.73 with 16, 1.93 with 24; 2 tracers 1.25 with 16, 1.26 with 24).
constexpr int stream_batch_rows(int np) { return np == 2 ? 24 : np == 3 ? 20 : 16; }
constexpr int stream_blocks(int np, int rows) { return np <= 2 && rows == 16 ? 2 : 1; }

template <int NP, int ZR>
__global__ void __launch_bounds__(32 * ZR, stream_blocks(NP, ZR)) k_mdfl_stream(MixArgs a, int n0, int L) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int k0 = blockIdx.z * L, k1 = k0 + L < a.g.nk ? k0 + L : a.g.nk;
  stream_tile<NP, ZR>(a, n0, blockIdx.x, blockIdx.y, k0, k1, *reinterpret_cast<StreamSmem<NP, ZR>*>(smem_raw));
}

DEVI int find_entry_m(const int* prefix, int count, int b) {
  int lo = 0, hi = count;
  while (hi - lo > 1) {
    int mid = (lo + hi) >> 1;
    if (prefix[mid] <= b) lo = mid;
    else hi = mid;
  }
  return lo;
}

// Persistent: the resident blocks take (domain, tile, level segment) items from an
// atomic counter, largest domains first.
template <int NP, int ZR>
__global__ void __launch_bounds__(32 * ZR, stream_blocks(NP, ZR))
    kb_mdfl_stream(const MixArgs* __restrict__ d, BatchWork w, int* counter) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int item;
  for (;;) {
    if (threadIdx.x == 0) item = atomicAdd(counter, 1);
    __syncthreads();
    const int it = item;
    __syncthreads();
    if (it >= w.tm) return;
    const int e = find_entry_m(w.pm, w.count, it);
    const MixArgs& a = d[w.entries[e]];
    const int local = it - w.pm[e];
    const int ntx = (a.g.ni + TI - 1) / TI, nty = (a.g.nj + ZR - 5) / (ZR - 4);
    const int k0 = local / (ntx * nty) * w.seg, k1 = k0 + w.seg < a.g.nk ? k0 + w.seg : a.g.nk;
    stream_tile<NP, ZR>(a, 0, local % ntx, local / ntx % nty, k0, k1,
                        *reinterpret_cast<StreamSmem<NP, ZR>*>(smem_raw));
  }
}

long tiles_of(const Geo& g, int rows) { return (long)((g.ni + TI - 1) / TI) * ((g.nj + rows - 5) / (rows - 4)); }

template <int NP, int ZR>
int run(mom5gpu_domain* d, const MixArgs& a, int n0) {
  const Geo& g = d->geo;
  constexpr size_t smem = sizeof(StreamSmem<NP, ZR>);
  const int L = stream_levels(tiles_of(g, ZR), g.nk, a.ntr, ZR);
  dim3 grid((g.ni + TI - 1) / TI, (g.nj + ZR - 5) / (ZR - 4), (g.nk + L - 1) / L);
  k_mdfl_stream<NP, ZR><<<grid, 32 * ZR, smem, d->stream>>>(a, n0, L);
  count_launches(d, 1);
  return MOM5GPU_OK;
}

template <int NP, int ZR>
int run_batch(const MixArgs* m, const BatchWork& w, int bps, int sms, int* counter, cudaStream_t s) {
  const int blocks = bps < stream_blocks(NP, ZR) ? bps : stream_blocks(NP, ZR);
  cudaMemsetAsync(counter, 0, sizeof(int), s);
  kb_mdfl_stream<NP, ZR><<<blocks * sms, 32 * ZR, sizeof(StreamSmem<NP, ZR>), s>>>(m, w, counter);
  return MOM5GPU_OK;
}

// The dynamic shared memory of every tile height of NP pairs, on the current device.
template <int NP, int ZR>
bool configure(bool batch) {
  const void* k = batch ? (const void*)kb_mdfl_stream<NP, ZR> : (const void*)k_mdfl_stream<NP, ZR>;
  return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(StreamSmem<NP, ZR>)) ==
         cudaSuccess;
}

template <int NP>
bool configure_rows(bool batch) {
  return configure<NP, 16>(batch) && configure<NP, stream_rows(NP)>(batch) && configure<NP, 24>(batch);
}

// f<NP, ZR>() for ntr tracers (1..10) and a tile height of stream_tile_rows
#define STREAM_DISPATCH_ROWS(NP, F, ...)                                    \
  (rows == 24 ? F<NP, 24>(__VA_ARGS__) : rows == 16 ? F<NP, 16>(__VA_ARGS__) : F<NP, stream_rows(NP)>(__VA_ARGS__))
#define STREAM_DISPATCH(F, ...)                                             \
  (ntr <= 2   ? STREAM_DISPATCH_ROWS(1, F, __VA_ARGS__)                     \
   : ntr <= 4 ? STREAM_DISPATCH_ROWS(2, F, __VA_ARGS__)                     \
   : ntr <= 6 ? STREAM_DISPATCH_ROWS(3, F, __VA_ARGS__)                     \
   : ntr <= 8 ? STREAM_DISPATCH_ROWS(4, F, __VA_ARGS__)                     \
              : STREAM_DISPATCH_ROWS(5, F, __VA_ARGS__))

}  // namespace

int stream_tile_rows(int tuned, int ntr, bool batch) {
  const int np = (ntr + 1) / 2;
  return tuned == 16 || tuned == 24 ? tuned : batch ? stream_batch_rows(np) : stream_rows(np);
}

long stream_tiles(const Geo& g, int rows) { return tiles_of(g, rows); }

// Levels per segment of a launch of `tiles` tiles.  A domain with few tiles gives
// the level march few blocks, each a long latency-bound chain; cutting it into
// segments multiplies the blocks for about two levels more per segment (its
// prologue and the z pass of the level above).  Of all cuts the cheapest by this
// model, in level times of a block alone on its SM: each SM works through its
// share of the blocks one after another, two that share the SM taking 1.55 of one
// (measured).  Its choice, whole columns and the best of all lengths, us a step:
// 255x181x40, 4 tracers 127 (8 levels), 174, 124; 300x200x35, 4 tracers 122 (12 levels),
// 172, 120; 330x210x30, 10 tracers 267 (10 levels), 365, 255; 500x300x40, 4 tracers 292 (20
// levels), 308, 292; 37x29x12, 2 tracers 12.3 (2 levels), 34.8, 12.3.
int stream_levels(long tiles, int nk, int ntr, int rows) {
  const bool two = stream_blocks((ntr + 1) / 2, rows) == 2;
  int best = nk;
  double cost = 0.0;
  for (int want = 1; want == 1 || want <= nk / 2; ++want) {
    const int L = (nk + want - 1) / want, n = (nk + L - 1) / L;
    const long b = (tiles * n + kSms - 1) / kSms;
    const double c = (two ? 1.55 * (b / 2) + b % 2 : (double)b) * (L + (n > 1 ? 2.0 : 1.0));
    if (want == 1 || c < cost) {
      cost = c;
      best = L;
    }
  }
  return best;
}

int launch_mixed_stream(mom5gpu_domain* d, const MixArgs& a, int n0) {
  const int ntr = a.ntr, rows = stream_tile_rows(d->tune_mixed_rows, ntr, false);
  return STREAM_DISPATCH(run, d, a, n0);
}

int prepare_mixed(int ntr, bool batch) {
  const int np = ntr < 10 ? (ntr + 1) / 2 : 5;
  return (np < 1 || configure_rows<1>(batch)) && (np < 2 || configure_rows<2>(batch)) &&
                 (np < 3 || configure_rows<3>(batch)) && (np < 4 || configure_rows<4>(batch)) &&
                 (np < 5 || configure_rows<5>(batch))
             ? MOM5GPU_OK
             : MOM5GPU_ECUDA;
}

int launch_batch_mixed(const MixArgs* mix, const BatchWork& w, int ntr, int tuned_rows, int blocks_per_sm, int sms,
                       int* counter, cudaStream_t s) {
  if (w.tm <= 0) return MOM5GPU_OK;
  const int rows = stream_tile_rows(tuned_rows, ntr, true);
  return STREAM_DISPATCH(run_batch, mix, w, blocks_per_sm, sms, counter, s);
}

}  // namespace mom5
