// Kernel parameter blocks and launchers of the FDAS hot path.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>

#include "hsum_boxes.cuh"

namespace fdas {

constexpr int kTile = 2048;          // FFT / tile size (gen_info.h:33, 42)
constexpr int kMaxPlanes = 16;       // harmonic planes supported by the kernels
constexpr int kSortCap = 8192;       // boundary records one CTA ranks in shared memory
constexpr int kMaxCompat = 2048;     // entries per plane of the fixed-size list
constexpr int kSelBuckets = 2048;    // power buckets of the top-K selection (float bits 30..20)
constexpr int kFinSlices = 8;        // CTAs per plane that write the fixed-size list (slices of its entries)

// device status bits (per buffer set)
constexpr int kStatusHsumTimeout = 1;
constexpr int kStatusRecheckOverflow = 2;
constexpr int kStatusCandidateOverflow = 4;
constexpr int kStatusSelectionOverflow = 8;
constexpr int kStatusFtcTimeout = 16;

// Device-side waits.  kWaitNs is the default bound after which a wait is
// reported as timed out (FtcParams / HsumParams::timeout_ns may lower it);
// kDrainNs bounds the wait for a kernel's own copies in flight before it
// exits after a timeout, so no CTA ends with a copy into its shared memory
// still pending.
constexpr long long kWaitNs = 2000000000LL;
constexpr long long kDrainNs = 2000000000LL;

// Candidate record key: plane << 48 | row << 32 | bin.  Ascending key order is
// (harmonic, template, bin) -- the order of hsum.py's list.
__host__ __device__ inline unsigned long long cand_key(int plane, int row, int bin) {
  return ((unsigned long long)(unsigned)plane << 48) | ((unsigned long long)(unsigned)row << 32) | (unsigned)bin;
}

// Programmatic dependent launch: a kernel launched with `pdl` may start while
// the kernel before it on the stream still runs, and reads or writes global
// memory only after grid_wait(); the kernel before lets it start with
// grid_release() (or by ending).  Both do nothing without the launch attribute.
// Hides launch latency and prologues, which bound short spectra: the
// allocation-free FT convolution of 4096 bins takes 10.2 us with it and 12.3 without,
// of 100003 x 43 rows 20.5 / 23.6, a search of 32768 bins 53 / 71 us, of 2^21 bins 642 /
// 673; an event between two kernels costs the same 2 us as a plain launch.
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// Where a kernel's work ends, by %globaltimer (32 ns steps here), or nothing: written by
// its last block (blocks start in order, so short ones of equal work end within a
// block's time of it), or the latest of all blocks, into a word that starts from zero.
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ void stamp_last_block(unsigned long long *at) {
  if (at && blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) *at = global_ns();
}
__device__ __forceinline__ void stamp_latest(unsigned long long *at) {
  if (at && threadIdx.x == 0) atomicMax(at, global_ns());
}
// where a kernel starts, by its first block
__device__ __forceinline__ void stamp_first_block(unsigned long long *at) {
  if (at && blockIdx.x == 0 && threadIdx.x == 0) *at = global_ns();
}
// for a kernel that writes no end time, by the kernel after it where that starts
__device__ __forceinline__ void stamp_if_none(unsigned long long *at) {
  if (at && blockIdx.x == 0 && threadIdx.x == 0) atomicCAS(at, 0ull, global_ns());
}
template <typename Kernel, typename... Args>
cudaError_t launch_kernel(Kernel kern, dim3 grid, dim3 block, int smem, cudaStream_t s, bool pdl, Args... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = (size_t)smem;
  c.stream = s;
  c.attrs = &at;
  c.numAttrs = pdl ? 1 : 0;
  return cudaLaunchKernelEx(&c, kern, args...);
}
// Lets a kernel be launched with `bytes` of dynamic shared memory, every launch of it alike.
template <typename Kernel>
cudaError_t allow_smem(Kernel kern, int bytes) {
  return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}
// A kernel whose launches differ in shared memory.  The limit is one per kernel and
// device, shared by every handle and thread, so setting it and launching are one step
// under a lock: else a thread with a smaller launch lowers it between another's call and
// its launch, which then fails (18 of 2000 series FFTs of 2^20 points beside a thread
// with 4096).  One limit for all of a kernel's launches instead makes searches that run
// side by side slower (eight served requests 770 -> 800 us with harmonic summing and
// the histogram at their largest): what an SM sets aside follows the limit, not the launch.
inline std::mutex &smem_limit_lock() {
  static std::mutex lock;
  return lock;
}
template <typename Kernel, typename... Args>
cudaError_t launch_sized(Kernel kern, dim3 grid, dim3 block, int smem, cudaStream_t s, bool pdl, Args... args) {
  const std::lock_guard<std::mutex> hold(smem_limit_lock());
  const cudaError_t e = allow_smem(kern, smem);
  return e != cudaSuccess ? e : launch_kernel(kern, grid, block, smem, s, pdl, args...);
}

// ---- (a) overlap-save tiling + forward FFT (tile_input.cl.mako, fft_4p.cl)
// One trial of a batched search: its tiles are the global tiles
// [tile_begin, next trial's tile_begin), its spectrum starts at input_offset of
// the batch input, its FOP (n_templates rows of `stride` floats) at fop_offset.
struct BatchTrial {
  long long tile_begin;
  long long input_offset;
  long long fop_offset;
  long long stride;
  int n_bins;
  int pad_;
};

// trial of global tile `tile` (trials sorted by tile_begin; binary search)
__device__ __forceinline__ int batch_trial_of(const BatchTrial *tr, int n, long long tile) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (tr[mid].tile_begin <= tile) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

struct TileParams {
  const float2 *input;    // N spectrum bins
  float2 *copy = nullptr; // N bins: where the input is host memory, its copy for the later kernels
  int n_bins;
  int n_tiles;
  int overlap;            // O
  int payload;            // P = 2048 - O
  float2 *tiles;          // n_tiles x 2048, natural bin order
  const float2 *twiddle;  // e^(+2 pi i j / 2048), j < 2048
  const BatchTrial *trials = nullptr;  // batched search: n_tiles spans all trials
  int n_trials = 0;
  // template rows to bring into the kernels' form by CTAs of their own (the
  // allocation-free call): natural order, scaled by 2^-11
  const float2 *tmpl_src = nullptr;
  float2 *tmpl_dst = nullptr;
  int n_tmpl = 0;
  int tmpl_p4 = 0;           // the source is in p4 order
  unsigned *zero = nullptr;  // words to zero before the following kernels run (a search's control words)
  int n_zero = 0;
  unsigned long long *stamp = nullptr;  // end time (stage times of a search enqueued in one go)
};

// ---- (c) template multiply + inverse FFT + |.|^2 + discard (mux_and_mult,
//      square_and_discard)
struct FtcParams {
  const float2 *tiles;    // n_tiles x 2048
  const float2 *tmpl;     // n_templates x 2048 spectra, natural order, scaled by 2^-11
  float *fop;             // n_templates x stride
  long long fop_stride;
  int n_bins;
  int n_tiles;
  int overlap;
  int payload;
  int row_begin;          // first FOP row of the part
  int n_rows;             // rows of the part
  const float2 *twiddle;
  int *status;
  long long timeout_ns;
  int ctas_per_sm;        // 1: the pair form, half an SM (leaves room for harmonic summing); else the group form
  int group_tiles = 8;    // group form: tiles per CTA and step (set by launch_ftc)
  int variant = 0;        // FFT split: 0 default, 1 one warp per item (64 x 32), 2 a warp pair (32 x 64);
                          // 3 / 4: tensor-core DFT factors with split BF16 / FP16 operands
  const BatchTrial *trials = nullptr;  // batched search: tiles of all trials, FOPs per trial
  int n_trials = 0;
  long long tile_begin = 0;  // batched search: global index of the launch's first tile
  int inject_stall = 0;      // test hook: the first template copy (of each CTA, or of each warp pair in the
                             // pair form) is announced on its barrier but not issued, so that wait runs
                             // out (nothing is in flight)
  // forward transform of the tiles on the tensor cores (precision form):
  // items are tiles, read from `input` (n_bins spectrum values) and written
  // to `tiles_out` as complex spectra
  const float2 *input = nullptr;
  float2 *tiles_out = nullptr;
  unsigned long long *stamp = nullptr;        // end time (group form)
  // start time, the tiling's end for the pair form, whose registers are at their limit:
  // it writes no end time, and with this store at its head it compiles to 522 us at 2^21
  // bins x 85 rows, without it to 545
  unsigned long long *stamp_begin = nullptr;
};

// ---- (d) harmonic summing + thresholds + candidate compaction (preload,
//      delay, detect, store_cands; hms_baseline.cl.mako)
struct HsumParams {
  const float *fop;
  long long stride;
  int n_bins;
  int half;               // n_templates / 2: row of template t is half + t
  int n_planes;
  int tlo[2];             // first |t| of the negative / positive half; > half disables it
  float trig[kMaxPlanes]; // fast-path trigger: a cell needs a closer look if HP >= trig
  float hi[kMaxPlanes];   // candidate if HP > hi
  float lo[kMaxPlanes];   // recheck if lo <= HP <= hi (lo = +inf: never)
  // staging boxes: plane 1 is kHsBins bins x 4 NW rows; plane j >= 2 is bw[j] bins
  // (from (f0/j) rounded down to 4) x bh[j] rows (trunc(t/j) of the half)
  int bw[kMaxPlanes + 1];
  int bh[kMaxPlanes + 1];
  int soff[kMaxPlanes + 1]; // float offset of plane j's box in a stage (128-byte aligned)
  int stage_floats;         // floats per pipeline stage
  unsigned stage_bytes;     // bytes the TMA copies deliver per stage
  unsigned *item_counter;   // dynamic work distribution
  unsigned long long *cand_key;  // [cap] records, any order
  float *cand_pwr;               // [cap]
  unsigned *cand_total;          // records appended (may exceed cap)
  unsigned *cand_count;          // [plane] hits per plane
  int cand_cap;
  uint4 *rc_list;         // recheck entries (plane, row, bin, 0)
  unsigned *rc_count;
  int rc_cap;
  int *status;
  long long timeout_ns;   // bound on every wait
  int lean;               // 1: fewer stages and registers (shares an SM with the FT convolution)
  int inject_stall = 0;   // test hook: the first stage of every CTA is announced on its barriers
                          // but its copies are not issued, so the consumers' waits run out
  unsigned long long *stamp = nullptr;  // end time of the FT convolution, where its kernel wrote none
};

// 2-D tensor maps of the FOP (rows x stride floats), one box shape per plane
struct HsumMaps {
  CUtensorMap map[kMaxPlanes + 1];
};

// ---- FP64 recheck of near-threshold cells
struct RecheckParams {
  const float2 *input;    // the spectrum the FOP was computed from
  int n_bins;
  int n_planes;
  int half;
  const float4 *taps;     // n_templates x tap_pitch time-domain taps as float pairs
                          // (re hi, im hi, re lo, im lo): tap = hi + lo to 2^-48
  const int *tap_len;     // taps per template
  int tap_pitch;
  double thr[kMaxPlanes];
  const uint4 *rc_list;
  const unsigned *rc_count;
  int rc_cap;
  unsigned long long *cand_key;
  float *cand_pwr;
  unsigned *cand_total;
  unsigned *cand_count;
  int cand_cap;
  int *status;
};

// ---- deterministic top-K per plane + fixed-size list
struct SelectParams {
  const unsigned long long *cand_key;
  const float *cand_pwr;
  const unsigned *cand_total;
  const unsigned *cand_count;   // [plane]
  int cand_cap;
  int n_planes;
  int per_plane;          // K: entries per plane in the fixed-size list
  unsigned *hist;         // [plane][kSelBuckets], left zeroed after use
  unsigned *ticket;       // last-block detection of the histogram kernel
  int *sel_bucket;        // [plane] boundary bucket (-1: take every hit)
  unsigned *sure_count;   // [plane] records above the boundary bucket
  unsigned *bound_count;  // [plane] records in the boundary bucket
  unsigned long long *sel_key;  // [plane][2][kSortCap]: sure list, boundary list
  float *sel_pwr;
  uint32_t *compat_loc;   // [plane][per_plane]
  float *compat_pwr;
  uint32_t *host_loc;     // the list once more, in the set's pinned host memory
  float *host_pwr;
  uint32_t *user_loc;     // and in the caller's, where that is pinned too (or null)
  float *user_pwr;
  unsigned long long *host_key;  // the first n_host_rec records, in pinned host memory
  float *host_rec_pwr;
  unsigned n_host_rec;
  uint32_t invalid_location;
  int *status;
  const unsigned *ctrl;   // n_ctrl control words, copied to pinned host memory at the end
  unsigned *host_ctrl;
  int n_ctrl;
  unsigned long long *stamp;  // [plane][kFinSlices] end times of the last kernel's CTAs, in pinned host memory
};

// ---- template spectra / taps in FP64
struct SpectraParams {
  const double2 *taps;    // n_templates x tap_pitch
  const int *tap_len;
  int tap_pitch;
  int n_templates;
  const double2 *twiddle64;  // e^(-2 pi i j / 2048)
  float2 *spectra;        // n_templates x 2048, natural, scaled by 2^-11
};

struct TapsParams {
  const float2 *spectra;  // n_templates x 2048 natural, unscaled
  int n_templates;
  int n_taps;             // taps to recover per template
  const double2 *twiddle64;
  double2 *taps;          // n_templates x tap_pitch
  int *tap_len;
  int tap_pitch;
};

// ---- upstream: spectrum of a real series (ft_conv.py:134-143)
struct SeriesParams {
  const float2 *samples;  // the 2N samples as N complex values (p.z, or the caller's device memory: only read)
  float2 *z;              // N complex: the N-bin spectrum on exit
  float2 *host;           // and once more in pinned host memory, or null
  float2 *scratch;        // N complex
  const float4 *tw;       // series_twiddle_count(n) entries
  int n;                  // N
  float scale;            // applied to every output bin (1 / (2N) in ft_conv.py)
};
// one pass of an N-point FFT: radix R over columns j < m = N / R, ns = product of
// the radices before; in steps of radix[] inside a CTA of B columns
struct SeriesPass {
  int R, m, ns;
  int unit;               // 2N / (ns R): table steps per twiddle exponent
  int B, log_b;
  int n_steps, threads;
  int radix[8];
};
constexpr int kTwFine = 2048;  // entries of the fine twiddle table
// passes of an N-point FFT; -1 if N has a factor other than 2, 3, 5, 7
int series_plan(int n, SeriesPass *pass, int max_passes);
size_t series_twiddle_count(int n);
cudaError_t launch_series_twiddles(float4 *tw, int n, cudaStream_t s);
cudaError_t launch_series_spectrum(const SeriesParams &p, cudaStream_t s);

cudaError_t launch_tile_fft(const TileParams &p, cudaStream_t s, bool pdl = false);
cudaError_t launch_ftc(const FtcParams &p, cudaStream_t s, bool pdl = false);
// precision form: inverse DFT on tcgen05 with split FP16 (f16) or BF16 operands
cudaError_t launch_ftc_tc(const FtcParams &p, bool f16, cudaStream_t s);
// precision form: tiling + forward DFT of the tiles on tcgen05, the same DFT
// factors conjugated; status / timeout as for the FT convolution
cudaError_t launch_tile_tc(const TileParams &p, bool f16, int *status, long long timeout_ns, cudaStream_t s);
cudaError_t launch_hsum(const HsumParams &p, const HsumMaps &m, cudaStream_t s, bool pdl = false);
constexpr int kHsMaxSmem = 227 * 1024;  // what an SM has for one CTA
// consumer warps of the harmonic-summing kernel for `half` (4 templates each)
int hsum_warps(int half);
cudaError_t launch_recheck(const RecheckParams &p, cudaStream_t s, bool pdl = false);
cudaError_t launch_split_taps(double2 *taps, long long n, cudaStream_t s);
cudaError_t launch_select(const SelectParams &p, cudaStream_t s, bool pdl = false);
cudaError_t launch_spectra(const SpectraParams &p, cudaStream_t s);
cudaError_t launch_taps(const TapsParams &p, cudaStream_t s);

// SM count of the current device, queried on every call (a process may drive
// GPUs with different SM counts; the query costs well under a microsecond)
int current_sm_count();

// shared memory bytes needed by launch_hsum for a given plane geometry
int hsum_smem_bytes(const HsumParams &p);
constexpr int kStatusHsumSetup = 32;

}  // namespace fdas
