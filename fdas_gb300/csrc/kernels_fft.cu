// (a) overlap-save tiling + forward FFT, (c) fused template multiply,
// inverse FFT, power and overlap discard, and the FP64 template precompute.
#include <climits>
#include <cstdlib>
#include <cstring>

#include "fft2048.cuh"
#include "kernels.cuh"

namespace fdas {

constexpr int kWarpsPerCta = 8;

// Four warps per tile, 16 values per thread: 2048 = 16 x 16 x 8, DFT16, DFT16 and
// two DFT8 with two exchanges through one 16.5 KB buffer.  With n = n0 + 128 n1,
// n0 = m0 + 8 m1, k = k0 + 16 k1 + 256 k2:
//   thread n0         Y[n0][k0] = DFT16_n1(x[n0 + 128 n1]) w^(-n0 k0)
//   thread (m0, k0)   U[m0][k1] = DFT16_m1(Y[m0 + 8 m1][k0]) w^(-16 m0 k1)
//   thread c, c + 128 X[c + 256 k2] = DFT8_m0(U[m0][k1]), c = k0 + 16 k1
// so loads and stores are unit-stride.  One warp per tile (64 values a lane) was
// bound by that warp's chain; tiling at 2^21 / 2^19 / 2^15 bins: 10.3 / 4.8 / 2.7 us
// against 16.2 / 11.3 / 9.5.  At 2^21 the 1289 CTAs of 8 per SM are one wave and a
// bit; 17 MB are read and 21 written (5.6 us at the copy rate).  Tile i covers spectrum bins [i P - O,
// i P + P): bins below 0 (the first tile's overlap) and from N on (the last
// tile's padding) read as zero -- tile_input.cl.mako:42-94 / ft_conv.py:165-180.
constexpr int kTileThreads = 128;
constexpr int kTilePitch = 129;  // odd: the column reads of the first exchange meet no bank twice
// HOST: the input is pinned host memory, and its copy is left at p.copy.
// TMPL: CTAs past the tiles bring a template row each into the kernels' form (by a
// kernel of its own before the tiling, the allocation-free call of 4096 bins took
// 12.0 us against 10.4, of 100003 bins x 43 rows 21.3 / 20.5, of 2^19 93.6 / 89.4).

// p4 position 4 s + j holds natural bin bitrev2(j) * 512 + s
// (tmpl-gen.py:145-153).  Rows are read in order; scaled by 2^-11 (the inverse
// transform's 1/2048, exact in float).
__device__ __forceinline__ void convert_template(const TileParams &p, int row, int t) {
  const float2 *src = p.tmpl_src + (long long)row * kTile + t;
  float2 *dst = p.tmpl_dst + (long long)row * kTile;
  float2 v[16];
  sfor<16>([&](auto I) { v[decltype(I)::value] = src[128 * decltype(I)::value]; });
  sfor<16>([&](auto I) {
    constexpr int i = decltype(I)::value;
    const int q = 128 * i + t;
    const int k = p.tmpl_p4 ? (((q & 1) << 1) | ((q >> 1) & 1)) * 512 + (q >> 2) : q;
    dst[k] = make_float2(v[i].x * (1.0f / 2048.0f), v[i].y * (1.0f / 2048.0f));
  });
}

template <bool BATCH, bool HOST, bool TMPL>
__global__ void __launch_bounds__(kTileThreads, 8) tile_fft_kernel(TileParams p) {
  __shared__ float2 ex[16 * kTilePitch];
  const int t = threadIdx.x;
  const int tile = blockIdx.x;
  grid_release();
  if constexpr (TMPL)
    if (tile >= p.n_tiles) {
      grid_wait();
      convert_template(p, tile - p.n_tiles, t);
      return;
    }
  const int m0 = t >> 4, k0 = t & 15;
  float2 w[16];  // twiddles, there before the tile is
  sfor<15>([&](auto K) {
    constexpr int k = decltype(K)::value + 1;
    w[k] = __ldg(p.twiddle + k * t);  // k t < 2048
  });
  const float2 *input = p.input;
  int n_bins = p.n_bins;
  long long local = tile;
  if constexpr (BATCH) {  // batched: the trial's own spectrum and tile numbering
    const BatchTrial &tr = p.trials[batch_trial_of(p.trials, p.n_trials, tile)];
    input += tr.input_offset;
    n_bins = tr.n_bins;
    local = tile - tr.tile_begin;
  }
  grid_wait();
  if (blockIdx.x == 0)
    for (int i = t; i < p.n_zero; i += kTileThreads) p.zero[i] = 0u;
  const long long start = local * p.payload - p.overlap + t;
  float2 v[16];
  sfor<16>([&](auto N1) {
    constexpr int n1 = decltype(N1)::value;
    const long long b = start + 128 * n1;
    v[n1] = (b >= 0 && b < n_bins) ? input[b] : make_float2(0.f, 0.f);
  });
  if constexpr (HOST)  // the bins past the overlap are this tile's own
    sfor<16>([&](auto N1) {
      constexpr int n1 = decltype(N1)::value;
      const long long b = start + 128 * n1;
      if (t + 128 * n1 >= p.overlap && b < n_bins) p.copy[b] = v[n1];
    });
  // (the table holds w^j = e^(+2 pi i j / 2048); conjugated here)
  auto conj_mul = [](float2 a, float2 b) {
    return make_float2(fmaf(a.x, b.x, a.y * b.y), fmaf(a.y, b.x, -a.x * b.y));
  };
  dft16<-1, 0>(v);
  sfor<16>([&](auto K) {
    constexpr int k = decltype(K)::value;
    float2 y = v[pos16(k)];
    if constexpr (k > 0) y = conj_mul(y, w[k]);
    ex[k * kTilePitch + t] = y;
  });
  sfor<15>([&](auto K) {
    constexpr int k = decltype(K)::value + 1;
    w[k] = __ldg(p.twiddle + 16 * k * m0);  // < 2048
  });
  __syncthreads();
  sfor<16>([&](auto M1) {
    constexpr int m1 = decltype(M1)::value;
    v[m1] = ex[k0 * kTilePitch + m0 + 8 * m1];
  });
  __syncthreads();
  dft16<-1, 0>(v);
  sfor<16>([&](auto K) {
    constexpr int k = decltype(K)::value;
    float2 y = v[pos16(k)];
    if constexpr (k > 0) y = conj_mul(y, w[k]);
    ex[256 * m0 + k0 + 16 * k] = y;
  });
  __syncthreads();
  float2 *out = p.tiles + (long long)tile * kTile + t;
  sfor<2>([&](auto C) {
    constexpr int c = decltype(C)::value;
    float2 u[8];
    sfor<8>([&](auto M) {
      constexpr int m = decltype(M)::value;
      u[m] = ex[256 * m + 128 * c + t];
    });
    dft8<-1, 0, 1>(u);
    sfor<8>([&](auto K) {
      constexpr int k = decltype(K)::value;
      out[128 * c + 256 * k] = u[k];
    });
  });
  stamp_last_block(p.stamp);
}

// ------------------------------------------------------------ TMA helpers
__device__ __forceinline__ uint32_t smem_addr(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(smem_addr(bar)), "r"(parity)
      : "memory");
  return done != 0;
}
__device__ __forceinline__ uint64_t gtimer() {
  uint64_t t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, long long timeout_ns) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = gtimer();
  while (!mbar_try_wait(bar, parity))
    if ((long long)(gtimer() - t0) > timeout_ns) return false;
  return true;
}
// 16 KB template spectrum -> this warp's exchange buffer (async proxy)
__device__ __forceinline__ void prefetch_template(float *ex, const float2 *src, uint64_t *bar) {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  mbar_arrive_expect_tx(bar, kTile * 8);
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_addr(ex)),
      "l"(src), "r"((uint32_t)(kTile * 8)), "r"(smem_addr(bar))
      : "memory");
}

// Where the outputs of (global tile, FOP row) go: the row's start, the bin of
// the tile's first output (before the discard) and the row length.
struct FopTarget {
  float *out;
  long long base;
  int n_bins;
};
// The trial of a warp's (or pair's) current item in the batched search, its
// fields held in registers.  A warp's items only move forward (item += grid
// size), so after one binary search at the first item the trial is found by
// walking forward from the previous one -- usually no step at all -- instead
// of a dependent chain of loads per item.
struct TrialCursor {
  long long next_begin;  // first global tile of the next trial
  long long tile_begin;  // first global tile of this trial
  long long fop_offset;
  long long stride;
  int t;
  int n_bins;
};
__device__ __forceinline__ void cursor_load(const FtcParams &p, TrialCursor &c) {
  const BatchTrial &tr = p.trials[c.t];
  c.tile_begin = tr.tile_begin;
  c.fop_offset = tr.fop_offset;
  c.stride = tr.stride;
  c.n_bins = tr.n_bins;
  c.next_begin = c.t + 1 < p.n_trials ? p.trials[c.t + 1].tile_begin : LLONG_MAX;
}
template <bool BATCH>
__device__ __forceinline__ void cursor_start(const FtcParams &p, int tile, TrialCursor &c) {
  if constexpr (BATCH) {
    c.t = batch_trial_of(p.trials, p.n_trials, p.tile_begin + tile);  // the launch may cover a range of tiles
    cursor_load(p, c);
  }
}
template <bool BATCH>
__device__ __forceinline__ void cursor_seek(const FtcParams &p, int tile, TrialCursor &c) {
  if constexpr (BATCH) {
    while (p.tile_begin + tile >= c.next_begin) {
      ++c.t;
      cursor_load(p, c);
    }
  }
}
template <bool BATCH>
__device__ __forceinline__ FopTarget fop_target(const FtcParams &p, int tile, int row, const TrialCursor &c) {
  if constexpr (!BATCH)
    return FopTarget{p.fop + (long long)row * p.fop_stride, (long long)tile * p.payload - p.overlap, p.n_bins};
  return FopTarget{p.fop + c.fop_offset + (long long)row * c.stride,
                   (p.tile_begin + tile - c.tile_begin) * p.payload - p.overlap, c.n_bins};
}

template <bool BATCH>
__global__ void __launch_bounds__(256, 1) ftc_kernel(FtcParams p) {
  extern __shared__ float4 smem_f4[];
  __shared__ uint64_t bars[kWarpsPerCta];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float *ex = reinterpret_cast<float *>(smem_f4) + warp * kExFloats;
  uint64_t *bar = &bars[warp];
  const int n_items = p.n_tiles * p.n_rows;
  const int stride = gridDim.x * kWarpsPerCta;
  int item = blockIdx.x * kWarpsPerCta + warp;
  if (lane == 0) {
    mbar_init(bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  const TwiddleBases tb = load_twiddle_bases<+1>(p.twiddle, lane);
  if (item < n_items && lane == 0)
    prefetch_template(ex, p.tmpl + (long long)(p.row_begin + item % p.n_rows) * kTile, bar);
  uint32_t parity = 0;
  TrialCursor cur;
  if (item < n_items) cursor_start<BATCH>(p, item / p.n_rows, cur);
  for (; item < n_items; item += stride) {
    const int tile = item / p.n_rows;
    const int row = p.row_begin + (item - tile * p.n_rows);
    cursor_seek<BATCH>(p, tile, cur);
    const float2 *s = p.tiles + (long long)tile * kTile + lane;
    float2 v[64];
    sfor<64>([&](auto K) {
      constexpr int k = decltype(K)::value;
      v[k] = __ldg(s + 32 * k);
    });
    if (!mbar_wait(bar, parity, p.timeout_ns)) {
      if (lane == 0) atomicOr(p.status, kStatusFtcTimeout);
      mbar_wait(bar, parity, kDrainNs);  // bounded: let the copy land before exiting
      return;
    }
    parity ^= 1u;
    const float2 *t = reinterpret_cast<const float2 *>(ex) + lane;
    sfor<64>([&](auto K) {
      constexpr int k = decltype(K)::value;
      v[k] = cmul(v[k], t[32 * k]);
    });
    const int next = item + stride;
    ifft2048_core(v, tb, ex, lane, [&]() {
      if (next < n_items && lane == 0)
        prefetch_template(ex, p.tmpl + (long long)(p.row_begin + next % p.n_rows) * kTile, bar);
    });
    const FopTarget tg = fop_target<BATCH>(p, tile, row, cur);
    sfor<2>([&](auto C) {
      constexpr int c = decltype(C)::value;
      sfor<32>([&](auto D) {
        constexpr int d = decltype(D)::value;
        const int n = lane + 32 * c + 64 * d;
        const long long b = tg.base + n;
        const float2 y = v[32 * c + pos32(d)];
        if (n >= p.overlap && b < tg.n_bins) tg.out[b] = fmaf(y.x, y.x, y.y * y.y);
      });
    });
  }
}

// ---------------------------------------------------------------------------
// Pair form, one CTA of 4 pairs per SM: half an SM's registers, so that harmonic
// summing fits beside it (one warp pair per (tile, template) item, 32 values per
// thread, <= 128 registers).  The pair buffer
// (16.9 KB) holds the TMA-prefetched template spectrum of the item, then the
// pass-1 exchange; the next item's template is prefetched into it as soon as
// both warps have read the exchange back.
constexpr int kPairsPerCta = 4;

__device__ __forceinline__ void pair_sync(int pair) {
  asm volatile("bar.sync %0, %1;" ::"r"(pair + 1), "r"(64) : "memory");
}
// barrier over the pair that also ANDs a predicate across its 64 threads
__device__ __forceinline__ bool pair_and(int pair, bool v) {
  unsigned r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "bar.red.and.pred q, %2, %3, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"((unsigned)v), "r"(pair + 1), "r"(64)
      : "memory");
  return r != 0;
}

template <bool BATCH>
__global__ void __launch_bounds__(256, 2) ftc2_kernel(FtcParams p) {
  extern __shared__ float4 smem_f4[];
  __shared__ uint64_t bars[kPairsPerCta];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int pair = warp >> 1, h = warp & 1;
  const int tp = 32 * h + lane;  // thread of the pair
  float *buf_f = reinterpret_cast<float *>(smem_f4) + pair * kEx2Floats;
  float2 *twt = reinterpret_cast<float2 *>(reinterpret_cast<float *>(smem_f4) + kPairsPerCta * kEx2Floats);
  float2 *buf = reinterpret_cast<float2 *>(buf_f);
  uint64_t *bar = &bars[pair];
  const int n_items = p.n_tiles * p.n_rows;
  const int stride = gridDim.x * kPairsPerCta;
  int item = blockIdx.x * kPairsPerCta + pair;
  if (tp == 0) {
    mbar_init(bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  fill_twiddle2(twt, p.twiddle);
  stamp_first_block(p.stamp_begin);
  __syncthreads();
  if (item < n_items && tp == 0) {
    if (p.inject_stall) mbar_arrive_expect_tx(bar, kTile * 8);  // test hook: a copy that never comes
    else prefetch_template(buf_f, p.tmpl + (long long)(p.row_begin + item % p.n_rows) * kTile, bar);
  }
  uint32_t parity = 0;
  const int m = 16 * h + (lane & 15);
  const int g = lane >> 4;
  // (tile, row) of the item, advanced by the grid stride without divisions
  const int st_tiles = stride / p.n_rows, st_rows = stride - st_tiles * p.n_rows;
  int tile = item / p.n_rows, rr = item - tile * p.n_rows;
  TrialCursor cur;
  if (item < n_items) cursor_start<BATCH>(p, tile, cur);
  for (; item < n_items; item += stride) {
    const int row = p.row_begin + rr;
    int next_tile = tile + st_tiles, next_rr = rr + st_rows;
    if (next_rr >= p.n_rows) {
      next_rr -= p.n_rows;
      ++next_tile;
    }
    cursor_seek<BATCH>(p, tile, cur);
    const float2 *s = p.tiles + (long long)tile * kTile + tp;
    float2 v[32];
    sfor<32>([&](auto A) {
      constexpr int a = decltype(A)::value;
      v[a] = __ldg(s + 64 * a);
    });
    // the decision to go on is made uniform over the pair
    if (!pair_and(pair, mbar_wait(bar, parity, p.timeout_ns))) {
      if (tp == 0) atomicOr(p.status, kStatusFtcTimeout);
      // bounded: let the copy land before exiting (the test hook issued none)
      if (!p.inject_stall) mbar_wait(bar, parity, kDrainNs);
      return;
    }
    parity ^= 1u;
    sfor<32>([&](auto A) {
      constexpr int a = decltype(A)::value;
      v[a] = cmul(v[a], buf[64 * a + tp]);
    });
    pair_sync(pair);  // template read by both warps: the buffer takes the exchange
    ifft2_pass1(v, twt, buf, tp);
    pair_sync(pair);  // exchange written
    const int next = item + stride;
    float pw[32];
    ifft2_pass2(buf, h, lane, pw, [&]() {
      pair_sync(pair);  // exchange read by both warps: prefetch the next template
      if (next < n_items && tp == 0)
        prefetch_template(buf_f, p.tmpl + (long long)(p.row_begin + next_rr) * kTile, bar);
    });
    // output n = m + 128 g + c, c = 32 r + 256 d2 known at compile time: the
    // discard (n >= O) and the row end (bin < n_bins) become two 32-bit
    // limits on c per thread and item
    const FopTarget tg = fop_target<BATCH>(p, tile, row, cur);
    const int mb = m + 128 * g;
    const long long first = tg.base + mb;  // bin of c = 0 (negative in the first tile)
    const long long room = (long long)tg.n_bins - first;
    const int lo = p.overlap - mb, hi = room < kTile ? (int)room : kTile;
    const unsigned long long dst =
        reinterpret_cast<unsigned long long>(tg.out) + 4ull * static_cast<unsigned long long>(first);
    sfor<4>([&](auto R) {
      constexpr int r = decltype(R)::value;
      sfor<8>([&](auto D2) {
        constexpr int d2 = decltype(D2)::value;
        constexpr int c = 32 * r + 256 * d2;
        if (c >= lo && c < hi) *reinterpret_cast<float *>(dst + 4ull * c) = pw[8 * r + d2];
      });
    });
    tile = next_tile;
    rr = next_rr;
  }
}

// ---------------------------------------------------------------------------
// Group form, the FT convolution wherever it has the SMs for itself: 8 warp
// pairs per CTA, one CTA per SM, each pair with one tile of a group of
// consecutive tiles, all of them on the same template row at about the same time.
// The template rows pass through a ring of shared-memory slots, one 16 KB TMA
// copy for all pairs of the CTA.  The pair's tile spectrum and its twiddles stay
// in tensor memory over the rows, used as 128 words of private storage per thread
// (32 lanes x 128 columns per warp): registers hold one transform only, and
// neither passes through L1 / shared memory again.
// Work: the steps (group, row) in row-major order are split evenly over the
// grid, so every CTA has the same number of steps to within one whatever the
// number of tiles.
// Bound by the shared-memory pipe and the FMA pipe about alike (2^19 bins x 85
// rows: 67% and 65% busy, math-pipe throttling first among the stalls, 475
// shared-memory wavefronts per item); the pair form above has 654 and its L1TEX
// pipe 78% busy.  FT convolution at 2^21 / 2^19 / 2^15 bins x 85 rows: 303 / 81 /
// 11.1 us against 432 / 118 / 19.4 us of the pair form.  The same with 6 pairs and the
// tile in registers (168 a thread) took 361 us, 4 pairs of two rows each 488 us;
// the twiddle products all packed 336 us, all scalar 345 us; pass 2 with the real
// and imaginary parts of two DFT8s side by side (all packed, but re-paired after the
// exchange) 322, an mbarrier in place of the barrier before the exchange 321.
constexpr int kGroupPairs = 8;
constexpr int kGroupRing = 5;  // what 227 KB hold beside eight pair buffers
constexpr int kGroupSmem = (kGroupRing * 2 * kTile + kGroupPairs * kEx2Floats) * (int)sizeof(float);
constexpr int kGroupTmemCols = 512;
// columns of a thread's 128: tile spectrum, then the twiddle sets of pass 2
constexpr int kTmTile = 0, kTmTw = 64;

struct GroupRing {
  uint64_t full[kGroupRing];  // copy landed
  unsigned used[kGroupRing];  // pairs that have read the slot's row
  unsigned issued[kGroupRing];
  int abort;
  uint32_t tmem;
};

// Wait for a slot.  After a timeout the CTA goes on without waiting (its FOP is
// reported as timed out), so no thread leaves a barrier of the others open.
__device__ __forceinline__ void group_wait(GroupRing &ring, int slot, uint32_t parity, const FtcParams &p) {
  if (mbar_try_wait(&ring.full[slot], parity)) return;
  volatile int *stop = &ring.abort;
  if (*stop) return;
  const uint64_t t0 = gtimer();
  while (!mbar_try_wait(&ring.full[slot], parity)) {
    if (*stop) return;
    if ((long long)(gtimer() - t0) > p.timeout_ns) {
      atomicOr(p.status, kStatusFtcTimeout);
      *stop = 1;
      return;
    }
  }
}

// Tensor memory as the thread's own storage (32x32b: one word per lane and
// column).  A load's registers hold its values after tm_wait_ld on them.
#define TM_OUT4(v, i) "=f"(v[i].x), "=f"(v[i].y), "=f"(v[i + 1].x), "=f"(v[i + 1].y)
#define TM_IO4(v, i) "+f"(v[i].x), "+f"(v[i].y), "+f"(v[i + 1].x), "+f"(v[i + 1].y)
#define TM_IN4(v, i) "f"(v[i].x), "f"(v[i].y), "f"(v[i + 1].x), "f"(v[i + 1].y)
#define TM_16(M, v, i) M(v, i), M(v, i + 2), M(v, i + 4), M(v, i + 6), M(v, i + 8), M(v, i + 10), M(v, i + 12), M(v, i + 14)
__device__ __forceinline__ void tm_ld16(uint32_t addr, float2 *v) {  // 16 complex values
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : TM_16(TM_OUT4, v, 0)
      : "r"(addr)
      : "memory");
}
__device__ __forceinline__ void tm_st16(uint32_t addr, const float2 *v) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31};" ::TM_16(TM_IN4, v, 0),
      "r"(addr)
      : "memory");
}
__device__ __forceinline__ void tm_wait_ld16(float2 *v) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" : TM_16(TM_IO4, v, 0)::"memory");
}
__device__ __forceinline__ void tm_ld_tw(uint32_t addr, TwistedTw &t) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=f"(t.t4.x), "=f"(t.t4.y), "=f"(t.t2.x), "=f"(t.t2.y), "=f"(t.t1.x), "=f"(t.t1.y), "=f"(t.t1p.x),
                 "=f"(t.t1p.y)
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void tm_st_tw(uint32_t addr, const TwistedTw &t) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%8], {%0,%1,%2,%3,%4,%5,%6,%7};" ::"f"(t.t4.x),
               "f"(t.t4.y), "f"(t.t2.x), "f"(t.t2.y), "f"(t.t1.x), "f"(t.t1.y), "f"(t.t1p.x), "f"(t.t1p.y), "r"(addr)
               : "memory");
}
__device__ __forceinline__ void tm_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// The first set of the second DFT8 fetched while the DFT8s before it run: 308 -> 303 us
// at 2^21 bins x 85 rows; the batched form (24 trials 4652 us) took 4664 with it.
template <bool BATCH>
struct TmemTwiddles {
  static constexpr bool kEarly = !BATCH;
  uint32_t base;
  __device__ __forceinline__ void issue(int k, TwistedTw &t) const { tm_ld_tw(base + kTmTw + 8 * k, t); }
  __device__ __forceinline__ void wait(TwistedTw &t) const {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+f"(t.t4.x), "+f"(t.t4.y), "+f"(t.t2.x), "+f"(t.t2.y), "+f"(t.t1.x), "+f"(t.t1.y), "+f"(t.t1p.x),
                   "+f"(t.t1p.y)::"memory");
  }
};

template <bool BATCH>
__global__ void __launch_bounds__(64 * kGroupPairs, 1) ftcg_kernel(FtcParams p) {
  extern __shared__ float4 smem_f4[];
  __shared__ GroupRing ring;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int pair = warp >> 1;
  const int tp = threadIdx.x & 63;  // thread of the pair
  const int m = 16 * (warp & 1) + (lane & 15), g = lane >> 4;
  float *slots = reinterpret_cast<float *>(smem_f4);
  float2 *buf = reinterpret_cast<float2 *>(slots + kGroupRing * 2 * kTile + pair * kEx2Floats);
  const int gt = p.group_tiles;  // tiles of a group: the pairs that work
  const long long n_steps = (long long)((p.n_tiles + gt - 1) / gt) * p.n_rows;
  const long long first_step = n_steps * blockIdx.x / gridDim.x;
  const int steps = (int)(n_steps * (blockIdx.x + 1) / gridDim.x - first_step);
  int group = (int)(first_step / p.n_rows);
  int rr = (int)(first_step - (long long)group * p.n_rows);

  grid_release();
  if (threadIdx.x == 0) {
    for (int i = 0; i < kGroupRing; ++i) {
      mbar_init(&ring.full[i], 1);
      ring.used[i] = 0;
      ring.issued[i] = 0;
    }
    ring.abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  // (past L1: each value is read once per group)
  auto load_tile = [&](int tile, float2 *v) {
    const float2 *s = p.tiles + (long long)tile * kTile + tp;
    sfor<32>([&](auto A) {
      constexpr int a = decltype(A)::value;
      v[a] = __ldcg(s + 64 * a);
    });
  };
  uint32_t tm;
  {  // up to grid_wait nothing that the kernels before have written
    const TwistedTw tws[5] = {twisted_first(p.twiddle, m, g), twisted_second(p.twiddle, m, g, 0),
                              twisted_second(p.twiddle, m, g, 1), twisted_second(p.twiddle, m, g, 2),
                              twisted_second(p.twiddle, m, g, 3)};
    if (warp == 0) {
      // registers keep any other CTA of this size off the SM, so the columns are free
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&ring.tmem)),
                   "r"(kGroupTmemCols));
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    grid_wait();
    if (threadIdx.x == 0)
      for (int i = 0; i < kGroupRing && i < steps; ++i) {
        if (i == 0 && p.inject_stall) {  // test hook: a copy that never comes
          mbar_arrive_expect_tx(&ring.full[0], kTile * 8);
          continue;
        }
        prefetch_template(slots + i * 2 * kTile, p.tmpl + (long long)(p.row_begin + (rr + i) % p.n_rows) * kTile,
                          &ring.full[i]);
        ring.issued[i] = 1;
      }
    __syncwarp();
    float2 v[32];
    load_tile(min(group * gt + pair, p.n_tiles - 1), v);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // a warp reaches the 32 lanes of its quadrant; the four warps of a quadrant
    // take 128 columns each
    tm = ring.tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(128 * (warp >> 2));
    sfor<5>([&](auto K) { tm_st_tw(tm + kTmTw + 8 * decltype(K)::value, tws[decltype(K)::value]); });
    tm_st16(tm + kTmTile, v);
    tm_st16(tm + kTmTile + 32, v + 16);
    tm_wait_st();
  }
  const TmemTwiddles<BATCH> tw{tm};

  bool active = false, fresh = true, inner = false;
  int lo = 0, hi = 0;
  unsigned long long dst = 0;  // of output c = 0 in the step's FOP row
  unsigned long long row_bytes = 0;
  TrialCursor cur;
  if constexpr (BATCH) cur.next_begin = -1;
  int slot = 0;
  uint32_t parity = 0;
  int ahead = (rr + kGroupRing) % p.n_rows;  // row of the step a slot is refilled for
  for (int i = 0; i < (pair < gt ? steps : 0); ++i) {
    if (fresh) {  // first step or a new group: this pair's tile
      const int tile = group * gt + pair;
      active = tile < p.n_tiles;
      if (active) {
        if (i > 0) {
          float2 v[32];
          load_tile(tile, v);
          tm_st16(tm + kTmTile, v);
          tm_st16(tm + kTmTile + 32, v + 16);
          tm_wait_st();
        }
        if constexpr (BATCH) {
          if (cur.next_begin < 0) cursor_start<BATCH>(p, tile, cur);
          cursor_seek<BATCH>(p, tile, cur);
        }
        const FopTarget tg = fop_target<BATCH>(p, tile, p.row_begin, cur);
        if constexpr (BATCH) row_bytes = 4ull * (unsigned long long)cur.stride;
        else row_bytes = 4ull * (unsigned long long)p.fop_stride;
        // output n = mb + c, c = 32 r + 256 d2 known at compile time: the
        // discard (n >= O) and the row end become two limits on c
        const int mb = m + 128 * g;
        const long long first_bin = tg.base + mb;
        const long long room = (long long)tg.n_bins - first_bin;
        lo = p.overlap - mb;
        hi = room < kTile ? (int)room : kTile;
        // all but the last tiles of a row keep no output below 256 and every
        // one from 512 on (at the usual overlaps)
        inner = p.overlap >= 256 && p.overlap <= 512 && tg.base + kTile <= tg.n_bins;
        dst = reinterpret_cast<unsigned long long>(tg.out) + 4ull * static_cast<unsigned long long>(first_bin) +
              row_bytes * (unsigned long long)rr;
      }
      fresh = false;
    }
    // the last pair to have read a slot refills it with the row kGroupRing steps on
    auto release = [&]() {
      if (tp == 0) {
        __threadfence_block();
        if (atomicAdd(&ring.used[slot], 1u) == (unsigned)gt - 1u) {
          ring.used[slot] = 0;
          __threadfence_block();
          if (i + kGroupRing < steps && !*reinterpret_cast<volatile int *>(&ring.abort)) {
            ring.issued[slot] += 1;
            prefetch_template(slots + slot * 2 * kTile, p.tmpl + (long long)(p.row_begin + ahead) * kTile,
                              &ring.full[slot]);
          }
        }
      }
      __syncwarp();
    };
    if (active) {
      float2 v[32];
      tm_ld16(tm + kTmTile, v);
      tm_ld16(tm + kTmTile + 32, v + 16);
      group_wait(ring, slot, parity, p);
      __syncwarp();
      tm_wait_ld16(v);
      tm_wait_ld16(v + 16);
      const float2 *row = reinterpret_cast<const float2 *>(slots + slot * 2 * kTile) + tp;
      twisted_pass1(v, [&](int a) { return row[64 * a]; });
      pair_sync(pair);  // template row and the previous item's exchange read by both warps
      twisted_store(v, buf, tp);
      pair_sync(pair);  // exchange written
      const unsigned long long out = dst;
      if (inner) {
        twisted_pass2(buf, tw, tp, release, [&](auto R, auto D2, float pw) {
          constexpr int r = decltype(R)::value, d2 = decltype(D2)::value, c = 32 * r + 256 * d2;
          if (d2 >= 2 || (d2 == 1 && c >= lo)) *reinterpret_cast<float *>(out + 4ull * c) = pw;
        });
      } else {
        twisted_pass2(buf, tw, tp, release, [&](auto R, auto D2, float pw) {
          constexpr int r = decltype(R)::value, d2 = decltype(D2)::value, c = 32 * r + 256 * d2;
          if (c >= lo && c < hi) *reinterpret_cast<float *>(out + 4ull * c) = pw;
        });
      }
      __syncwarp();
    } else {
      group_wait(ring, slot, parity, p);
      pair_sync(pair);  // no tile in the last group: the slot is handed on
      release();
    }
    if (++slot == kGroupRing) {
      slot = 0;
      parity ^= 1u;
    }
    if (++ahead == p.n_rows) ahead = 0;
    dst += row_bytes;
    if (++rr == p.n_rows) {
      rr = 0;
      ++group;
      fresh = true;
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  stamp_latest(p.stamp);
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(ring.tmem), "r"(kGroupTmemCols));
  }
  // every copy that was issued has landed before the CTA ends (after a
  // timeout: waited for, bounded)
  if (threadIdx.x == 0 && ring.abort)
    for (int i = 0; i < kGroupRing; ++i)
      if (ring.issued[i] && !(i == 0 && p.inject_stall)) mbar_wait(&ring.full[i], (ring.issued[i] - 1) & 1u, kDrainNs);
}

// FP64 DFT of the time-domain taps -> float spectra scaled by 2^-11.
__global__ void spectra_kernel(SpectraParams p) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  const int r = blockIdx.y;
  if (k >= kTile || r >= p.n_templates) return;
  const double2 *h = p.taps + (long long)r * p.tap_pitch;
  const int len = p.tap_len[r];
  double re = 0.0, im = 0.0;
  for (int q = 0; q < len; ++q) {
    const double2 w = p.twiddle64[(q * k) & (kTile - 1)];
    const double2 x = h[q];
    re += x.x * w.x - x.y * w.y;
    im += x.x * w.y + x.y * w.x;
  }
  const double scale = 1.0 / 2048.0;
  p.spectra[(long long)r * kTile + k] = make_float2((float)(re * scale), (float)(im * scale));
}

// FP64 inverse DFT of float spectra -> the first n_taps time-domain taps.
__global__ void taps_kernel(TapsParams p) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  const int r = blockIdx.y;
  if (r >= p.n_templates) return;
  if (q == 0) p.tap_len[r] = p.n_taps;
  if (q >= p.n_taps) return;
  const float2 *sp = p.spectra + (long long)r * kTile;
  double re = 0.0, im = 0.0;
  for (int k = 0; k < kTile; ++k) {
    const double2 w = p.twiddle64[(q * k) & (kTile - 1)];  // e^(-i..): use conjugate
    const float2 x = sp[k];
    re += (double)x.x * w.x + (double)x.y * w.y;
    im += (double)x.y * w.x - (double)x.x * w.y;
  }
  p.taps[(long long)r * p.tap_pitch + q] = make_double2(re / 2048.0, im / 2048.0);
}

int current_sm_count() {
  int dev = 0, n_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n_sm <= 0) {
    cudaGetLastError();
    return 1;
  }
  return n_sm;
}

static int ex_smem_bytes() { return kWarpsPerCta * kExFloats * (int)sizeof(float); }

cudaError_t launch_tile_fft(const TileParams &p, cudaStream_t s, bool pdl) {
  auto kern = p.trials   ? tile_fft_kernel<true, false, false>
              : p.copy   ? tile_fft_kernel<false, true, false>
              : p.n_tmpl ? tile_fft_kernel<false, false, true>
                         : tile_fft_kernel<false, false, false>;
  return launch_kernel(kern, dim3(p.n_tiles + p.n_tmpl), dim3(kTileThreads), 0, s, pdl, p);
}

// FFT variant of the FT convolution: the forms of two warps per item (default:
// the group form, or the pair form where one CTA per SM shall leave room for
// harmonic summing) or the one-warp form; FDAS_FTC_VARIANT=1warp selects the latter.
static int ftc_variant() {
  static int v = -1;
  if (v < 0) {
    const char *e = getenv("FDAS_FTC_VARIANT");
    v = (e && strcmp(e, "1warp") == 0) ? 1 : 2;
  }
  return v;
}

// Tiles per group of the group form: a step of 1 .. 8 tiles takes 1.24, 1.30,
// 1.95, 2.00, 2.65, 2.70, 3.40, 3.45 us (slope over the rounds at 2^19 bins x 85
// rows; an odd pair leaves two of the four schedulers a warp short), and the
// launch as long as the CTA with the most steps.  Eight for long spectra (2^19:
// 82 us, six 86, four 95); short ones do not fill their last round: 65536 bins
// x 85 rows 16 us with six against 19 with eight, 2^17 27 against 29.
static long long group_steps(int n_tiles, int n_rows, int gt) { return (long long)((n_tiles + gt - 1) / gt) * n_rows; }
static int group_tiles(int n_tiles, int n_rows, int n_sm) {
  static const int step_ns[kGroupPairs] = {1240, 1300, 1950, 2000, 2650, 2700, 3400, 3450};
  int best = kGroupPairs;
  long long best_ns = 0;
  for (int gt = kGroupPairs; gt >= 1; --gt) {
    const long long ns = (group_steps(n_tiles, n_rows, gt) + n_sm - 1) / n_sm * step_ns[gt - 1];
    if (gt == kGroupPairs || ns < best_ns) {
      best = gt;
      best_ns = ns;
    }
  }
  return best;
}

cudaError_t launch_ftc(const FtcParams &p, cudaStream_t s, bool pdl) {
  if (p.n_rows <= 0 || p.n_tiles <= 0) return cudaSuccess;
  const int n_sm = current_sm_count();
  if ((p.variant == 3 || p.variant == 4) && !p.trials) return launch_ftc_tc(p, p.variant == 4, s);
  const long long items = (long long)p.n_tiles * p.n_rows;
  if ((p.variant ? p.variant : ftc_variant()) == 1 && !p.inject_stall) {  // (no test hook in the one-warp form)
    const int smem = ex_smem_bytes();
    auto kern = p.trials ? ftc_kernel<true> : ftc_kernel<false>;
    cudaError_t e = allow_smem(kern, smem);
    if (e != cudaSuccess) return e;
    const long long ctas = (items + kWarpsPerCta - 1) / kWarpsPerCta;
    kern<<<(int)(ctas < n_sm ? ctas : n_sm), 256, smem, s>>>(p);
  } else if (p.ctas_per_sm != 1) {
    auto kern = p.trials ? ftcg_kernel<true> : ftcg_kernel<false>;
    cudaError_t e = allow_smem(kern, kGroupSmem);
    if (e != cudaSuccess) return e;
    FtcParams q = p;
    q.group_tiles = group_tiles(p.n_tiles, p.n_rows, n_sm);
    const long long steps = group_steps(p.n_tiles, p.n_rows, q.group_tiles);
    return launch_kernel(kern, dim3((unsigned)(steps < n_sm ? steps : n_sm)), dim3(64 * kGroupPairs), kGroupSmem, s,
                         pdl, q);
  } else {
    const int smem = (kPairsPerCta * kEx2Floats + kTw2Floats) * (int)sizeof(float);
    auto kern = p.trials ? ftc2_kernel<true> : ftc2_kernel<false>;
    cudaError_t e = allow_smem(kern, smem);
    if (e != cudaSuccess) return e;
    const long long ctas = (items + kPairsPerCta - 1) / kPairsPerCta;
    kern<<<(int)(ctas < n_sm ? ctas : n_sm), 256, smem, s>>>(p);
  }
  return cudaGetLastError();
}

cudaError_t launch_spectra(const SpectraParams &p, cudaStream_t s) {
  dim3 grid(kTile / 128, p.n_templates);
  spectra_kernel<<<grid, 128, 0, s>>>(p);
  return cudaGetLastError();
}

cudaError_t launch_taps(const TapsParams &p, cudaStream_t s) {
  dim3 grid((p.n_taps + 127) / 128, p.n_templates);
  taps_kernel<<<grid, 128, 0, s>>>(p);
  return cudaGetLastError();
}

}  // namespace fdas
