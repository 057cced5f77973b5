// (d) harmonic summing, thresholding and candidate compaction; FP64 recheck of
// near-threshold cells; per-plane sort and the fixed-size candidate list.
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include <utility>
#include <type_traits>

#include "kernels.cuh"

namespace fdas {

template <typename F, int... I>
__device__ __forceinline__ void hs_sfor_impl(F &&f, std::integer_sequence<int, I...>) {
  (f(std::integral_constant<int, I>{}), ...);
}
template <int N, typename F>
__device__ __forceinline__ void hs_sfor(F &&f) {
  hs_sfor_impl(f, std::make_integer_sequence<int, N>{});
}

// ------------------------------------------------------------------ PTX helpers
__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t phase) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(smem_u32(bar)), "r"(phase)
      : "memory");
  return done != 0;
}
__device__ __forceinline__ uint64_t globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
// one record appended to the global list (single-thread use)
__device__ __forceinline__ void global_append(unsigned long long *keys, float *pwrs, unsigned *total, int cap,
                                              int *status, unsigned long long key, float pwr) {
  const unsigned g = atomicAdd(total, 1u);
  if (g < (unsigned)cap) {
    keys[g] = key;
    pwrs[g] = pwr;
  } else {
    atomicOr(status, kStatusCandidateOverflow);
  }
}

// Per-CTA hit counts per plane (shared memory), added to the global counts
// when the CTA ends.
struct EmitBuf {
  unsigned pc[kMaxPlanes];  // hits per plane of this CTA
};

// Persistent harmonic summing.  Work item = (256-bin block, sign half),
// handed out dynamically through a global counter.  A CTA has NW consumer
// warps -- warp w owns templates |t| = 4w + k (k < 4), lane l the bins
// f0 + 4 l + c and f0 + 128 + 4 l + c (c < 4), i.e. a 4 x 8 tile of cells --
// and one producer warp.  For every item the producer issues one 2-D TMA
// tensor copy per plane (cp.async.bulk.tensor.2d): plane 1 as 256 bins x 4 NW
// rows, plane j >= 2 as the rows trunc(t/j) of the half over bins
// [(f0/j) & ~3, ...); rows and bins outside the FOP are zero-filled by the
// hardware (they only feed masked cells).  kHsStages stages deep: full / empty
// mbarriers, every wait bounded by %globaltimer.
//
// In the bounds planes 2, 4, 8 and 16 read their values with 8- and 4-byte loads at
// compile-time offsets, the others at offsets from products by 16-bit reciprocals;
// in the sums of a whole tile the eight bins of a lane map onto offsets from two
// divisions per plane, and the four rows onto two staged rows split at a
// warp-uniform point.
//
// HP_1 = FOP[t][f], HP_j = HP_{j-1} + FOP[trunc(t/j)][f/j] accumulated in FP32
// in this order -- hsum.py:95-120 / hms_baseline.cl.mako:55-84 -- so the
// values match hsum.py bit for bit for the same FOP.  A cell is a candidate of
// plane j if HP_j > thr_j (strict, hsum.py:134 / detect.cl.mako:185).
//
// The warps first look at upper bounds of the sums of their lanes' 4 x 4 cell
// groups only; where no group's bound reaches a plane's band the item is done.
// A few groups that do are summed one cell per lane (hs_few_groups); for more,
// the warp sums its whole tile and emits at the planes that some bound reached
// (hs_emit_item), which searches with many hits spend their time on: 2^20 bins x 85
// rows x 8 planes with 0.1 / 0.3 / 1 / 10% of a plane above its threshold take 574 /
// 1183 / 1460 / 3000 us a stage, against 1399 / 1640 / 1850 / 3450 with up to eight
// few groups, a reservation per plane and the exact sums once more to mark the planes,
// and 928 / 1250 / 1650 / 3300 without bounds.  The exact sums
// of every cell cost 692 instructions per warp and item at about 5.6 clocks
// each, and so held a stage for longer than its copies take; with the bounds
// the copies set the pace.  Stage time (noise, with selection) at 2^21 bins x
// 85 rows x 8 planes, 2^20 x 85 x 16, 300007 x 43 x 16, 2^15 x 85 x 8: 141 /
// 110 / 37 / 12 us against 238 / 297 / 113 / 40 before the bounds, the block order below
// and the dependent launches; three strong signals at 2^21: 240 against 292.
constexpr int kHsHeader = 1536;  // bytes before the stages: barriers, parameters, items
struct HsItem {
  int f0, sgn, tlo;
};

__device__ __forceinline__ HsItem hs_item(const HsumParams &p, int it) {
  // items enumerate (block, half) over the enabled halves.  Slots of the block
  // order with o trailing one bits run down from the top of the lowest
  // nb / 2^o blocks, so blocks b, b / 2, b / 4, ... are staged at about the
  // same time and the sub-harmonic boxes of planes 2, 4, 8 (and 6 with 3) find
  // the lower blocks in L2: at 2^21 bins 141 us a stage on noise and 240 with
  // three strong signals, against 160 and 255 from the highest block down.
  // Each octave starts with its highest blocks: a signal's harmonic images
  // cover wider bin ranges at higher bins (plane j sums f/k for k <= j), so the
  // items that emit most are handed out early and light ones end the launch.
  const bool neg = p.tlo[0] <= p.half, pos = p.tlo[1] <= p.half;
  const int nb = (p.n_bins + kHsBins - 1) / kHsBins;
  int slot, halfsel;
  if (neg && pos) { slot = it >> 1; halfsel = it & 1; }
  else { slot = it; halfsel = pos ? 1 : 0; }
  const int o = __ffs(~slot) - 1;
  const int blk = (nb >> o) - 1 - (slot >> (o + 1));
  return HsItem{blk * kHsBins, halfsel ? 1 : -1, p.tlo[halfsel]};
}

__device__ __forceinline__ int hs_n_items(const HsumParams &p) {
  const int nb = (p.n_bins + kHsBins - 1) / kHsBins;
  return nb * ((p.tlo[0] <= p.half) + (p.tlo[1] <= p.half));
}

__device__ __forceinline__ float fmax3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_wait_parity(uint64_t *bar, uint32_t parity, long long timeout_ns) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = globaltimer_ns();
  while (!mbar_try_wait(bar, parity))
    if ((long long)(globaltimer_ns() - t0) > timeout_ns) return false;
  return true;
}
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, int x, int y, uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], "
      "[%4];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
      : "memory");
}

// smem row of staged row r (r = |t| or trunc(|t|/j)) in a box of bh rows: the
// boxes hold FOP rows in ascending order, i.e. reversed for the negative half
__device__ __forceinline__ int srow(int r, int bh, int sgn) { return sgn > 0 ? r : bh - 1 - r; }

// (a0, a1) += (b0, b1) as one packed FP32 pair instruction (add.rn.f32x2,
// sm_100 and later): each half is an ordinary round-to-nearest FP32 add, so
// the sums are the scalar ones bit for bit
__device__ __forceinline__ void add2(float &a0, float &a1, float b0, float b1) {
  unsigned long long a, b, d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(a) : "f"(a0), "f"(a1));
  asm("mov.b64 %0, {%1, %2};" : "=l"(b) : "f"(b0), "f"(b1));
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a0), "=f"(a1) : "l"(d));
}

// Plane 1 of the warp's tile: 4 templates x 8 bins; cells outside the
// item's rows or beyond n_bins are -inf (they never reach a threshold)
template <int NW>
__device__ __forceinline__ void hs_load_plane1(float (&acc)[4][8], const float *stage, const HsumParams &p,
                                               int f0, int sgn, int tlo, int t0, int F) {
  const int H = p.half;
  const float *r1 = stage + p.soff[1] + (F - f0);
#pragma unroll
  for (int kk = 0; kk < 4; ++kk) {
    const float *rr = r1 + srow(t0 + kk, 4 * NW, sgn) * kHsBins;
    const float4 q0 = *reinterpret_cast<const float4 *>(rr);
    const float4 q1 = *reinterpret_cast<const float4 *>(rr + 128);
    acc[kk][0] = q0.x; acc[kk][1] = q0.y; acc[kk][2] = q0.z; acc[kk][3] = q0.w;
    acc[kk][4] = q1.x; acc[kk][5] = q1.y; acc[kk][6] = q1.z; acc[kk][7] = q1.w;
    if (!((t0 + kk <= H) && (t0 + kk >= tlo))) {
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[kk][e] = -CUDART_INF_F;
    }
  }
  if (f0 + kHsBins > p.n_bins) {
#pragma unroll
    for (int kk = 0; kk < 4; ++kk)
#pragma unroll
      for (int e = 0; e < 8; ++e)
        if (F + (e & 3) + ((e >> 2) << 7) >= p.n_bins) acc[kk][e] = -CUDART_INF_F;
  }
}

// Plane j >= 2 added for any j given at run time: the same values in the same
// order as the kernel's specialised per-plane code, so the sums are the same
// bit for bit
__device__ __forceinline__ void hs_add_plane_any(float (&acc)[4][8], const float *stage, const HsumParams &p,
                                                 int j, int f0, int sgn, int t0, int F) {
  const int a0 = (f0 / j) & ~3;
  const int bw = p.bw[j];
  const int rb = t0 / j;
  const int kstar = j - (t0 - rb * j);  // first k with trunc((t0+k)/j) = rb + 1
  const float *r0 = stage + p.soff[j] + srow(rb, p.bh[j], sgn) * bw - a0;
  const float *r1 = r0 + sgn * bw;
  // (F + c) / j = qa + [ra + c >= j] + [ra + c >= 2 j] for c < 4 <= 2 j
  const int qa = F / j, ra = F - qa * j;
  const int qb = (F + 128) / j, rg = F + 128 - qb * j;
  float c0[8], c1[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const int r = (e < 4 ? ra : rg) + (e & 3);
    const int o = (e < 4 ? qa : qb) + (r >= j ? 1 : 0) + (r >= 2 * j ? 1 : 0);
    c0[e] = r0[o];
    c1[e] = kstar < 4 ? r1[o] : 0.f;
  }
#pragma unroll
  for (int kk = 0; kk < 4; ++kk)
#pragma unroll
    for (int e = 0; e < 8; e += 2) {
      const bool second = kk >= kstar;
      add2(acc[kk][e], acc[kk][e + 1], second ? c1[e] : c0[e], second ? c1[e + 1] : c0[e + 1]);
    }
}

// The lanes' cells of `mask` (bit c = cell 8 k + e: template |t| = t0 + k,
// bin F + (e & 3) + 128 (e >> 2)) get consecutive slots from `pos`, cell by
// cell, so every store instruction of the warp writes one contiguous run
template <typename Put>
__device__ __forceinline__ void hs_scatter(const float (&acc)[4][8], unsigned mask, unsigned pos, int row0, int sgn,
                                           int F, Put &&put) {
  const unsigned below = (1u << (threadIdx.x & 31)) - 1u;
#pragma unroll
  for (int c = 0; c < 32; ++c) {
    const unsigned m = __ballot_sync(0xffffffffu, (mask >> c) & 1u);
    if (m) {
      if ((mask >> c) & 1u)
        put(pos + __popc(m & below), acc[c >> 3][c & 7], row0 + sgn * (c >> 3), F + (c & 3) + (((c >> 2) & 1) << 7));
      pos += __popc(m);
    }
  }
}

// Hits of plane `plane` (0-based) to the global list -- one reservation for
// the warp -- and cells within the band to the FP64 recheck list
__device__ __forceinline__ void hs_emit_plane(const float (&acc)[4][8], const HsumParams &p, EmitBuf *eb, int plane,
                                              int row0, int sgn, int F) {
  const int lane = threadIdx.x & 31;
  const float hi = p.hi[plane], lo = p.lo[plane];
  unsigned hmask = 0, nmask = 0;
#pragma unroll
  for (int c = 0; c < 32; ++c) {
    const float a = acc[c >> 3][c & 7];
    if (a > hi) hmask |= 1u << c;
    else if (a >= lo) nmask |= 1u << c;
  }
  const unsigned nall = __reduce_add_sync(0xffffffffu, (unsigned)__popc(nmask));
  if (nall) {
    unsigned base = 0;
    if (lane == 0) base = atomicAdd(p.rc_count, nall);
    uint4 *list = p.rc_list;
    const unsigned cap = (unsigned)p.rc_cap;
    int *status = p.status;
    hs_scatter(acc, nmask, __shfl_sync(0xffffffffu, base, 0), row0, sgn, F, [&](unsigned g, float, int row, int bin) {
      if (g < cap) list[g] = make_uint4((unsigned)plane, (unsigned)row, (unsigned)bin, 0u);
      else atomicOr(status, kStatusRecheckOverflow);
    });
  }
  const unsigned total = __reduce_add_sync(0xffffffffu, (unsigned)__popc(hmask));
  if (total) {
    unsigned base = 0;
    if (lane == 0) base = atomicAdd(p.cand_total, total);
    base = __shfl_sync(0xffffffffu, base, 0);
    unsigned long long *keys = p.cand_key;
    float *pwrs = p.cand_pwr;
    const unsigned cap = (unsigned)p.cand_cap;
    hs_scatter(acc, hmask, base, row0, sgn, F, [&](unsigned g, float v, int row, int bin) {
      if (g < cap) {
        keys[g] = cand_key(plane, row, bin);
        pwrs[g] = v;
      }
    });
    if (lane == 0) {
      atomicAdd(&eb->pc[plane], total);
      if (base + total > cap) atomicOr(p.status, kStatusCandidateOverflow);
    }
  }
}

// Emission for one item (rare; the warp calls it together, before it releases
// the stage): the sums are recomputed plane by plane from the staged boxes
// and the planes marked in `need` (bit j - 1) are emitted.
template <int NW>
__device__ __forceinline__ void hs_emit_item_body(const HsumParams &p, const float *stage, EmitBuf *eb, int f0,
                                                  int sgn, int tlo, int t0, unsigned need) {
  const int F = f0 + 4 * (threadIdx.x & 31);
  const int row0 = p.half + sgn * t0;
  float acc[4][8];
  hs_load_plane1<NW>(acc, stage, p, f0, sgn, tlo, t0, F);
#pragma unroll 1
  for (int j = 1; j <= p.n_planes; ++j) {
    if (j > 1) hs_add_plane_any(acc, stage, p, j, f0, sgn, t0, F);
    if ((need >> (j - 1)) & 1u) hs_emit_plane(acc, p, eb, j - 1, row0, sgn, F);
    if (!(need >> j)) break;
  }
}

// The same out of line (the hot loop keeps its code and registers); `pp` is
// the CTA's shared-memory copy of the parameters.  Used where registers are
// plentiful: at the lean variant's 80 registers the call's saves would spill
// in the hot loop, so that variant inlines the body.
template <int NW>
__device__ __noinline__ void hs_emit_item(const HsumParams *pp, const float *stage, EmitBuf *eb, int f0, int sgn,
                                          int tlo, int t0, unsigned need) {
  hs_emit_item_body<NW>(*pp, stage, eb, f0, sgn, tlo, t0, need);
}

// Where a warp's four rows lie in the staged box of plane j: float offset in the
// stage of the first row trunc(t0 / j) and, in the upper half-word, of the last,
// trunc((t0 + 3) / j) (the rows in between are one of the two).
template <int NW>
__device__ __forceinline__ unsigned hs_row_offsets(const HsumParams &p, int j, int t0, int sgn) {
  if (j == 1) return (unsigned)(sgn > 0 ? t0 : 4 * NW - 4 - t0) * kHsBins;
  const int a = srow(t0 / j, p.bh[j], sgn), b = srow((t0 + 3) / j, p.bh[j], sgn);
  return (unsigned)(p.soff[j] + a * p.bw[j]) | (unsigned)(p.soff[j] + b * p.bw[j]) << 16;
}

// Upper bounds of the sums in the lane's two 4 x 4 cell groups: per plane the
// largest value any of a group's cells adds.  Rounded addition is monotone, so
// a bound below a plane's band leaves no cell of the group in it -- which
// settles 98% of the warps on noise at 8 planes with a third of the instructions
// that every cell's own sums take.
struct HsBounds {
  float a, b;
  unsigned hit_a, hit_b;  // planes (bit j - 1) whose band the bound reaches
};
__device__ __forceinline__ float fmax4(float4 v) { return fmaxf(fmax3(v.x, v.y, v.z), v.w); }
__device__ __forceinline__ void hs_bound_plane1(HsBounds &u, const float *stage, unsigned row, float trig, int lane) {
  const float4 *r = reinterpret_cast<const float4 *>(stage + row) + lane;
  const float4 a0 = r[0], a1 = r[kHsBins / 4], a2 = r[2 * (kHsBins / 4)], a3 = r[3 * (kHsBins / 4)];
  const float4 b0 = r[32], b1 = r[kHsBins / 4 + 32], b2 = r[2 * (kHsBins / 4) + 32], b3 = r[3 * (kHsBins / 4) + 32];
  u.a = fmaxf(fmax3(fmax4(a0), fmax4(a1), fmax4(a2)), fmax4(a3));
  u.b = fmaxf(fmax3(fmax4(b0), fmax4(b1), fmax4(b2)), fmax4(b3));
  u.hit_a = u.a >= trig ? 1u : 0u;
  u.hit_b = u.b >= trig ? 1u : 0u;
}
// `where`: f0 mod j | (f0 / j - box start) << 8
template <int j>
__device__ __forceinline__ void hs_bound_plane(HsBounds &u, const float *stage, unsigned rows, int where, float trig,
                                               int lane) {
  const unsigned r0 = rows & 0xffffu, r1 = rows >> 16;
  if constexpr (j == 2) {
    const float2 *q0 = reinterpret_cast<const float2 *>(stage + r0) + lane;
    const float2 *q1 = reinterpret_cast<const float2 *>(stage + r1) + lane;
    const float2 a0 = q0[0], b0 = q0[32], a1 = q1[0], b1 = q1[32];
    u.a += fmaxf(fmax3(a0.x, a0.y, a1.x), a1.y);
    u.b += fmaxf(fmax3(b0.x, b0.y, b1.x), b1.y);
  } else if constexpr (hs_one_value(j)) {  // one value for the group
    const float *q = stage + r0 + lane / (j / 4);
    u.a += q[0];
    u.b += q[128 / j];
  } else {
    // bins F .. F + 3 take at most two values, at F / j and (F + 3) / j; numbers
    // below 300 divided by j <= 16 by a 16-bit reciprocal, exactly
    constexpr unsigned M = 65536u / j + 1;
    const unsigned x = (unsigned)(where & 0xff) + 4u * lane, o = (unsigned)where >> 8;
    const unsigned qa = (x * M) >> 16, ha = ((x + 3) * M) >> 16;
    const unsigned qb = ((x + 128) * M) >> 16, hb = ((x + 131) * M) >> 16;
    const float *s0 = stage + r0 + o, *s1 = stage + r1 + o;
    u.a += fmaxf(fmax3(s0[qa], s0[ha], s1[qa]), s1[ha]);
    u.b += fmaxf(fmax3(s0[qb], s0[hb], s1[qb]), s1[hb]);
  }
  if (u.a >= trig) u.hit_a |= 1u << (j - 1);
  if (u.b >= trig) u.hit_b |= 1u << (j - 1);
}

// The cells of a few 4 x 4 groups (bit l of hit_a / hit_b: lane l's group of
// the first / second half of the bins), one cell per lane and two groups at a
// time: their sums, and the hits and near-threshold cells among them.  On noise
// a warp that does not pass on its bounds has one or two such groups, so this
// is a fifth of the work of the whole tile's exact sums.  One reservation in the list
// serves all planes of the two groups (one per plane: 2^17 bins x 85 x 8 with 0.1% of
// the cells above the threshold 270 us a stage, 244 so).  Up to 16 groups: with eight
// 0.1 / 0.3% take 895 / 1128 us a stage at 2^20 bins x 85 x 8 against 574 / 1183, and
// three strong signals the same.
constexpr int kHsFewGroups = 16;
template <int MAXP, int NW>
__device__ __forceinline__ void hs_few_groups(const HsumParams &p, const float *stage, EmitBuf *eb, int f0, int sgn,
                                              int tlo, int t0, unsigned hit_a, unsigned hit_b) {
  const int lane = threadIdx.x & 31;
  unsigned long long todo = (unsigned long long)hit_b << 32 | hit_a;
#pragma unroll 1
  while (todo) {
    int grp = __ffsll(todo) - 1;
    todo &= todo - 1;
    bool live = true;
    if (lane >= 16) {  // the upper half-warp takes the next group, if there is one
      live = todo != 0;
      grp = live ? __ffsll(todo) - 1 : grp;
    }
    todo &= todo - 1;  // (0 stays 0)
    const int t = t0 + ((lane >> 2) & 3), off = 4 * (grp & 31) + (grp & 32) * 4 + (lane & 3);
    live = live && t <= p.half && t >= tlo && f0 + off < p.n_bins;
    float hp[MAXP];
    hp[0] = stage[p.soff[1] + srow(t, 4 * NW, sgn) * kHsBins + off];
    hs_sfor<MAXP - 1>([&](auto JJ) {
      constexpr int j = decltype(JJ)::value + 2;
      if (j <= p.n_planes) {
        const int a0 = (f0 / j) & ~3;
        hp[j - 1] = stage[p.soff[j] + srow(t / j, p.bh[j], sgn) * p.bw[j] + (f0 + off) / j - a0];
      }
    });
    unsigned hits = 0, near = 0;
    hs_sfor<MAXP>([&](auto JJ) {
      constexpr int i = decltype(JJ)::value;
      if (i < p.n_planes) {
        if constexpr (i > 0) hp[i] = hp[i - 1] + hp[i];
        if (hp[i] > p.hi[i]) hits |= 1u << i;
        else if (hp[i] >= p.lo[i]) near |= 1u << i;
      }
    });
    if (!live) hits = near = 0;
    const int row = p.half + sgn * t, bin = f0 + off;
    const unsigned below = (1u << lane) - 1u;
    // one reservation for the hits of all planes, stored plane by plane
    const unsigned total = __reduce_add_sync(0xffffffffu, (unsigned)__popc(hits));
    if (total) {
      unsigned base = 0;
      if (lane == 0) {
        base = atomicAdd(p.cand_total, total);
        if (base + total > (unsigned)p.cand_cap) atomicOr(p.status, kStatusCandidateOverflow);
      }
      unsigned at = __shfl_sync(0xffffffffu, base, 0);
      hs_sfor<MAXP>([&](auto JJ) {
        constexpr int i = decltype(JJ)::value;
        if (i < p.n_planes) {
          const unsigned mh = __ballot_sync(0xffffffffu, (hits >> i) & 1u);
          const unsigned g = at + __popc(mh & below);
          if (((hits >> i) & 1u) && g < (unsigned)p.cand_cap) {
            p.cand_key[g] = cand_key(i, row, bin);
            p.cand_pwr[g] = hp[i];
          }
          if (mh && lane == 0) atomicAdd(&eb->pc[i], (unsigned)__popc(mh));
          at += __popc(mh);
        }
      });
    }
    if (__any_sync(0xffffffffu, near)) {
      hs_sfor<MAXP>([&](auto JJ) {
        constexpr int i = decltype(JJ)::value;
        if (i < p.n_planes) {
          const unsigned mn = __ballot_sync(0xffffffffu, (near >> i) & 1u);
          if (mn) {
            unsigned base = 0;
            if (lane == 0) base = atomicAdd(p.rc_count, (unsigned)__popc(mn));
            const unsigned g = __shfl_sync(0xffffffffu, base, 0) + __popc(mn & below);
            if ((near >> i) & 1u) {
              if (g < (unsigned)p.rc_cap) p.rc_list[g] = make_uint4((unsigned)i, (unsigned)row, (unsigned)bin, 0u);
              else atomicOr(p.status, kStatusRecheckOverflow);
            }
          }
        }
      });
    }
  }
}
// NW consumer warps cover the rows of a half, 4 each: 16 for banks above 87
// rows, 11 above 47, else 6, whose stages are half as large so that five fit
// (2^21 bins x 43 rows x 8 planes 133 us a stage against 155 with 11 warps and
// 44-row boxes, 300007 x 43 x 16 64 against 71; a second group of 6 warps
// taking every other stage changed neither).
template <int MAXP, int NW, int kHsStages, int MINB>
__global__ void __launch_bounds__(32 * (NW + 1), MINB) hsum_kernel(const __grid_constant__ HsumParams p,
                                                                    const __grid_constant__ HsumMaps m) {
  extern __shared__ __align__(1024) float hs_smem[];
  // per stage: `full` completes when the plane-1 box has landed, `full2` when
  // the sub-harmonic boxes have, so the consumers start on plane 1 while the
  // rest of the stage is still arriving
  uint64_t *full = reinterpret_cast<uint64_t *>(hs_smem);  // [kHsStages]
  uint64_t *full2 = full + kHsStages;                        // [kHsStages]
  uint64_t *empty = full2 + kHsStages;                       // [kHsStages]
  HsumParams *sp = reinterpret_cast<HsumParams *>(hs_smem + 32);  // copy for the emitter
  // per stage: [0] f0 of the item (-1: stop mark), [1] 2 tlo + (positive half),
  // [j] f0 mod j | (f0 / j - start of the staged bins) << 8
  int *item_at = reinterpret_cast<int *>(hs_smem + 200);  // [kHsStages][kItemWords]
  constexpr int kItemWords = MAXP + 1;
  float *stages = hs_smem + kHsHeader / 4;
  EmitBuf &eb = *reinterpret_cast<EmitBuf *>(stages + kHsStages * p.stage_floats);
  unsigned *rows = reinterpret_cast<unsigned *>(&eb + 1);  // [NW][half][kMaxPlanes + 1]: hs_row_offsets
  constexpr int kRows1 = 4 * NW;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int H = p.half;
  const int P = p.n_planes;
  const int n_items = hs_n_items(p);

  if (threadIdx.x == 0) {
    for (int s = 0; s < kHsStages; ++s) {
      mbar_init(full + s, 1);
      mbar_init(full2 + s, 1);
      mbar_init(empty + s, NW);
    }
    fence_mbar_init();
  }
  if (threadIdx.x < kMaxPlanes) eb.pc[threadIdx.x] = 0;
  static_assert(sizeof(HsumParams) % 4 == 0 && 128 + sizeof(HsumParams) <= 800, "header holds the parameters");
  static_assert(kHsStages * 3 * 8 <= 128 && 800 + kHsStages * kItemWords * 4 <= kHsHeader, "barriers and items in the header");
  for (int i = threadIdx.x; i < (int)(sizeof(HsumParams) / 4); i += blockDim.x)
    reinterpret_cast<int *>(sp)[i] = reinterpret_cast<const int *>(&p)[i];
  for (int i = threadIdx.x; i < NW * 2 * (kMaxPlanes + 1); i += blockDim.x) {
    const int j = i % (kMaxPlanes + 1), wh = i / (kMaxPlanes + 1);
    rows[i] = j >= 1 && j <= P ? hs_row_offsets<NW>(p, j, 4 * (wh >> 1), wh & 1 ? 1 : -1) : 0u;
  }
  grid_release();
  grid_wait();
  stamp_if_none(p.stamp);
  __syncthreads();

  if (warp == NW) {
    // ------------------------------------------------------------ producer
    if (lane == 0) {
      // The first item is the CTA's own index, the others come from the global
      // counter, requested ahead: two at a time (the halves of a block) while
      // there are plenty, so that an atomic, which takes about as long as an
      // item of a small bank, is out for two items; one at a time towards the
      // end, which keeps it even.  2^21 bins x 43 rows: 134 us a stage against
      // 147 one at a time; four at a time 131, but 263 against 245 where
      // signals make neighbouring items slow (85 rows, three strong signals).
      const int grid = gridDim.x;
      int cur = blockIdx.x, cur_n = 1, used = 0;
      auto request = [&](int seen, int &n) {
        n = seen + 8 * grid < n_items ? 2 : 1;
        return grid + (int)atomicAdd(p.item_counter, (unsigned)n);
      };
      int nxt_n, nxt = request(cur, nxt_n);
      // per stage: the use whose copies may still be in flight (-1: none).  A
      // stage's copies have landed once the consumers released it.
      int pending[kHsStages];
#pragma unroll
      for (int q = 0; q < kHsStages; ++q) pending[q] = -1;
      for (int s = 0;; ++s) {
        const int st = s % kHsStages, use = s / kHsStages;
        if (use >= 1 && !mbar_wait_parity(empty + st, (use - 1) & 1, p.timeout_ns)) {
          atomicOr(p.status, kStatusHsumTimeout);
          // let every copy in flight land (bounded), so that the stop mark
          // below arrives on a completed phase and no copy outlives the CTA
          bool drained = true;
#pragma unroll
          for (int q = 0; q < kHsStages; ++q)
            if (pending[q] >= 0) {
              drained &= mbar_wait_parity(full + q, pending[q] & 1, kDrainNs);
              drained &= mbar_wait_parity(full2 + q, pending[q] & 1, kDrainNs);
              pending[q] = -1;
            }
          // (a stage the test hook announced without copies has a phase that
          // never completes: no stop mark on it -- its consumers have left)
          if (drained && !(p.inject_stall && st == 0)) {
            item_at[st * kItemWords] = -1;
            mbar_arrive(full + st);
          }
          break;
        }
#pragma unroll
        for (int q = 0; q < kHsStages; ++q)
          if (q == st) pending[q] = -1;  // released by the consumers: its copies have landed
        if (used == cur_n) {
          cur = nxt;
          cur_n = nxt_n;
          used = 0;
          if (cur < n_items) nxt = request(cur, nxt_n);
        }
        const int it = cur + used++;
        if (it >= n_items) {
          item_at[st * kItemWords] = -1;
          mbar_arrive(full + st);  // plain arrival: the stage carries the stop mark
          break;
        }
        const HsItem item = hs_item(p, it);
        int *at = item_at + st * kItemWords;
        at[0] = item.f0;
        at[1] = 2 * item.tlo + (item.sgn > 0);
        hs_sfor<MAXP - 1>([&](auto JJ) {  // j known at compile time: divisions by constants
          constexpr int j = decltype(JJ)::value + 2;
          const int q = item.f0 / j;
          at[j] = (item.f0 - q * j) | (q & 3) << 8;
        });
        const unsigned bytes1 = (unsigned)(p.bw[1] * p.bh[1]) * 4u;
        if (p.inject_stall && s == 0) {  // test hook: announced, never issued -- nothing in flight
          mbar_arrive_expect_tx(full + st, bytes1);
          mbar_arrive_expect_tx(full2 + st, p.stage_bytes - bytes1 + 16u);
          continue;
        }
#pragma unroll
        for (int q = 0; q < kHsStages; ++q)
          if (q == st) pending[q] = use;
        float *stage = stages + st * p.stage_floats;
        mbar_arrive_expect_tx(full + st, bytes1);
        tma_load_2d(stage + p.soff[1], &m.map[1], item.f0, item.sgn > 0 ? H : H - (kRows1 - 1), full + st);
        mbar_arrive_expect_tx(full2 + st, p.stage_bytes - bytes1);  // 0 bytes with one plane: a plain arrival
        hs_sfor<MAXP - 1>([&](auto JJ) {  // j known at compile time: divisions by constants
          constexpr int j = decltype(JJ)::value + 2;
          if (j <= P) {
            const int a0 = (item.f0 / j) & ~3;
            tma_load_2d(stage + p.soff[j], &m.map[j], a0, item.sgn > 0 ? H : H - (p.bh[j] - 1), full2 + st);
          }
        });
      }
      // consumers that stopped on a timeout leave stages unconsumed: their
      // copies land before the CTA ends (returns at once when they have)
#pragma unroll
      for (int q = 0; q < kHsStages; ++q)
        if (pending[q] >= 0) {
          mbar_wait_parity(full + q, pending[q] & 1, kDrainNs);
          mbar_wait_parity(full2 + q, pending[q] & 1, kDrainNs);
        }
    }
  } else {
    // ------------------------------------------------------------ consumers
    const int t0 = 4 * warp;
    const unsigned *my_rows = rows + warp * 2 * (kMaxPlanes + 1);
    for (int s = 0;; ++s) {
      const int st = s % kHsStages, use = s / kHsStages;
      if (!mbar_wait_parity(full + st, use & 1, p.timeout_ns)) {
        if (lane == 0) atomicOr(p.status, kStatusHsumTimeout);
        break;
      }
      const int *at = item_at + st * kItemWords;
      const int f0 = at[0];
      if (f0 < 0) break;
      const int sgn = (at[1] & 1) ? 1 : -1, tlo = at[1] >> 1;
      const float *stage = stages + st * p.stage_floats;
      HsBounds u;
      const unsigned *rj = my_rows + (sgn > 0 ? kMaxPlanes + 1 : 0);
      hs_bound_plane1(u, stage, rj[1], p.trig[0], lane);
      if (!mbar_wait_parity(full2 + st, use & 1, p.timeout_ns)) {
        if (lane == 0) atomicOr(p.status, kStatusHsumTimeout);
        break;
      }
      hs_sfor<MAXP - 1>([&](auto JJ) {
        constexpr int j = decltype(JJ)::value + 2;
        if (j <= P)
          hs_bound_plane<j>(u, stage, rj[j], at[j], p.trig[j - 1], lane);
      });
      const unsigned hit_a = __ballot_sync(0xffffffffu, u.hit_a != 0), hit_b = __ballot_sync(0xffffffffu, u.hit_b != 0);
      if (hit_a | hit_b) {
        if (__popc(hit_a) + __popc(hit_b) <= kHsFewGroups) {
          hs_few_groups<MAXP, NW>(p, stage, &eb, f0, sgn, tlo, t0, hit_a, hit_b);
        } else {
          const unsigned need = __reduce_or_sync(0xffffffffu, u.hit_a | u.hit_b);
          if constexpr (MINB >= 2) hs_emit_item_body<NW>(p, stage, &eb, f0, sgn, tlo, t0, need);
          else hs_emit_item<NW>(sp, stage, &eb, f0, sgn, tlo, t0, need);
        }
      }

      // release the stage to the producer
      __syncwarp();
      if (lane == 0) mbar_arrive(empty + st);
    }
  }

  // ---- per-plane hit counts of the CTA
  __syncthreads();
  if (threadIdx.x < P && eb.pc[threadIdx.x]) atomicAdd(p.cand_count + threadIdx.x, eb.pc[threadIdx.x]);
}

constexpr int kSelUnroll = 4;  // records per thread in flight in the selection passes
constexpr int kRcUnroll = 8;   // taps per lane in flight in the FP64 recheck

// FP64 taps -> float pairs in place: (re hi, im hi, re lo, im lo) with
// hi = fl32(c), lo = fl32(c - hi), so c = hi + lo to 2^-48 relative.  The
// recheck then forms its products on the FP32 pipe; GB300's FP64 rate is
// about 1/64 of its FP32 rate.
__global__ void split_taps_kernel(double2 *taps, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const double2 c = taps[i];
    const float hr = __double2float_rn(c.x), hm = __double2float_rn(c.y);
    const float lr = __double2float_rn(c.x - (double)hr), lm = __double2float_rn(c.y - (double)hm);
    reinterpret_cast<float4 *>(taps)[i] = make_float4(hr, hm, lr, lm);
  }
}

// (s, t) += a (bh + bl) in double-float arithmetic: a bh = p + pe exactly
// (FMA), s + p = u + e exactly (Knuth's two-sum), the small terms gathered in
// t.  Rounded intrinsics keep the compiler from fusing the error-free steps.
__device__ __forceinline__ void df_add_prod(float &s, float &t, float a, float bh, float bl) {
  const float pr = __fmul_rn(a, bh);
  const float pe = fmaf(a, bh, -pr);
  const float u = __fadd_rn(s, pr);
  const float bb = __fsub_rn(u, s);
  const float e = __fadd_rn(__fsub_rn(s, __fsub_rn(u, bb)), __fsub_rn(pr, bb));
  t = __fadd_rn(t, __fadd_rn(e, fmaf(a, bl, pe)));
  s = u;
}

// FP64-grade recheck: a CTA per entry (grid-stride), warp j computes the FOP
// cell FOP(trunc(t/(j+1)), bin/(j+1)) = |sum_q X[g - q] h_r[q]|^2
// (ft_conv.py:201-205) with its lanes over the taps -- per lane in
// double-float arithmetic (about 2^-44 relative), then in FP64 across the
// lanes; warp 0 sums the planes in order j = 1..k (hsum.py:95-120) in FP64
// and compares with the threshold.  A noise-like search has a handful of entries, so
// the launch lasts as long as one of them: a warp for each plane, 16 above 8 planes
// (8 warps took two turns: harmonic-summing stage of 2^20 bins x 16 planes 134.3 ->
// 129.5 us, of 300007 bins x 43 rows 52.0 -> 51.1).  Up to 8 planes half of those
// would be idle, and an SM holds three CTAs of 8 warps but one of 16: 413 entries
// (2^21 bins, three strong signals) 10.6 against 14.6 us.  (32 warps per SM are launched,
// four CTAs of 8 or two of 16: what is not resident at once follows as others end.)
__global__ void __launch_bounds__(512) recheck_kernel(RecheckParams p) {
  __shared__ double cell[kMaxPlanes];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nwarps = blockDim.x >> 5;
  grid_release();
  grid_wait();
  const unsigned n = min(*p.rc_count, (unsigned)p.rc_cap);
  for (unsigned e = blockIdx.x; e < n; e += gridDim.x) {
    const uint4 ent = p.rc_list[e];
    const int plane = (int)ent.x, row = (int)ent.y, bin = (int)ent.z;
    const int t = row - p.half;
    for (int j = warp + 1; j <= plane + 1; j += nwarps) {
      const int tj = (t >= 0) ? t / j : -((-t) / j);
      const int r = p.half + tj;
      const int g = bin / j;
      const int qn = min(p.tap_len[r], g + 1);
      const float4 *h = p.taps + (long long)r * p.tap_pitch;
      float rs = 0.f, rt = 0.f, is = 0.f, it = 0.f;  // double-float sums of re and im
      // taps q = lane + 32 u in ascending order; the loads of a pass are all
      // issued before the arithmetic, so one memory latency covers 256 taps
      for (int q0 = 0; q0 < qn; q0 += 32 * kRcUnroll) {
        float2 x[kRcUnroll];
        float4 c[kRcUnroll];
#pragma unroll
        for (int u = 0; u < kRcUnroll; ++u) {
          const int q = q0 + lane + 32 * u;
          x[u] = q < qn ? p.input[g - q] : make_float2(0.f, 0.f);
          c[u] = q < qn ? h[q] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int u = 0; u < kRcUnroll; ++u) {
          if (q0 + lane + 32 * u < qn) {
            // re += x.re c.re - x.im c.im, im += x.re c.im + x.im c.re
            df_add_prod(rs, rt, x[u].x, c[u].x, c[u].z);
            df_add_prod(rs, rt, -x[u].y, c[u].y, c[u].w);
            df_add_prod(is, it, x[u].x, c[u].y, c[u].w);
            df_add_prod(is, it, x[u].y, c[u].x, c[u].z);
          }
        }
      }
      double re = (double)rs + (double)rt, im = (double)is + (double)it;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        re += __shfl_xor_sync(0xffffffffu, re, o);
        im += __shfl_xor_sync(0xffffffffu, im, o);
      }
      if (lane == 0) cell[j - 1] = re * re + im * im;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      double hp = 0.0;
      for (int j = 0; j <= plane; ++j) hp += cell[j];
      if (hp > p.thr[plane]) {
        atomicAdd(p.cand_count + plane, 1u);
        global_append(p.cand_key, p.cand_pwr, p.cand_total, p.cand_cap, p.status, cand_key(plane, row, bin),
                      (float)hp);
      }
    }
    __syncthreads();
  }
}

// ------------------------------------------- deterministic top-K per plane
// The fixed-size list keeps, per plane, the K strongest hits (power
// descending, location ascending on ties) in location order.  Hits are stored
// unordered by the harmonic-summing kernel.  Selection: a histogram of each
// plane's powers over 2048 buckets (float bits 30..20, powers are >= 0) built
// in shared memory per CTA; the last CTA finds the bucket where the count from
// the top reaches K; the records above it ("sure") and in it ("boundary") are
// gathered; kFinSlices CTAs per plane each rank the boundary records and then
// order their slice of the kept ones by location, both by direct rank
// computation.

__device__ __forceinline__ int pwr_bucket(float pw) { return (int)((__float_as_uint(pw) >> 20) & 0x7ffu); }

__global__ void __launch_bounds__(1024) select_hist_kernel(SelectParams p) {
  extern __shared__ unsigned sh_hist[];  // [n_planes][kSelBuckets]
  __shared__ bool last;
  __shared__ bool over[kMaxPlanes];  // plane has more hits than K
  __shared__ int n_over;
  const int nb = p.n_planes * kSelBuckets;
  grid_release();
  grid_wait();
  if (threadIdx.x == 0) n_over = 0;
  __syncthreads();
  if (threadIdx.x < kMaxPlanes) {
    over[threadIdx.x] = threadIdx.x < p.n_planes && p.cand_count[threadIdx.x] > (unsigned)p.per_plane;
    if (over[threadIdx.x]) atomicAdd(&n_over, 1);
  }
  __syncthreads();
  if (n_over == 0) {
    // every plane keeps all its hits: no histogram, no boundary bucket (the
    // counts are final, so every CTA takes this branch)
    if (blockIdx.x == 0 && threadIdx.x < p.n_planes) p.sel_bucket[threadIdx.x] = -1;
    return;
  }
  for (int i = threadIdx.x; i < nb; i += blockDim.x) sh_hist[i] = 0u;
  __syncthreads();
  const unsigned n = min(*p.cand_total, (unsigned)p.cand_cap);
  // warp-uniform loop, kSelUnroll records per lane in flight; lanes that hit
  // the same (plane, bucket) -- common, since a signal's hits have similar
  // powers -- add once, through their leader
  const unsigned ln = threadIdx.x & 31;
  const unsigned stride = gridDim.x * blockDim.x;
  for (unsigned base = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < n; base += kSelUnroll * stride) {
    unsigned long long k[kSelUnroll];
    float w[kSelUnroll];
#pragma unroll
    for (int u = 0; u < kSelUnroll; ++u) {
      const unsigned i = base + u * stride + ln;
      k[u] = i < n ? p.cand_key[i] : ~0ull;
      w[u] = i < n ? p.cand_pwr[i] : 0.f;
    }
#pragma unroll
    for (int u = 0; u < kSelUnroll; ++u) {
      const int plane = (int)(k[u] >> 48);
      const unsigned slot = (k[u] != ~0ull && over[plane]) ? (unsigned)(plane * kSelBuckets + pwr_bucket(w[u]))
                                                            : 0xffffffffu;
      const unsigned peers = __match_any_sync(0xffffffffu, slot);
      if (slot != 0xffffffffu && ln == (unsigned)(__ffs(peers) - 1)) atomicAdd(sh_hist + slot, (unsigned)__popc(peers));
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < nb; i += blockDim.x)
    if (sh_hist[i]) atomicAdd(p.hist + i, sh_hist[i]);
  // the last CTA to finish picks the boundary bucket of every plane
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(p.ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  // the summed histograms into shared memory (one coalesced pass), so the
  // boundary search below is not a chain of dependent global loads
  for (int i = threadIdx.x; i < nb; i += blockDim.x) sh_hist[i] = __ldcg(p.hist + i);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp < p.n_planes) {
    const int plane = warp;
    const unsigned K = (unsigned)p.per_plane;
    if (!over[plane]) {
      if (lane == 0) p.sel_bucket[plane] = -1;
    } else {
      const unsigned *h = sh_hist + plane * kSelBuckets;
      // strongest first: chunk c covers buckets [2048 - 32 (c+1), 2048 - 32 c)
      unsigned above = 0;
      int found = -1;
      for (int c = 0; c < kSelBuckets / 32 && found < 0; ++c) {
        const int b = kSelBuckets - 1 - 32 * c - lane;
        unsigned v = h[b];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const unsigned u = __shfl_up_sync(0xffffffffu, v, o);
          if (lane >= o) v += u;
        }
        const unsigned hit = __ballot_sync(0xffffffffu, above + v >= K);
        if (hit) found = kSelBuckets - 1 - 32 * c - (__ffs(hit) - 1);
        else above += __shfl_sync(0xffffffffu, v, 31);
      }
      if (lane == 0) p.sel_bucket[plane] = found;  // -1: fewer stored than K (overflow), take all
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < nb; i += blockDim.x) p.hist[i] = 0u;
  if (threadIdx.x == 0) *p.ticket = 0u;
}

__global__ void __launch_bounds__(256) select_gather_kernel(SelectParams p) {
  __shared__ int sb_of[kMaxPlanes];
  grid_release();
  grid_wait();
  if (threadIdx.x < kMaxPlanes) sb_of[threadIdx.x] = threadIdx.x < p.n_planes ? p.sel_bucket[threadIdx.x] : -1;
  __syncthreads();
  const unsigned n = min(*p.cand_total, (unsigned)p.cand_cap);
  const unsigned stride = gridDim.x * blockDim.x;
  for (unsigned base = blockIdx.x * blockDim.x + threadIdx.x; base < n; base += kSelUnroll * stride) {
    unsigned long long k[kSelUnroll];
    float w[kSelUnroll];
#pragma unroll
    for (int u = 0; u < kSelUnroll; ++u) {
      const unsigned i = base + u * stride;
      k[u] = i < n ? p.cand_key[i] : ~0ull;
      w[u] = i < n ? p.cand_pwr[i] : 0.f;
    }
#pragma unroll
    for (int u = 0; u < kSelUnroll; ++u) {
      if (k[u] == ~0ull) continue;
      const unsigned long long key = k[u];
      const int plane = (int)(key >> 48);
      const float pw = w[u];
      if (const unsigned i = base + u * stride; i < p.n_host_rec) {
        p.host_key[i] = key;
        p.host_rec_pwr[i] = pw;
      }
      const int sb = sb_of[plane];
      const int b = pwr_bucket(pw);
      int list = -1;
      unsigned *cnt = nullptr;
      if (sb < 0 || b > sb) { list = 0; cnt = p.sure_count + plane; }
      else if (b == sb) { list = 1; cnt = p.bound_count + plane; }
      if (list >= 0) {
        const unsigned idx = atomicAdd(cnt, 1u);
        if (idx < (unsigned)kSortCap) {
          const size_t o = ((size_t)plane * 2 + list) * kSortCap + idx;
          p.sel_key[o] = key;
          p.sel_pwr[o] = pw;
        } else {
          atomicOr(p.status, kStatusSelectionOverflow);
        }
      }
    }
  }
}

// "a is stronger than b": power descending, key ascending on ties
__device__ __forceinline__ bool stronger(float pa, unsigned long long ka, float pb, unsigned long long kb) {
  return pa > pb || (pa == pb && ka < kb);
}

__global__ void __launch_bounds__(1024) select_finalize_kernel(SelectParams p) {
  extern __shared__ __align__(16) unsigned char fz_smem[];
  grid_wait();
  const int plane = blockIdx.x;
  const int K = p.per_plane;
  unsigned long long *bkey = reinterpret_cast<unsigned long long *>(fz_smem);  // [kSortCap] boundary
  float *bpwr = reinterpret_cast<float *>(bkey + kSortCap);
  unsigned long long *fin = reinterpret_cast<unsigned long long *>(bpwr + kSortCap);  // [kMaxCompat] kept
  float *finp = reinterpret_cast<float *>(fin + kMaxCompat);
  const int a = (int)min(p.sure_count[plane], (unsigned)kSortCap);
  const int b = (int)min(p.bound_count[plane], (unsigned)kSortCap);
  const size_t base = (size_t)plane * 2 * kSortCap;
  // the sure records are all kept (fewer than K unless every hit was taken)
  const int keep_a = min(a, K);
  for (int i = threadIdx.x; i < keep_a; i += blockDim.x) {
    fin[i] = p.sel_key[base + i];
    finp[i] = p.sel_pwr[base + i];
  }
  for (int i = threadIdx.x; i < b; i += blockDim.x) {
    bkey[i] = p.sel_key[base + kSortCap + i];
    bpwr[i] = p.sel_pwr[base + kSortCap + i];
  }
  __syncthreads();
  // boundary records: rank among themselves, keep the c strongest
  const int c = max(0, min(K - keep_a, b));
  for (int i = threadIdx.x; i < b; i += blockDim.x) {
    const unsigned long long ki = bkey[i];
    const float pi = bpwr[i];
    int rank = 0;
    for (int j = 0; j < b; ++j) rank += stronger(bpwr[j], bkey[j], pi, ki);
    if (rank < c) {
      fin[keep_a + rank] = ki;
      finp[keep_a + rank] = pi;
    }
  }
  __syncthreads();
  const int kept = keep_a + c;
  uint32_t *cl = p.compat_loc + (size_t)plane * K, *hl = p.host_loc + (size_t)plane * K,
           *ul = p.user_loc ? p.user_loc + (size_t)plane * K : nullptr;
  float *cp = p.compat_pwr + (size_t)plane * K, *hp = p.host_pwr + (size_t)plane * K,
        *up = p.user_pwr ? p.user_pwr + (size_t)plane * K : nullptr;
  auto put = [&](int at, uint32_t loc, float pwr) {
    cl[at] = loc;
    cp[at] = pwr;
    hl[at] = loc;
    hp[at] = pwr;
    if (ul) ul[at] = loc;
    if (up) up[at] = pwr;
  };
  // the control words are final: the kernels before have ended
  if (blockIdx.x == 0 && blockIdx.y == 0)
    for (int i = threadIdx.x; i < p.n_ctrl; i += blockDim.x) p.host_ctrl[i] = p.ctrl[i];
  // this CTA's slice [lo, hi) of the K entries: the kept records i in it are
  // placed, the unused positions in it (i >= kept) padded
  const int per = (K + (int)gridDim.y - 1) / (int)gridDim.y;
  const int lo = (int)blockIdx.y * per, hi = min(K, lo + per);
  // order the kept records by location: position = number of smaller keys,
  // counted by a warp per record (lanes over the other records)
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  for (int i = lo + warp; i < min(hi, kept); i += nwarps) {
    const unsigned long long ki = fin[i];
    unsigned pos = 0;
    for (int j = lane; j < kept; j += 32) pos += fin[j] < ki ? 1u : 0u;
    pos = __reduce_add_sync(0xffffffffu, pos);
    if (lane == 0) {
      const unsigned row = (unsigned)(ki >> 32) & 0xffffu, bin = (unsigned)(ki & 0xffffffffu);
      // gen_info.h:62-64: ((h-1)&7)<<29 | (row&0x7f)<<22 | (bin&0x3fffff)
      put((int)pos, (((unsigned)plane & 7u) << 29) | ((row & 0x7fu) << 22) | (bin & 0x3fffffu), finp[i]);
    }
  }
  for (int i = max(lo, kept) + (int)threadIdx.x; i < hi; i += blockDim.x) {
    put(i, p.invalid_location, -1.0f);
  }
  // (the planes' CTAs take 4 to 30 us, by their boundary records)
  if (p.stamp && threadIdx.x == 0) p.stamp[plane * kFinSlices + blockIdx.y] = global_ns();
}

// ----------------------------------------------------------------- launchers
int hsum_warps(int half) {
  const int w = (half + 1 + 3) / 4;
  return w <= 6 ? 6 : w <= 11 ? 11 : 16;
}
static int hsum_stages(const HsumParams &p) {
  switch (hsum_warps(p.half)) {
    case 6: return p.lean ? 3 : 5;
    case 11: return p.lean ? 2 : 3;
    default: return 2;
  }
}

int hsum_smem_bytes(const HsumParams &p) {
  return kHsHeader + hsum_stages(p) * p.stage_floats * 4 + (int)sizeof(EmitBuf) +
         hsum_warps(p.half) * 2 * (kMaxPlanes + 1) * 4;
}

template <int MAXP, int NW, int STAGES, int MINB>
static cudaError_t launch_hsum_t(const HsumParams &p, const HsumMaps &m, cudaStream_t s, bool pdl) {
  const int smem = hsum_smem_bytes(p);
  auto kern = hsum_kernel<MAXP, NW, STAGES, MINB>;
  const int n_sm = current_sm_count();
  const int items = (p.n_bins + kHsBins - 1) / kHsBins * 2;
  return launch_sized(kern, dim3(items < n_sm ? items : n_sm), dim3(32 * (NW + 1)), smem, s, pdl, p, m);
}

cudaError_t launch_hsum(const HsumParams &p, const HsumMaps &m, cudaStream_t s, bool pdl) {
  const bool few = p.n_planes <= 8;
  switch (hsum_warps(p.half)) {
    case 6:
      if (p.lean) return launch_hsum_t<8, 6, 3, 2>(p, m, s, pdl);
      return few ? launch_hsum_t<8, 6, 5, 1>(p, m, s, pdl) : launch_hsum_t<16, 6, 5, 1>(p, m, s, pdl);
    case 11:
      // lean: 2 stages and a register budget that fits next to one FT-convolution CTA
      if (p.lean) return launch_hsum_t<8, 11, 2, 2>(p, m, s, pdl);
      return few ? launch_hsum_t<8, 11, 3, 1>(p, m, s, pdl) : launch_hsum_t<16, 11, 3, 1>(p, m, s, pdl);
    default:
      // (code for 16 planes at 8: 2^17 bins x 127 rows with 0.1 / 0.3% of a plane above its
      // threshold 250 / 462 us a stage against 220 / 354, noise 52 / 49)
      return few ? launch_hsum_t<8, 16, 2, 1>(p, m, s, pdl) : launch_hsum_t<16, 16, 2, 1>(p, m, s, pdl);
  }
}

cudaError_t launch_split_taps(double2 *taps, long long n, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  const long long blocks = (n + 255) / 256;
  split_taps_kernel<<<(int)(blocks < 1024 ? blocks : 1024), 256, 0, s>>>(taps, n);
  return cudaGetLastError();
}

cudaError_t launch_recheck(const RecheckParams &p, cudaStream_t s, bool pdl) {
  const int warps = p.n_planes <= 8 ? 8 : 16;
  return launch_kernel(recheck_kernel, dim3(32 / warps * current_sm_count()), dim3(32 * warps), 0, s, pdl, p);
}

cudaError_t launch_select(const SelectParams &p, cudaStream_t s, bool pdl) {
  const int n_sm = current_sm_count();
  // More than half of what an SM has, so that it has room for one CTA: these may start
  // while the recheck's still hold SMs, and with 64 KB for 8 planes there were two on
  // some SMs and none on others (2^17 bins x 8 planes, 80 million hits: 1419 us a
  // search against 942; released at the recheck's end instead, they lose the SMs to the
  // other set's FT convolution: the loop over both sets at 2^21 1960 -> 2007 us; the
  // 128 KB of 16 planes for all: 1133).
  constexpr int kOnePerSm = 116 * 1024;
  static_assert(2 * kOnePerSm > kHsMaxSmem, "one CTA per SM");
  const int planes_smem = p.n_planes * kSelBuckets * 4;
  cudaError_t e = launch_sized(select_hist_kernel, dim3(n_sm), dim3(1024),
                               planes_smem > kOnePerSm ? planes_smem : kOnePerSm, s, pdl, p);
  if (e != cudaSuccess) return e;
  if ((e = launch_kernel(select_gather_kernel, dim3(4 * n_sm), dim3(256), 0, s, pdl, p)) != cudaSuccess) return e;
  const int fsmem = (kSortCap + kMaxCompat) * (8 + 4);
  e = allow_smem(select_finalize_kernel, fsmem);
  if (e != cudaSuccess) return e;
  return launch_kernel(select_finalize_kernel, dim3(p.n_planes, kFinSlices), dim3(1024), fsmem, s, pdl, p);
}

}  // namespace fdas
