// Upstream step: the normalised spectrum of a real time series
// (ft_conv.py:134-143: ``ft = fft(samples) / n_samp``, first N bins kept).
//
// The 2N real samples are read as N complex values z[n] = x[2n] + i x[2n+1]
// (no copy), transformed by an N-point complex FFT, and split into the
// spectrum of the real series:
//   X[k] = (Z[k] + conj Z[N-k]) / 2 - i e^(-i pi k / N) (Z[k] - conj Z[N-k]) / 2.
// The N-point FFT is a mixed-radix Stockham auto-sort FFT following the radix-R
// formulation of Govindaraju et al., "High performance discrete Fourier
// transforms on graphics processors" (SC 2008), with composite radices: a pass
// takes R = up to 1024 points of B neighbouring columns through shared memory,
// where the same formulation splits R into steps of 2 to 16 points, so a transform
// of 2^21 points is three passes over memory (128 = 16 x 8 each), one of 10^6 two
// (1000 = 10 x 10 x 10).  FP32 arithmetic; twiddles e^(-i pi x / N), x < 2 N, are
// products of two small tables held as float pairs (FP64 values as hi + lo), a
// thread's factors of a pass a geometric sequence in float pairs (two look-ups
// instead of a gather per point), and their low parts are part of the products:
// the error stays below that of radix-8 passes with rounded twiddles (2^21 / 10^6
// points: 1.65e-7 / 1.69e-7 of the norm against 1.68e-7 / 1.82e-7).
// The call on device samples at 2^21 / 10^6 / 2^18 points: 54 / 37 / 26 us against
// 112 / 82 / 45 with one pass per radix and the samples copied first, and 76 / 68 /
// 36 with steps of prime or power-of-two size, 64-bit index divisions per point and a
// copy through shared memory before the store: the passes issued 25,000 cycles of
// instructions per SM, 13 of their 18 us at 10^6 points.  What is left is latency:
// four to five kernels of 6 to 10 us and the call's launch and wait.  2048 points per
// CTA (1024 or 4096: the same to 5 % slower), a thread per item of the step with the
// fewest items (256 for all: 61 against 43 us at 10^6 in three passes).
#include <cuda_runtime.h>

#include <algorithm>
#include <functional>

#include "fft2048.cuh"
#include "kernels.cuh"

namespace fdas {

// tw[0 .. kTwFine): e^(-i pi x / N), then e^(-i pi kTwFine y / N), y < 2 N / kTwFine
// + 1, each as (re hi, im hi, re lo, im lo)
__global__ void series_twiddle_kernel(float4 *tw, int n, int count) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const double x = i < kTwFine ? (double)i : (double)(i - kTwFine) * kTwFine;
  double s, c;
  sincospi(-x / (double)n, &s, &c);
  const float ch = (float)c, sh = (float)s;
  tw[i] = make_float4(ch, sh, (float)(c - (double)ch), (float)(s - (double)sh));
}

// A complex number as float pairs: re = x + z, im = y + w to about 2^-46
struct Df2 {
  float x, y, z, w;
};
// (a + al)(c + cl) - (b + bl)(d + dl) as hi + lo: the float products with their
// rounding errors (fused multiply-adds), two-sum of the products
__device__ __forceinline__ void df_cross(float a, float al, float c, float cl, float b, float bl, float d, float dl,
                                         float &hi, float &lo) {
  const float p = a * c, q = b * d;
  const float pe = fmaf(a, c, -p), qe = fmaf(b, d, -q);
  const float s = p - q, bb = s - p;
  const float e = ((p - (s - bb)) - (q + bb)) + ((pe - qe) + (fmaf(a, cl, al * c) - fmaf(b, dl, bl * d)));
  hi = s + e;
  lo = (s - hi) + e;
}
__device__ __forceinline__ Df2 df_mul(Df2 f, Df2 g) {
  Df2 r;
  df_cross(f.x, f.z, g.x, g.z, f.y, f.w, g.y, g.w, r.x, r.z);
  df_cross(f.x, f.z, g.y, g.w, -f.y, -f.w, g.x, g.z, r.y, r.w);
  return r;
}
// v w, the factor's low parts included: one rounding less
__device__ __forceinline__ float2 cmul_df(float2 v, Df2 w) {
  return make_float2(fmaf(v.x, w.x, fmaf(-v.y, w.y, fmaf(v.x, w.z, -v.y * w.w))),
                     fmaf(v.x, w.y, fmaf(v.y, w.x, fmaf(v.x, w.w, v.y * w.z))));
}
// e^(-i pi x / N) for 0 <= x < 2 N
__device__ __forceinline__ Df2 series_tw(const float4 *__restrict__ tw, unsigned x) {
  const float4 f = __ldg(tw + (x & (kTwFine - 1))), g = __ldg(tw + kTwFine + x / kTwFine);
  return df_mul(Df2{f.x, f.y, f.z, f.w}, Df2{g.x, g.y, g.z, g.w});
}

// Forward DFT of size R on v[OFF + STRIDE n], in place and in natural order for
// R <= 8; odd sizes from the sums and differences of v[n] and v[R - n].
template <int R, int OFF, int STRIDE>
__device__ __forceinline__ void dft_prime(float2 *v) {
  if constexpr (R == 2 || R == 4 || R == 8) {
    dft_small<-1, R, OFF, STRIDE>(v);
  } else {
    constexpr int H = R / 2;
    float2 sum[H], dif[H], x0 = v[OFF];
    sfor<H>([&](auto I) {
      constexpr int n = decltype(I)::value + 1;
      const float2 a = v[OFF + STRIDE * n], b = v[OFF + STRIDE * (R - n)];
      sum[n - 1] = cadd(a, b);
      dif[n - 1] = csub(a, b);
      v[OFF] = cadd(v[OFF], sum[n - 1]);
    });
    sfor<H>([&](auto K) {
      constexpr int k = decltype(K)::value + 1;
      float2 c = x0, d = make_float2(0.f, 0.f);  // sum of cos terms; of sin terms
      sfor<H>([&](auto I) {
        constexpr int n = decltype(I)::value + 1;
        c = cfma_real(kCos<R, (n * k) % R>, sum[n - 1], c);
        d = cfma_real(kSin<R, (n * k) % R>, dif[n - 1], d);
      });
      // exp(-i t) = cos t - i sin t: -i d = (d.y, -d.x)
      v[OFF + STRIDE * k] = make_float2(c.x + d.y, c.y - d.x);
      v[OFF + STRIDE * (R - k)] = make_float2(c.x - d.y, c.y + d.x);
    });
  }
}
// Sizes of a step: 2 to 10, 12, 14, 15 and 16.  6, 10, 12, 14 and 15 are products
// A B of coprime factors: with n = B n1 + A n2 mod R the factors between the two
// stages are 1 (Good, "The interaction algorithm and practical Fourier analysis",
// 1958), which saves their products and roundings; 9 and 16 are 3 x 3 and 4 x 4.
template <int R>
struct Split {
  static constexpr int A =
      R == 6 || R == 9 ? 3 : R == 10 || R == 15 ? 5 : R == 12 ? 3 : R == 14 ? 7 : R == 16 ? 4 : R;
  static constexpr int B = R / A;
  static constexpr bool coprime = B > 1 && A != B;
};
template <int R>
__device__ __forceinline__ void dft_any(float2 *v) {
  constexpr int A = Split<R>::A, B = Split<R>::B;
  if constexpr (B == 1) {
    dft_prime<R, 0, 1>(v);
  } else if constexpr (Split<R>::coprime) {
    float2 u[R];
    sfor<R>([&](auto I) {
      constexpr int n1 = decltype(I)::value % A, n2 = decltype(I)::value / A;
      u[A * n2 + n1] = v[(B * n1 + A * n2) % R];
    });
    sfor<B>([&](auto N2) { dft_prime<A, A * decltype(N2)::value, 1>(u); });
    sfor<A>([&](auto K1) { dft_prime<B, decltype(K1)::value, A>(u); });
    sfor<R>([&](auto I) { v[decltype(I)::value] = u[decltype(I)::value]; });
  } else {
    sfor<B>([&](auto N2) { dft_prime<A, decltype(N2)::value, B>(v); });
    sfor<A>([&](auto K1) {
      sfor<B>([&](auto N2) {
        constexpr int k1 = decltype(K1)::value, n2 = decltype(N2)::value;
        v[B * k1 + n2] = rot<-1, R, n2 * k1>(v[B * k1 + n2]);
      });
    });
    sfor<A>([&](auto K1) { dft_prime<B, B * decltype(K1)::value, 1>(v); });
  }
}
// register of output k
template <int R>
__host__ __device__ constexpr int dft_at(int k) {
  constexpr int A = Split<R>::A, B = Split<R>::B;
  return B == 1 ? k : Split<R>::coprime ? A * (k % B) + k % A : B * (k % A) + k / A;
}

// One pass of composite radix R: for the columns j < M = N / R, k = j mod ns,
//   v[r] = in[j + r M] e^(-2 pi i k r / (ns R)),  v = DFT_R(v),
//   out[(j / ns) ns R + k + r ns] = v[r],
// B columns per CTA, in steps of radix Q in the same formulation with R in place
// of N: the first reads memory, the last writes it, what lies between goes through
// shared memory, [r][column] in rows of B + 1 values.  A thread works on one column
// (its k and output offset are divided out once); in the last step of the first
// pass (ns = 1, a column's outputs are neighbours) the lanes follow the rows.
template <int Q>
__device__ __forceinline__ void pass_step(const SeriesPass &p, bool first, bool last, const float2 *__restrict__ in,
                                          float2 *__restrict__ out, const float2 *src, float2 *dst, const float4 *wr,
                                          const float4 *__restrict__ tw, unsigned j0, unsigned cols, unsigned sns) {
  const unsigned rows = (unsigned)p.R / Q, pitch = p.B + 1;
  const bool across = last && p.ns == 1;
  unsigned b = threadIdx.x & (p.B - 1);
  unsigned k = 0;
  float2 *o = out;
  Df2 ratio{1.f, 0.f, 0.f, 0.f};
  unsigned step = 0;
  if (p.ns > 1 && (first || last)) {
    const unsigned j = j0 + b, blk = j / (unsigned)p.ns;
    k = j - blk * p.ns;
    o += (size_t)blk * p.ns * p.R + k;
    step = k * (unsigned)p.unit;  // k 2N / (ns R)
    if (first) ratio = series_tw(tw, step * rows);
  }
  for (unsigned w = threadIdx.x; w < rows * p.B; w += blockDim.x) {
    unsigned jj = w >> p.log_b;
    if (across) {
      b = w / rows;
      jj = w - b * rows;
      o = out + (size_t)(j0 + b) * p.R;
    }
    if (b >= cols) continue;
    float2 v[Q];
    unsigned at = jj * Q, kk = 0;
    if (first) {
      const float2 *i0 = in + j0 + b;
      sfor<Q>([&](auto I) {
        constexpr int i = decltype(I)::value;
        v[i] = i0[(size_t)((jj + i * rows) * p.m)];
      });
      if (p.ns > 1) {
        // a geometric sequence over the thread's points, kept in float pairs: each
        // factor is as good as a table entry, and two look-ups serve all of them
        Df2 f = series_tw(tw, step * jj);
        sfor<Q>([&](auto I) {
          constexpr int i = decltype(I)::value;
          v[i] = cmul_df(v[i], f);
          if constexpr (i + 1 < Q) f = df_mul(f, ratio);
        });
      }
    } else {
      const unsigned blk = last ? 0 : jj / sns;
      kk = jj - blk * sns;
      at = blk * sns * Q + kk;
      sfor<Q>([&](auto I) {
        constexpr int i = decltype(I)::value;
        v[i] = src[(jj + i * rows) * pitch + b];
      });
      const unsigned unit = last ? kk : kk * (p.R / (sns * Q));
      sfor<Q - 1>([&](auto I) {
        constexpr int i = decltype(I)::value + 1;
        const float4 f = wr[unit * i];
        v[i] = cmul_df(v[i], Df2{f.x, f.y, f.z, f.w});
      });
    }
    dft_any<Q>(v);
    if (last) {
      sfor<Q>([&](auto I) {
        constexpr int i = decltype(I)::value;
        o[(size_t)((jj + i * rows) * p.ns)] = v[dft_at<Q>(i)];
      });
    } else {
      sfor<Q>([&](auto I) {
        constexpr int i = decltype(I)::value;
        dst[(at + i * sns) * pitch + b] = v[dft_at<Q>(i)];
      });
    }
  }
}

__global__ void __launch_bounds__(512) series_pass_kernel(const float2 *__restrict__ in, float2 *__restrict__ out,
                                                          SeriesPass p, const float4 *__restrict__ tw) {
  extern __shared__ float2 fft_smem[];
  const unsigned pitch = p.B + 1;
  float4 *wr = reinterpret_cast<float4 *>(fft_smem);  // e^(-2 pi i x / R)
  float2 *buf[2] = {fft_smem + 2 * p.R, fft_smem + 2 * p.R + p.R * pitch};
  if (p.n_steps > 1)
    for (int x = threadIdx.x; x < p.R; x += blockDim.x) {
      const Df2 w = series_tw(tw, (unsigned)x * 2u * (unsigned)p.m);
      wr[x] = make_float4(w.x, w.y, w.z, w.w);
    }
  grid_wait();
  const unsigned j0 = blockIdx.x * p.B;
  const unsigned cols = min((unsigned)p.B, (unsigned)p.m - j0);
  unsigned sns = 1;
  const float2 *src = nullptr;
  for (int s = 0; s < p.n_steps; ++s) {
    float2 *dst = buf[s & 1];
    const bool first = s == 0, last = s + 1 == p.n_steps;
    switch (p.radix[s]) {
#define FDAS_STEP(Q) \
  case Q: pass_step<Q>(p, first, last, in, out, src, dst, wr, tw, j0, cols, sns); break;
      FDAS_STEP(2) FDAS_STEP(3) FDAS_STEP(4) FDAS_STEP(5) FDAS_STEP(6) FDAS_STEP(7) FDAS_STEP(8) FDAS_STEP(9)
      FDAS_STEP(10) FDAS_STEP(12) FDAS_STEP(14) FDAS_STEP(15)
#undef FDAS_STEP
      default: pass_step<16>(p, first, last, in, out, src, dst, wr, tw, j0, cols, sns); break;
    }
    sns *= p.radix[s];
    src = dst;
    if (!last) __syncthreads();
  }
  grid_release();
}

// Real-input split step, one thread per pair (k, N - k), 0 <= k <= N / 2;
// in place when z == x.  A pinned array of the caller's is written here too (10^6 bins
// 90.4 -> 84.7 us, 32768 bins 37 -> 28: the copy's own launch; the link's 43 us for
// 10^6 bins stay).
__global__ void __launch_bounds__(256) real_split_kernel(const float2 *z, float2 *x, float2 *host, int n,
                                                         float scale, const float4 *__restrict__ tw) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k > n / 2) return;
  const int kk = k ? n - k : 0;
  const Df2 w = series_tw(tw, (unsigned)k);
  grid_wait();
  const float2 a = z[k], b = z[kk];
  auto bin = [&](float2 za, float2 zb, float2 wq) {
    // Fe = (za + conj zb) / 2, Fo = (za - conj zb) / (2 i); X = Fe + e^(-i pi q / N) Fo
    const float2 fe = make_float2(0.5f * (za.x + zb.x), 0.5f * (za.y - zb.y));
    const float2 fo = make_float2(0.5f * (za.y + zb.y), -0.5f * (za.x - zb.x));
    return make_float2(scale * fmaf(-wq.y, fo.y, fmaf(wq.x, fo.x, fe.x)),
                       scale * fmaf(wq.x, fo.y, fmaf(wq.y, fo.x, fe.y)));
  };
  const float2 xk = bin(a, b, make_float2(w.x, w.y));
  if (kk != k && k != 0) {
    const float2 xkk = bin(b, a, make_float2(-w.x, w.y));  // e^(-i pi (N - k) / N) = -conj w
    x[kk] = xkk;
    if (host) host[kk] = xkk;
  }
  x[k] = xk;
  if (host) host[k] = xk;
}

// Fewest steps of the sizes above, the largest as small as that allows, large ones
// first
void step_split(int left, SeriesPass &best) {
  struct Search {
    int best_n = 9, best_max = 0, trial[8], found[8];
    void go(int left, int n, int limit) {
      if (left == 1) {
        if (n < best_n || (n == best_n && trial[0] < best_max)) {
          best_n = n;
          best_max = n ? trial[0] : 0;
          std::copy(trial, trial + n, found);
        }
        return;
      }
      if (n == 8) return;
      for (int q : {16, 15, 14, 12, 10, 9, 8, 7, 6, 5, 4, 3, 2})
        if (q <= limit && left % q == 0) {
          trial[n] = q;
          go(left / q, n + 1, q);
        }
    }
  } search;
  search.go(left, 0, 16);
  best.n_steps = search.best_n;
  std::copy(search.found, search.found + search.best_n, best.radix);
}

// Passes of composite radix <= kMaxR over the factors of n: as few as that
// allows, the factors dealt to the smallest product so far (equal passes).
int series_plan(int n, SeriesPass *pass, int max_passes) {
  constexpr int kMaxR = 512;
  int primes[32], np = 0;
  int rest = n;
  for (int f : {7, 5, 3, 2})
    while (rest % f == 0) {
      primes[np++] = f;
      rest /= f;
    }
  if (rest != 1) return -1;
  int count = 1, max_r = kMaxR;
  for (double r = kMaxR; r < (double)n; r *= 160.0) ++count;
  // two passes of up to 1024 instead of three of about 100 from 655360 points on, where
  // a pass more costs more than its CTAs of 8192 points wait (device samples, two
  // against three: 524288 34.5 / 31.5 us, 700000 35 / 35, 800000 36.0 / 39.8, 2^20 38 / 40.5, 10^6 37 / 42.5)
  if (n > 655360 && n <= 1024 * 1024) count = 2, max_r = 1024;
  for (;; ++count) {
    if (count > max_passes) return -1;
    int R[16];
    for (int i = 0; i < count; ++i) R[i] = 1;
    for (int i = 0; i < np; ++i) *std::min_element(R, R + count) *= primes[i];
    if (*std::max_element(R, R + count) > max_r) {
      max_r = kMaxR;
      continue;
    }
    std::sort(R, R + count, std::greater<int>());
    int ns = 1, used = 0;
    for (int i = 0; i < count; ++i) {
      if (R[i] == 1 && used > 0) continue;
      SeriesPass &p = pass[used++];
      p.R = R[i];
      p.m = n / R[i];
      p.ns = ns;
      p.unit = 2 * (p.m / ns);
      // columns: about 2048 points per CTA, at least 8 columns (64-byte rows)
      p.log_b = 3;
      while (p.R << (p.log_b + 1) <= 2048 && p.log_b < 5) ++p.log_b;
      p.B = 1 << p.log_b;
      p.n_steps = 0;
      step_split(p.R, p);
      // threads: one item each in the step that has the fewest
      p.threads = p.R > kMaxR ? 512 : 256;
      for (int s = 0; s < p.n_steps; ++s) p.threads = std::min(p.threads, (p.R / p.radix[s] * p.B + 31) & ~31);
      ns *= R[i];
    }
    return used;
  }
}

size_t series_twiddle_count(int n) { return (size_t)kTwFine + 2 * (size_t)n / kTwFine + 1; }

cudaError_t launch_series_twiddles(float4 *tw, int n, cudaStream_t s) {
  const int count = (int)series_twiddle_count(n);
  series_twiddle_kernel<<<(count + 255) / 256, 256, 0, s>>>(tw, n, count);
  return cudaGetLastError();
}

cudaError_t launch_series_spectrum(const SeriesParams &p, cudaStream_t s) {
  SeriesPass pass[16];
  const int np = series_plan(p.n, pass, 16);
  if (np < 0) return cudaErrorInvalidValue;
  const float2 *cur = p.samples;
  // ping-pong so that no pass reads what it writes; the split may work in place
  float2 *bufs[2] = {cur == p.z ? p.scratch : p.z, cur == p.z ? p.z : p.scratch};
  bool chained = false;
  for (int i = 0; i < np; ++i) {
    if (pass[i].n_steps == 0) continue;  // n = 1
    float2 *dst = bufs[i & 1];
    const SeriesPass &q = pass[i];
    const int buffers = std::min(q.n_steps - 1, 2);
    const int smem = (2 * q.R + buffers * q.R * (q.B + 1)) * (int)sizeof(float2);
    const cudaError_t e = launch_sized(series_pass_kernel, (unsigned)((q.m + q.B - 1) / q.B), q.threads, smem, s,
                                       chained, cur, dst, q, p.tw);
    if (e != cudaSuccess) return e;
    chained = true;
    cur = dst;
  }
  return launch_kernel(real_split_kernel, (p.n / 2 + 1 + 255) / 256, 256, 0, s, chained, cur, p.z, p.host, p.n, p.scale,
                       p.tw);
}

}  // namespace fdas
