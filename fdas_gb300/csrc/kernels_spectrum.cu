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
// takes R = up to 512 points of B neighbouring columns through shared memory,
// where the same formulation splits R into radices 16, 8, 4, 2, 3, 5, 7, so a
// transform of 2^21 points is three passes over memory (128 each) instead of
// seven of radix 8.  FP32 arithmetic; twiddles e^(-i pi x / N), x < 2 N, are
// products of two small tables held as float pairs (FP64 values as hi + lo), a
// thread's factors of a pass a geometric sequence in float pairs (two look-ups
// instead of a gather per point), and their low parts are part of the products:
// the error stays below that of radix-8 passes with rounded twiddles (2^21 / 10^6
// points: 1.65e-7 / 1.80e-7 of the norm against 1.68e-7 / 1.82e-7).
// The call on device samples at 2^21 / 10^6 / 2^18 points: 75 / 68 / 36 us against
// 112 / 82 / 45 with one pass per radix and the samples copied first; the passes
// are bound by the latency of their steps in shared memory (17 + 2 x 20 us at 2^21
// from cold, 8 MB/us), 2048 points per CTA (4096: 86 us, 1024: 82).
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

// forward DFT of odd size R on v[0..R) (direct, compile-time twiddles)
template <int R>
__device__ __forceinline__ void dft_odd(float2 *v) {
  float2 out[R];
  sfor<R>([&](auto K) {
    constexpr int k = decltype(K)::value;
    float2 acc = v[0];
    sfor<R - 1>([&](auto N1) {
      constexpr int n = decltype(N1)::value + 1;
      constexpr int j = (n * k) % R;
      acc = cadd(acc, rot<-1, R, j>(v[n]));
    });
    out[k] = acc;
  });
  sfor<R>([&](auto K) {
    constexpr int k = decltype(K)::value;
    v[k] = out[k];
  });
}
template <int R>
__device__ __forceinline__ void dft_any(float2 *v) {
  if constexpr (R == 2 || R == 4 || R == 8) dft_small<-1, R, 0, 1>(v);
  else if constexpr (R == 16) dft_composite<-1, 4, 4, 0, 1>(v);
  else dft_odd<R>(v);
}
// register of output k
template <int R>
__host__ __device__ constexpr int dft_at(int k) { return R == 16 ? 4 * (k % 4) + k / 4 : k; }

// One pass of composite radix R: for the columns j < M = N / R, k = j mod ns,
//   v[r] = in[j + r M] e^(-2 pi i k r / (ns R)),  v = DFT_R(v),
//   out[(j / ns) ns R + k + r ns] = v[r],
// B columns per CTA.  In shared memory [r][column], rows of B + 1 values (rows
// and columns are both read without conflicts); each step of radix Q reads one
// buffer and writes the other in the same formulation with R in place of N.
template <int Q>
__device__ __forceinline__ void pass_step(const SeriesPass &p, const float2 *__restrict__ in, const float2 *src, float2 *dst,
                                          const float4 *wr, const float4 *__restrict__ tw, long long j0, int cols,
                                          int sns) {
  const int rows = p.R / Q, pitch = p.B + 1;
  for (int w = threadIdx.x; w < rows * p.B; w += blockDim.x) {
    const int b = w & (p.B - 1), jj = w >> p.log_b;
    float2 v[Q];
    int at = jj * Q, kk = 0;
    if (!src) {  // the first step: from memory, with the twiddles of the pass
      if (b >= cols) continue;
      const long long j = j0 + b;
      sfor<Q>([&](auto I) {
        constexpr int i = decltype(I)::value;
        v[i] = in[j + (long long)(jj + i * rows) * p.m];
      });
      if (p.ns > 1) {
        // a geometric sequence over the thread's points, kept in float pairs: each
        // factor is as good as a table entry, and two look-ups serve all of them
        const unsigned step = (unsigned)(j % p.ns) * (unsigned)p.unit;  // k 2N / (ns R)
        Df2 w = series_tw(tw, step * (unsigned)jj);
        const Df2 ratio = series_tw(tw, step * (unsigned)rows);
        sfor<Q>([&](auto I) {
          constexpr int i = decltype(I)::value;
          v[i] = cmul_df(v[i], w);
          if constexpr (i + 1 < Q) w = df_mul(w, ratio);
        });
      }
    } else {
      const int blk = jj / sns;
      kk = jj - blk * sns;
      at = blk * sns * Q + kk;
      sfor<Q>([&](auto I) {
        constexpr int i = decltype(I)::value;
        v[i] = src[(jj + i * rows) * pitch + b];
      });
      const int unit = kk * (p.R / (sns * Q));
      sfor<Q - 1>([&](auto I) {
        constexpr int i = decltype(I)::value + 1;
        const float4 w = wr[unit * i];
        v[i] = cmul_df(v[i], Df2{w.x, w.y, w.z, w.w});
      });
    }
    dft_any<Q>(v);
    sfor<Q>([&](auto I) {
      constexpr int i = decltype(I)::value;
      dst[(at + i * sns) * pitch + b] = v[dft_at<Q>(i)];
    });
  }
}

__global__ void __launch_bounds__(256) series_pass_kernel(const float2 *__restrict__ in, float2 *__restrict__ out,
                                                          SeriesPass p, const float4 *__restrict__ tw) {
  extern __shared__ float2 fft_smem[];
  const int pitch = p.B + 1;
  float2 *buf[2] = {fft_smem, fft_smem + p.R * pitch};
  float4 *wr = reinterpret_cast<float4 *>(fft_smem + 2 * p.R * pitch);  // e^(-2 pi i x / R)
  for (int x = threadIdx.x; x < p.R; x += blockDim.x) {
    const Df2 w = series_tw(tw, (unsigned)x * 2u * (unsigned)p.m);
    wr[x] = make_float4(w.x, w.y, w.z, w.w);
  }
  const long long j0 = (long long)blockIdx.x * p.B;
  const int cols = (int)min((long long)p.B, p.m - j0);
  int sns = 1;
  const float2 *src = nullptr;
  for (int s = 0; s < p.n_steps; ++s) {
    float2 *dst = buf[s & 1];
    switch (p.radix[s]) {
      case 16: pass_step<16>(p, in, src, dst, wr, tw, j0, cols, sns); break;
      case 8: pass_step<8>(p, in, src, dst, wr, tw, j0, cols, sns); break;
      case 4: pass_step<4>(p, in, src, dst, wr, tw, j0, cols, sns); break;
      case 2: pass_step<2>(p, in, src, dst, wr, tw, j0, cols, sns); break;
      case 3: pass_step<3>(p, in, src, dst, wr, tw, j0, cols, sns); break;
      case 5: pass_step<5>(p, in, src, dst, wr, tw, j0, cols, sns); break;
      default: pass_step<7>(p, in, src, dst, wr, tw, j0, cols, sns); break;
    }
    sns *= p.radix[s];
    src = dst;
    __syncthreads();
  }
  if (p.ns == 1) {  // a column's R outputs are neighbours
    for (int i = threadIdx.x; i < cols * p.R; i += blockDim.x) {
      const int b = i / p.R, r = i - b * p.R;
      out[(j0 + b) * p.R + r] = src[r * pitch + b];
    }
  } else {
    for (int i = threadIdx.x; i < p.R * p.B; i += blockDim.x) {
      const int b = i & (p.B - 1), r = i >> p.log_b;
      if (b >= cols) continue;
      const long long j = j0 + b, blk = j / p.ns;
      out[blk * p.ns * p.R + (j - blk * p.ns) + (long long)r * p.ns] = src[r * pitch + b];
    }
  }
}

// Real-input split step, one thread per pair (k, N - k), 0 <= k <= N / 2;
// in place when z == x.
__global__ void __launch_bounds__(256) real_split_kernel(const float2 *z, float2 *x, int n, float scale,
                                                         const float4 *__restrict__ tw) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k > n / 2) return;
  const int kk = (n - k) % n;
  const float2 a = z[k], b = z[kk];
  const Df2 w = series_tw(tw, (unsigned)k);
  auto bin = [&](float2 za, float2 zb, float2 wq) {
    // Fe = (za + conj zb) / 2, Fo = (za - conj zb) / (2 i); X = Fe + e^(-i pi q / N) Fo
    const float2 fe = make_float2(0.5f * (za.x + zb.x), 0.5f * (za.y - zb.y));
    const float2 fo = make_float2(0.5f * (za.y + zb.y), -0.5f * (za.x - zb.x));
    return make_float2(scale * fmaf(-wq.y, fo.y, fmaf(wq.x, fo.x, fe.x)),
                       scale * fmaf(wq.x, fo.y, fmaf(wq.y, fo.x, fe.y)));
  };
  const float2 xk = bin(a, b, make_float2(w.x, w.y));
  if (kk != k && k != 0) x[kk] = bin(b, a, make_float2(-w.x, w.y));  // e^(-i pi (N - k) / N) = -conj w
  x[k] = xk;
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
  int count = 1;
  for (double r = kMaxR; r < (double)n; r *= 160.0) ++count;
  for (;; ++count) {
    if (count > max_passes) return -1;
    int R[16];
    for (int i = 0; i < count; ++i) R[i] = 1;
    for (int i = 0; i < np; ++i) *std::min_element(R, R + count) *= primes[i];
    if (*std::max_element(R, R + count) > kMaxR) continue;
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
      int left = p.R;
      for (int f : {7, 5, 3})
        while (left % f == 0) {
          p.radix[p.n_steps++] = f;
          left /= f;
        }
      // what is left is 2^e: fewest steps of at most 16, the large ones first
      int e = 0;
      while ((1 << e) < left) ++e;
      for (int steps = (e + 3) / 4; steps > 0; --steps) {
        const int q = (e + steps - 1) / steps;
        p.radix[p.n_steps++] = 1 << q;
        e -= q;
      }
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
  for (int i = 0; i < np; ++i) {
    if (pass[i].n_steps == 0) continue;  // n = 1
    float2 *dst = bufs[i & 1];
    const int smem = (2 * pass[i].R * (pass[i].B + 1) + 2 * pass[i].R) * (int)sizeof(float2);
    cudaError_t e = cudaFuncSetAttribute(series_pass_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    series_pass_kernel<<<(unsigned)((pass[i].m + pass[i].B - 1) / pass[i].B), 256, smem, s>>>(cur, dst, pass[i], p.tw);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    cur = dst;
  }
  real_split_kernel<<<(p.n / 2 + 1 + 255) / 256, 256, 0, s>>>(cur, p.z, p.n, p.scale, p.tw);
  return cudaGetLastError();
}

}  // namespace fdas
