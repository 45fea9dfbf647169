// FP32 image <-> grid transforms for sizes whose prime factors are 2, 3, 5 and
// 7: two passes over memory per direction, with the grid correction and the
// centring shifts inside them.
//
// The shifts cost nothing: for even n, with s(a, b) = (-1)^(a + b),
//   fftshift(FFT(ifftshift(x)))  = s FFT(s x)     (and likewise for the inverse),
// so they are signs applied while loading and storing.  The image is real, so
// only the columns v <= n/2 are transformed: the rest of the grid follows from
// F(u, v) = conj F(-u, -v), and the adjoint needs only the Hermitian half of the
// grid, (G(u, v) + conj G(-u, -v)) / 2, whose transform is the real part wanted.
//   image -> grid:  k_fft_rows_in    two image rows as one complex row; their
//                                    two half spectra into the left half of the
//                                    grid's own rows
//                   k_fft_cols_out   a few columns at a time, in place; each
//                                    also writes its mirror column
//   grid -> image:  k_fft_cols_in    Hermitian half, columns into the work array
//                   k_fft_rows_out   two rows as one complex row, corrected
// A line is transformed by decimation in frequency with radices 16, 8, 4, 2, 3,
// 5, 7: the first stage reads global memory, the last writes it (the columns) or
// the row's second buffer, the others work in place in shared memory; the
// digit-reversed order is undone by the last stage's stores.  Twiddles come from
// a table per stage, in the order in which a warp reads them, each rounded once
// from FP64.
//
// The passes move 20 n^2 bytes each way (cuFFT between shift kernels, complex
// both ways: 60 to 76).  Both directions at 4096^2 take 246 us, rows 45 to 55 us
// and columns 67 to 74 us (floor at the copy bandwidth: 59 us for both
// directions; with cuFFT 541 us); 2048^2 84 us (with cuFFT 145 us), 3072^2 176
// (348), 6144^2 740 (1356).  From 7168 on two columns fit a CTA instead of four and
// one CTA's rows an SM, so that each gets all of the SM's threads: 7680^2 1610 us (with
// cuFFT 2247), 8192^2 1722 (1978), 8000^2 1889 (1934), 7776^2 1948 (1858, the one
// size at which cuFFT is faster); with the threads of the smaller sizes 1996, 2013, 2270
// and 2496.  A line's trips through shared memory and the latency at 16 to 24 warps per SM
// bound them.  Tried at 4096^2: radix 8 with every stage through shared memory
// 322 us, twiddles gathered from one table of n roots 501 us; rows at two and four
// CTAs per SM 260 and 253 us; two columns of 128 threads per CTA 358 us (radix 8).
// Other sizes (a prime factor above 7, beyond 8192) stay with cuFFT.
#include <float.h>
#include <math.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <utility>
#include <vector>

#include "gb_common.cuh"
#include "gb_fft.cuh"
#include "gb_runtime.cuh"

namespace gb {
namespace {

constexpr int kMaxStages = 14;
constexpr int kRowRegs = 768;  // threads per SM that the rows' kernels leave registers for
constexpr int kColThreads = 512;  // for all of a CTA's columns

struct FftPlan {
  int n, stages;
  int radix[kMaxStages];
  int m[kMaxStages];     // distance between a butterfly's elements
  uint32_t mul[kMaxStages];  // b / m = (b * mul) >> 32 for b < 2^16
  int tw_at[kMaxStages];     // the stage's twiddles: [slot][j], exp(-2 pi i j k / (R m)) (tw_k)
  const float2* tw;
  const uint16_t* rev;  // the last stage's butterfly b has the frequencies rev[b] + k n / R
};

// Element i of a line in shared memory: its low four bits (the 16 eight-byte
// bank pairs) take those of i / 8 as well, so that elements 1, 8 or 64 apart all
// fall on different banks.
__device__ __forceinline__ int at(int i) { return i ^ ((i >> 3) & 15); }
// Lines are this far apart: four more than a multiple of 16, so that the four
// columns that a half-warp loads meet no bank conflict either.
__host__ __device__ constexpr int line(int n) { return ((n + 15) & ~15) + 4; }

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 rotm(float2 a) { return make_float2(a.y, -a.x); }  // -i a

template <int R>
__device__ __forceinline__ void dft(float2 (&x)[R]);

template <>
__device__ __forceinline__ void dft<2>(float2 (&x)[2]) {
  const float2 a = x[0];
  x[0] = cadd(a, x[1]);
  x[1] = csub(a, x[1]);
}
template <>
__device__ __forceinline__ void dft<4>(float2 (&x)[4]) {
  const float2 a = cadd(x[0], x[2]), b = csub(x[0], x[2]);
  const float2 c = cadd(x[1], x[3]), d = rotm(csub(x[1], x[3]));
  x[0] = cadd(a, c);
  x[1] = cadd(b, d);
  x[2] = csub(a, c);
  x[3] = csub(b, d);
}
template <>
__device__ __forceinline__ void dft<8>(float2 (&x)[8]) {
  constexpr float h = 0.70710678118654752440f;
  float2 e[4] = {x[0], x[2], x[4], x[6]}, o[4] = {x[1], x[3], x[5], x[7]};
  dft<4>(e);
  dft<4>(o);
  const float2 o1 = make_float2(h * (o[1].x + o[1].y), h * (o[1].y - o[1].x));
  const float2 o2 = rotm(o[2]);
  const float2 o3 = make_float2(h * (o[3].y - o[3].x), -h * (o[3].x + o[3].y));
  x[0] = cadd(e[0], o[0]);
  x[1] = cadd(e[1], o1);
  x[2] = cadd(e[2], o2);
  x[3] = cadd(e[3], o3);
  x[4] = csub(e[0], o[0]);
  x[5] = csub(e[1], o1);
  x[6] = csub(e[2], o2);
  x[7] = csub(e[3], o3);
}
template <>
__device__ __forceinline__ void dft<16>(float2 (&x)[16]) {
  // 4 x 4: columns, the twiddles exp(-2 pi i a b / 16), rows
  constexpr float c1 = 0.92387953251128675613f, s1 = 0.38268343236508977173f;
  constexpr float h = 0.70710678118654752440f;
  float2 y[4][4];
#pragma unroll
  for (int a = 0; a < 4; a++) {
    float2 c[4] = {x[a], x[a + 4], x[a + 8], x[a + 12]};
    dft<4>(c);
#pragma unroll
    for (int b = 0; b < 4; b++) y[b][a] = c[b];
  }
  y[1][1] = cmul(y[1][1], make_float2(c1, -s1));
  y[1][2] = make_float2(h * (y[1][2].x + y[1][2].y), h * (y[1][2].y - y[1][2].x));
  y[1][3] = cmul(y[1][3], make_float2(s1, -c1));
  y[2][1] = make_float2(h * (y[2][1].x + y[2][1].y), h * (y[2][1].y - y[2][1].x));
  y[2][2] = rotm(y[2][2]);
  y[2][3] = make_float2(h * (y[2][3].y - y[2][3].x), -h * (y[2][3].x + y[2][3].y));
  y[3][1] = cmul(y[3][1], make_float2(s1, -c1));
  y[3][2] = make_float2(h * (y[3][2].y - y[3][2].x), -h * (y[3][2].x + y[3][2].y));
  y[3][3] = cmul(y[3][3], make_float2(-c1, s1));
#pragma unroll
  for (int b = 0; b < 4; b++) {
    dft<4>(y[b]);
#pragma unroll
    for (int f = 0; f < 4; f++) x[b + 4 * f] = y[b][f];
  }
}
// Odd radices: sums and differences of the pairs k, R - k, then the cosine
// sums of the former and the sine sums of the latter.
template <int R>
__device__ __forceinline__ void dft_odd(float2 (&x)[R], const float (&c)[R / 2], const float (&s)[R / 2]) {
  constexpr int H = R / 2;
  float2 p[H], q[H];
#pragma unroll
  for (int k = 0; k < H; k++) {
    p[k] = cadd(x[k + 1], x[R - 1 - k]);
    q[k] = csub(x[k + 1], x[R - 1 - k]);
  }
  const float2 x0 = x[0];
#pragma unroll
  for (int k = 0; k < H; k++) x[0] = cadd(x[0], p[k]);
#pragma unroll
  for (int f = 1; f <= H; f++) {
    float2 a = x0, b = make_float2(0.f, 0.f);
#pragma unroll
    for (int k = 1; k <= H; k++) {
      const int t = f * k % R, u = t <= H ? t : R - t;  // cos and sin of 2 pi t / R
      const float cc = c[u - 1], ss = t <= H ? s[u - 1] : -s[u - 1];
      a.x = fmaf(cc, p[k - 1].x, a.x);
      a.y = fmaf(cc, p[k - 1].y, a.y);
      b.x = fmaf(ss, q[k - 1].x, b.x);
      b.y = fmaf(ss, q[k - 1].y, b.y);
    }
    const float2 ib = rotm(b);
    x[f] = cadd(a, ib);
    x[R - f] = csub(a, ib);
  }
}
template <>
__device__ __forceinline__ void dft<3>(float2 (&x)[3]) {
  const float c[1] = {-0.5f}, s[1] = {0.86602540378443864676f};
  dft_odd<3>(x, c, s);
}
template <>
__device__ __forceinline__ void dft<5>(float2 (&x)[5]) {
  const float c[2] = {0.30901699437494742410f, -0.80901699437494742410f};
  const float s[2] = {0.95105651629515357212f, 0.58778525229247312917f};
  dft_odd<5>(x, c, s);
}
template <>
__device__ __forceinline__ void dft<7>(float2 (&x)[7]) {
  const float c[3] = {0.62348980185873353053f, -0.22252093395631440429f, -0.90096886790241912624f};
  const float s[3] = {0.78183148246802980871f, 0.97492791218182360702f, 0.43388373911755812048f};
  dft_odd<7>(x, c, s);
}

// The twiddle exponents k that a stage's table holds, by slot: all of 1 .. R - 1,
// but for radices 8 and 16 only those from which one product gives the others
// (k = 4 b + a from 4 b and a).
__host__ __device__ constexpr int tw_slots(int R) { return R == 16 ? 6 : R == 8 ? 4 : R - 1; }
__host__ __device__ constexpr int tw_k(int R, int slot) {
  return R == 16 && slot >= 3 ? 4 * (slot - 2) : slot + 1;
}

// x[k] *= exp(-2 pi i j k / (R m)).
template <int R>
__device__ __forceinline__ void twiddle(float2 (&x)[R], const float2* __restrict__ tw, int m, int j) {
  constexpr int S = tw_slots(R);
  float2 w[S];
#pragma unroll
  for (int q = 0; q < S; q++) w[q] = __ldg(tw + q * m + j);
#pragma unroll
  for (int k = 1; k < R; k++) {
    if constexpr (R == 16) {
      const int a = k & 3, b = k >> 2;
      x[k] = cmul(x[k], b == 0 ? w[a - 1] : a == 0 ? w[2 + b] : cmul(w[2 + b], w[a - 1]));
    } else if constexpr (R == 8) {
      x[k] = cmul(x[k], k <= 4 ? w[k - 1] : cmul(w[3], w[k - 5]));
    } else {
      x[k] = cmul(x[k], w[k - 1]);
    }
  }
}

// The stages of a line by T threads, t of them this one.  First: elements from
// element(i, load(i)), a butterfly's loads all before the work on any of them;
// results into shared memory.
template <int R, class Load, class Element>
__device__ __forceinline__ void first_stage(float2* __restrict__ s, const FftPlan& p, int t, int T,
                                            Load load, Element element) {
  const int m = p.m[0];
  for (int j = t; j < m; j += T) {
    decltype(load(0)) raw[R];
#pragma unroll
    for (int k = 0; k < R; k++) raw[k] = load(j + k * m);
    float2 x[R];
#pragma unroll
    for (int k = 0; k < R; k++) x[k] = element(j + k * m, raw[k]);
    dft<R>(x);
    twiddle<R>(x, p.tw, m, j);
#pragma unroll
    for (int k = 0; k < R; k++) s[at(j + k * m)] = x[k];
  }
}

// In between: butterflies of R elements m apart, in place.
template <int R>
__device__ __forceinline__ void mid_stage(float2* __restrict__ s, const FftPlan& p, int q, int t,
                                          int T) {
  const int m = p.m[q], nb = p.n / R;
  const float2* tw = p.tw + p.tw_at[q];
  const uint32_t mul = p.mul[q];
  for (int b = t; b < nb; b += T) {
    const int blk = (int)__umulhi((uint32_t)b, mul);
    const int j = b - blk * m, base = blk * m * R + j;
    float2 x[R];
#pragma unroll
    for (int k = 0; k < R; k++) x[k] = s[at(base + k * m)];
    dft<R>(x);
    twiddle<R>(x, tw, m, j);
#pragma unroll
    for (int k = 0; k < R; k++) s[at(base + k * m)] = x[k];
  }
}

// Last: frequency f to store(f, value).
template <int R, class Store>
__device__ __forceinline__ void last_stage(const float2* __restrict__ s, const FftPlan& p, int t,
                                           int T, Store store) {
  const int nb = p.n / R;
  for (int b = t; b < nb; b += T) {
    const int f = __ldg(p.rev + b);
    float2 x[R];
#pragma unroll
    for (int k = 0; k < R; k++) x[k] = s[at(b * R + k)];
    dft<R>(x);
#pragma unroll
    for (int k = 0; k < R; k++) store(f + k * nb, x[k]);
  }
}

// The transform (exp(-2 pi i)) of the line whose element i is
// element(i, load(i)).
template <class Load, class Element, class Store>
__device__ __forceinline__ void line_fft(float2* __restrict__ s, const FftPlan& p, int t, int T,
                                         Load load, Element element, Store store) {
  switch (p.radix[0]) {
    case 16: first_stage<16>(s, p, t, T, load, element); break;
    case 8: first_stage<8>(s, p, t, T, load, element); break;
    case 4: first_stage<4>(s, p, t, T, load, element); break;
    case 3: first_stage<3>(s, p, t, T, load, element); break;
    case 5: first_stage<5>(s, p, t, T, load, element); break;
    default: first_stage<7>(s, p, t, T, load, element); break;
  }
  for (int q = 1; q < p.stages - 1; q++) {
    __syncthreads();
    switch (p.radix[q]) {
      case 16: mid_stage<16>(s, p, q, t, T); break;
      case 8: mid_stage<8>(s, p, q, t, T); break;
      case 4: mid_stage<4>(s, p, q, t, T); break;
      case 3: mid_stage<3>(s, p, q, t, T); break;
      case 5: mid_stage<5>(s, p, q, t, T); break;
      default: mid_stage<7>(s, p, q, t, T); break;
    }
  }
  __syncthreads();
  switch (p.radix[p.stages - 1]) {  // n is even: a power of two
    case 16: last_stage<16>(s, p, t, T, store); break;
    case 8: last_stage<8>(s, p, t, T, store); break;
    case 4: last_stage<4>(s, p, t, T, store); break;
    default: last_stage<2>(s, p, t, T, store); break;
  }
}

__device__ __forceinline__ float sign_of(int a) { return a & 1 ? -1.f : 1.f; }

// a / b.  A sky model is mostly zeros, for which the division would take its
// slow path.
__device__ __forceinline__ float correct(float a, float b) {
  if (a == 0.f && fabsf(b) > 0.f && fabsf(b) <= FLT_MAX) return b > 0.f ? a : -a;
  return a / b;
}

// Image rows 2 b and 2 b + 1, corrected and signed, as the real and imaginary
// part of one line; their half spectra are its even and odd parts.
template <int T>
__global__ void __launch_bounds__(T, kRowRegs / T)
    k_fft_rows_in(const float* __restrict__ x, const float* __restrict__ taper,
                  const __grid_constant__ FftPlan p, float2* __restrict__ g) {
  extern __shared__ __align__(16) float2 s[];
  const int n = p.n, i = 2 * blockIdx.x, t = threadIdx.x;
  float2* s2 = s + line(n);
  const float* x0 = x + (int64_t)i * n;
  const float* x1 = x0 + n;
  const float t0 = taper ? taper[i] : 1.f, t1 = taper ? taper[i + 1] : 1.f;
  line_fft(
      s, p, t, T,
      [&](int j) { return make_float3(__ldg(x0 + j), __ldg(x1 + j), taper ? __ldg(taper + j) : 1.f); },
      [&](int j, float3 q) {
        float a = q.x, b = q.y;
        if (taper) {
          a = correct(a, t0 * q.z);
          b = correct(b, t1 * q.z);
        }
        const float sg = sign_of(j);  // row i is even
        return make_float2(sg * a, -sg * b);
      },
      [&](int f, float2 a) { s2[at(f)] = a; });
  __syncthreads();
  float2* g0 = g + (int64_t)i * n;
  for (int v = t; v <= n / 2; v += T) {
    const float2 a = s2[at(v)], b = s2[at(v ? n - v : 0)];
    g0[v] = make_float2(0.5f * (a.x + b.x), 0.5f * (a.y - b.y));
    g0[n + v] = make_float2(0.5f * (a.y + b.y), 0.5f * (b.x - a.x));
  }
}

// C columns v0 .. of the half spectrum, in place, and their mirror columns.
template <int C>
__global__ void __launch_bounds__(kColThreads, 1)
    k_fft_cols_out(const __grid_constant__ FftPlan p, float2* __restrict__ g) {
  extern __shared__ __align__(16) float2 s[];
  const int n = p.n, h = n / 2;
  const int c = threadIdx.x % C, t = threadIdx.x / C, v = C * blockIdx.x + c;
  const int vl = min(v, h);  // the last CTA's spare columns transform a copy
  line_fft(
      s + c * line(n), p, t, kColThreads / C, [&](int u) { return g[(int64_t)u * n + vl]; },
      [](int, float2 a) { return a; },
      [&](int u, float2 a) {
        if (v > h) return;
        const float sg = sign_of(u + v);
        a.x *= sg;
        a.y *= sg;
        g[(int64_t)u * n + v] = a;
        if (v > 0 && v < h) g[(int64_t)(u ? n - u : 0) * n + (n - v)] = make_float2(a.x, -a.y);
      });
}

// The Hermitian half of the grid's columns v0 .., transformed (exp(+2 pi i):
// real and imaginary parts trade places on the way in and out) into w.
template <int C>
__global__ void __launch_bounds__(kColThreads, 1)
    k_fft_cols_in(const float2* __restrict__ g, const __grid_constant__ FftPlan p,
                  float2* __restrict__ w) {
  extern __shared__ __align__(16) float2 s[];
  const int n = p.n, h = n / 2;
  const int c = threadIdx.x % C, t = threadIdx.x / C, v = C * blockIdx.x + c;
  const int vl = min(v, h), vm = vl ? n - vl : 0;
  line_fft(
      s + c * line(n), p, t, kColThreads / C,
      [&](int u) {
        const float2 a = __ldg(g + (int64_t)u * n + vl);
        const float2 b = __ldg(g + (int64_t)(u ? n - u : 0) * n + vm);
        return make_float2(a.y - b.y, a.x + b.x);
      },
      [&](int u, float2 a) {
        const float sg = 0.5f * sign_of(u + vl);
        return make_float2(sg * a.x, sg * a.y);
      },
      [&](int i, float2 a) {
        if (v <= h) w[(int64_t)i * n + v] = make_float2(a.y, a.x);
      });
}

constexpr int kOut = 4;  // pixels of a row that a thread takes together

// Rows 2 b and 2 b + 1 of w, Hermitian along v, as one complex line: its
// transform's real part is the first image row, its imaginary part the second.
template <int T>
__global__ void __launch_bounds__(T, kRowRegs / T)
    k_fft_rows_out(const float2* __restrict__ w, const float* __restrict__ taper,
                   const __grid_constant__ FftPlan p, float* __restrict__ x) {
  extern __shared__ __align__(16) float2 s[];
  const int n = p.n, h = n / 2, i = 2 * blockIdx.x, t = threadIdx.x;
  float2* s2 = s + line(n);
  const float2* w0 = w + (int64_t)i * n;
  line_fft(
      s, p, t, T,
      [&](int v) {
        const int u = v <= h ? v : n - v;
        const float2 a = __ldg(w0 + u), b = __ldg(w0 + n + u);
        return make_float4(a.x, a.y, b.x, b.y);
      },
      [&](int v, float4 q) {
        float2 a = make_float2(q.x, q.y), b = make_float2(q.z, q.w);
        const float cj = v == 0 || v == h ? 0.f : v < h ? 1.f : -1.f;  // real at 0 and n / 2
        a.y = cj == 0.f ? 0.f : cj * a.y;
        b.y = cj == 0.f ? 0.f : cj * b.y;
        return make_float2(a.y + b.x, a.x - b.y);
      },
      [&](int f, float2 a) { s2[at(f)] = a; });
  __syncthreads();
  float* x0 = x + (int64_t)i * n;
  const float t0 = taper ? taper[i] : 1.f, t1 = taper ? taper[i + 1] : 1.f;
  for (int j0 = t; j0 < n; j0 += kOut * T) {
    float2 a[kOut];
    float tj[kOut];
#pragma unroll
    for (int k = 0; k < kOut; k++) {
      const int j = min(j0 + k * T, n - 1);
      a[k] = s2[at(j)];
      tj[k] = taper ? __ldg(taper + j) : 1.f;
    }
#pragma unroll
    for (int k = 0; k < kOut; k++) {
      const int j = j0 + k * T;
      const float sg = sign_of(j);
      const float u = sg * a[k].y, v = -sg * a[k].x;
      if (j < n) {
        x0[j] = taper ? correct(u, t0 * tj[k]) : u;
        x0[n + j] = taper ? correct(v, t1 * tj[k]) : v;
      }
    }
  }
}

// ---------------------------------------------------------------- tables
// The twiddles and the digit-reversal table of a size, made on first use
// and kept: at most a few hundred sizes have tables, of 10 n bytes each.
bool factor(int n, FftPlan* p) {
  int rest = n, q = 0;
  auto take = [&](int r) {
    while (rest % r == 0 && q < kMaxStages) {
      p->radix[q++] = r;
      rest /= r;
    }
  };
  // the odd radices first: the later stages, whose butterflies lie close
  // together, are then powers of two; at least two stages
  for (int r : {7, 5, 3}) take(r);
  int e = 0;
  for (; rest % 2 == 0; rest /= 2) e++;
  if (rest != 1 || q + (e + 3) / 4 > kMaxStages) return false;
  for (; e > 0; q++) {
    const int k = e == 4 && q == 0 ? 2 : e == 5 ? 3 : std::min(e, 4);
    p->radix[q] = 1 << k;
    e -= k;
  }
  if (q < 2) return false;
  p->n = n;
  p->stages = q;
  int m = n;
  for (int k = 0; k < q; k++) {
    m /= p->radix[k];
    p->m[k] = m;
    p->mul[k] = (uint32_t)(((1ull << 32) + m - 1) / m);
  }
  return true;
}

// Two host arrays into device memory, there for every stream once this returns: a
// plain cudaMemcpy from pageable memory may return when the data is staged, and
// runs on the default stream, which non-blocking streams do not wait for.
cudaError_t upload(void* d0, const void* h0, size_t n0, void* d1, const void* h1, size_t n1) {
  cudaStream_t up;
  cudaError_t e = cudaStreamCreateWithFlags(&up, cudaStreamNonBlocking);
  if (e != cudaSuccess) return e;
  e = cudaMemcpyAsync(d0, h0, n0, cudaMemcpyHostToDevice, up);
  if (e == cudaSuccess) e = cudaMemcpyAsync(d1, h1, n1, cudaMemcpyHostToDevice, up);
  const cudaError_t w = cudaStreamSynchronize(up);  // also where the second copy failed
  cudaStreamDestroy(up);
  return e != cudaSuccess ? e : w;
}

int fft_tables(int n, FftPlan* out) {
  static std::mutex mu;
  static std::map<std::pair<int, int>, FftPlan> plans;
  int dev = 0;
  GB_CUDA_TRY(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(mu);
  const auto key = std::make_pair(dev, n);
  const auto it = plans.find(key);
  if (it != plans.end()) {
    *out = it->second;
    return GB_OK;
  }
  FftPlan p;
  if (!factor(n, &p)) return GB_ERR_ARG;
  std::vector<float2> tw;
  tw.reserve(n);
  for (int q = 0; q < p.stages - 1; q++) {
    p.tw_at[q] = (int)tw.size();
    for (int k = 0; k < tw_slots(p.radix[q]); k++)
      for (int j = 0; j < p.m[q]; j++) {
        const double a = -2.0 * 3.141592653589793238462643383279502884 * j *
                         tw_k(p.radix[q], k) / ((double)p.radix[q] * p.m[q]);
        tw.push_back(make_float2((float)cos(a), (float)sin(a)));
      }
  }
  tw.resize(n);  // (a stage has fewer than R m entries, all stages fewer than n)
  const int last = p.radix[p.stages - 1];
  std::vector<uint16_t> rev(n / last);
  for (int b = 0; b < n / last; b++) {
    int f = 0, weight = 1;
    for (int q = 0; q < p.stages - 1; q++) {
      f += b * last / p.m[q] % p.radix[q] * weight;
      weight *= p.radix[q];
    }
    rev[b] = (uint16_t)f;
  }
  // A first call may come while a stream of this or another thread is captured:
  // the allocation and the copy are no part of that.
  struct Relaxed {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    Relaxed() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~Relaxed() { cudaThreadExchangeStreamCaptureMode(&mode); }
  } relaxed;
  void* d = nullptr;
  const int rc = dev_alloc(&d, sizeof(float2) * n + sizeof(uint16_t) * n, "FFT tables");
  if (rc) return rc;
  p.tw = (const float2*)d;
  p.rev = (const uint16_t*)(p.tw + n);
  const cudaError_t e = upload((void*)p.tw, tw.data(), sizeof(float2) * n, (void*)p.rev, rev.data(),
                               sizeof(uint16_t) * rev.size());
  if (e != cudaSuccess) {
    cudaFree(d);
    GB_CUDA_TRY(e);
  }
  plans[key] = p;
  *out = p;
  return GB_OK;
}

size_t line_bytes(int n, int lines) { return sizeof(float2) * (size_t)line(n) * lines; }

constexpr size_t kFftSmem = 224 * 1024;

// Columns per CTA: four where they fit (a row of them is one 32-byte sector).
int columns(int n) { return line_bytes(n, 4) <= kFftSmem ? 4 : 2; }

// Threads for a pair of rows: 256, and 512 where two CTAs' lines do not fit an SM.
int row_threads(int n) { return line_bytes(n, 4) <= kFftSmem ? 256 : 512; }

// The kernels' shared-memory limit, set once per device.
int set_limits() {
  static std::mutex mu;
  static bool done[64];
  int dev = 0;
  GB_CUDA_TRY(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(mu);
  if (dev >= 0 && dev < 64 && done[dev]) return GB_OK;
  for (const void* fn : {(const void*)k_fft_rows_in<256>, (const void*)k_fft_rows_in<512>,
                         (const void*)k_fft_rows_out<256>, (const void*)k_fft_rows_out<512>,
                         (const void*)k_fft_cols_out<4>, (const void*)k_fft_cols_out<2>,
                         (const void*)k_fft_cols_in<4>, (const void*)k_fft_cols_in<2>})
    GB_CUDA_TRY(
        cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFftSmem));
  if (dev >= 0 && dev < 64) done[dev] = true;
  return GB_OK;
}

}  // namespace

bool fft_size_ok(int n) {
  FftPlan p;
  return n >= 16 && n <= 8192 && n % 2 == 0 && factor(n, &p);
}

int fft_image_to_grid(const float* x, const float* taper, int n, float2* g, cudaStream_t s) {
  FftPlan p;
  int rc = fft_tables(n, &p);
  if (rc) return rc;
  const int C = columns(n), groups = (n / 2 + C) / C;
  if ((rc = set_limits())) return rc;
  if (row_threads(n) == 256)
    k_fft_rows_in<256><<<n / 2, 256, line_bytes(n, 2), s>>>(x, taper, p, g);
  else
    k_fft_rows_in<512><<<n / 2, 512, line_bytes(n, 2), s>>>(x, taper, p, g);
  if (C == 4)
    k_fft_cols_out<4><<<groups, kColThreads, line_bytes(n, 4), s>>>(p, g);
  else
    k_fft_cols_out<2><<<groups, kColThreads, line_bytes(n, 2), s>>>(p, g);
  GB_CUDA_TRY(cudaGetLastError());
  return GB_OK;
}

int fft_grid_to_image(const float2* g, const float* taper, int n, float2* w, float* x,
                      cudaStream_t s) {
  FftPlan p;
  int rc = fft_tables(n, &p);
  if (rc) return rc;
  const int C = columns(n), groups = (n / 2 + C) / C;
  if ((rc = set_limits())) return rc;
  if (C == 4)
    k_fft_cols_in<4><<<groups, kColThreads, line_bytes(n, 4), s>>>(g, p, w);
  else
    k_fft_cols_in<2><<<groups, kColThreads, line_bytes(n, 2), s>>>(g, p, w);
  if (row_threads(n) == 256)
    k_fft_rows_out<256><<<n / 2, 256, line_bytes(n, 2), s>>>(w, taper, p, x);
  else
    k_fft_rows_out<512><<<n / 2, 512, line_bytes(n, 2), s>>>(w, taper, p, x);
  GB_CUDA_TRY(cudaGetLastError());
  return GB_OK;
}

}  // namespace gb
