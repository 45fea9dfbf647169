// On-GPU w-kernel (GCF) generation, FP64.
//
// Semantics: the reference's GCF generator, MS4/kernel/cpu/gcf/GCF.cpp
// (screen :58-97, per-phase normalisation and extraction :16-52) with its
// centred backward FFT (MS4/kernel/cpu/fft/fft_dyn_padded.cpp:76-103:
// fftshift, unnormalised exp(+2 pi i) transform, fftshift), and the MS4 GPU
// kernels' split into screen / FFT / extract steps (MS4/kernel/gpu/gcf/
// GCF.cu:9-128).  The output layout is the MS6 one the gridders read:
// [ou + 8 ov][sy][sx].
//
// What is wanted of a plane is 8 S_p x 8 S_p of the (8 Smax)^2 samples of the
// transform of an Smax x Smax screen.  For the phase ou of the first axis,
//   F(8 a + ou) = sum_k (f(k) exp(2 pi i k ou / N)) exp(2 pi i k a / Smax),
// N = 8 Smax: eight transforms of length Smax of the screen turned by a phase,
// and likewise along the second axis.  So where Smax has no prime factor above 7:
//   k_gcf_first    the screen, eight columns at a time in shared memory, and the
//                  eight phases' transforms along the first axis; the S_p
//                  central samples of each into a work array;
//   k_gcf_second   eight lines of the work array at a time, the eight phases'
//                  transforms along the second axis, the S_p central samples of
//                  each, normalised, written as complex128 and/or complex64.
// The sum of a phase's real parts over the whole arena needs no arena: summed
// over a, the exponentials leave only k = 0, Smax^2 times the screen's centre.
// FP64 arithmetic bounds both kernels (the part's FP64 rate is 1/64 of its FP32
// rate); padded transforms of N x N by cuFFT do 2.5 times the arithmetic and move
// 134 MB through four passes.  32 planes, Smax 64, supports 8 to 64: 444 us of
// kernels against 1330 us, and 770 against 2310 us for the whole call, which made
// a 134 MB arena and a cuFFT plan each time.
//
// Other Smax, per batch of planes:
//   k_gcf_screen   screen(l, m) = taper(l) taper(m) (cos 2 pi ph, -sin 2 pi ph),
//                  ph = w (1 - sqrt(1 - l^2 - m^2)), written straight into the
//                  fftshift-ed position of a zeroed (8 Smax)^2 arena;
//   cufftExecZ2Z   CUFFT_INVERSE (exp(+2 pi i), unnormalised), batched;
//   k_gcf_sums     per (plane, phase) sum of real parts over the whole arena
//                  (the output's fftshift is an index map, applied on read);
//   k_gcf_extract  centred S_p x S_p taps per phase, divided by the phase
//                  sum, written as complex128 and/or complex64.
#include <cufft.h>

#include <algorithm>
#include <vector>

#include "gb_common.cuh"
#include "gb_runtime.cuh"

namespace gb {

struct GcfPlaneDev {
  double w;
  int32_t S;
  int64_t off;
};

// arena index of the fftshift-ed array for even N: (k + N/2) mod N
__device__ __forceinline__ int shift_idx(int k, int N) {
  const int h = N / 2;
  return k + h < N ? k + h : k + h - N;
}

__global__ void k_gcf_screen(const GcfPlaneDev* __restrict__ planes, int p0, int smax, int N,
                             double t2, const double* __restrict__ taper,
                             double2* __restrict__ arena) {
  const int b = blockIdx.z;
  const double w = planes[p0 + b].w;
  const int r = smax / 2;
  const double normer = t2 / (double)r;
  const int a0 = N / 2 - r;
  for (int ii = blockIdx.y * blockDim.y + threadIdx.y; ii < smax; ii += gridDim.y * blockDim.y)
    for (int jj = blockIdx.x * blockDim.x + threadIdx.x; jj < smax;
         jj += gridDim.x * blockDim.x) {
      const double x = (double)(ii - r) * normer;
      const double y = (double)(jj - r) * normer;
      const double ph = w * (1.0 - sqrt(1.0 - x * x - y * y));
      double s, c;
      sincos(2.0 * 3.141592653589793238462643383279502884 * ph, &s, &c);
      double tw = 1.0;
      if (taper) tw = taper[ii] * taper[jj];
      const int row = shift_idx(a0 + ii, N), col = shift_idx(a0 + jj, N);
      arena[(int64_t)b * N * N + (int64_t)row * N + col] = make_double2(c * tw, -s * tw);
    }
}

// ---------------------------------------------------------------- pruned transforms
constexpr int kGcfLines = 8;      // lines that a block transforms together
constexpr int kGcfThreads = 128;
constexpr int kGcfStages = 8;
// A block's shared memory: its lines of M values, before and after a transform.
constexpr size_t gcf_smem(int M) { return sizeof(double2) * 2 * kGcfLines * (M + 1); }
constexpr int kGcfSmem = (int)gcf_smem(GB_MAX_SUPPORT);

struct GcfFft {
  int M, N, stages;
  int radix[kGcfStages], m[kGcfStages];
  uint8_t pos[GB_MAX_SUPPORT];  // where frequency f of a line ends up
};

__device__ __forceinline__ double2 zadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 zsub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 zmul(double2 a, double2 b) {
  return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ double2 zrot(double2 a) { return make_double2(-a.y, a.x); }  // i a

// The transform exp(+2 pi i) of R values; `w` the roots exp(2 pi i t / N).
template <int R>
__device__ __forceinline__ void zdft(double2 (&x)[R], const double2* __restrict__ w, int N) {
  if constexpr (R == 2) {
    const double2 a = x[0];
    x[0] = zadd(a, x[1]);
    x[1] = zsub(a, x[1]);
  } else if constexpr (R == 4) {
    const double2 a = zadd(x[0], x[2]), b = zsub(x[0], x[2]);
    const double2 c = zadd(x[1], x[3]), d = zrot(zsub(x[1], x[3]));
    x[0] = zadd(a, c);
    x[1] = zadd(b, d);
    x[2] = zsub(a, c);
    x[3] = zsub(b, d);
  } else {  // 3, 5, 7: the sum itself
    double2 y[R];
#pragma unroll
    for (int f = 0; f < R; f++) {
      y[f] = x[0];
#pragma unroll
      for (int k = 1; k < R; k++)
        y[f] = zadd(y[f], f == 0 ? x[k] : zmul(x[k], __ldg(w + f * k % R * (N / R))));
    }
#pragma unroll
    for (int f = 0; f < R; f++) x[f] = y[f];
  }
}

// One stage of the block's lines, in place.
template <int R>
__device__ __forceinline__ void zstage(double2* __restrict__ s, int ld, const GcfFft& p, int q,
                                       const double2* __restrict__ w) {
  const int m = p.m[q], nb = p.M / R, step = p.N / (R * m);
  for (int e = threadIdx.x; e < kGcfLines * nb; e += kGcfThreads) {
    const int l = e / nb, b = e - l * nb, blk = b / m, j = b - blk * m;
    double2* z = s + l * ld + blk * m * R + j;
    double2 x[R];
#pragma unroll
    for (int k = 0; k < R; k++) x[k] = z[k * m];
    zdft<R>(x, w, p.N);
    if (m > 1) {
#pragma unroll
      for (int k = 1; k < R; k++) x[k] = zmul(x[k], __ldg(w + j * k * step));
    }
#pragma unroll
    for (int k = 0; k < R; k++) z[k * m] = x[k];
  }
}

// dst = the transforms of the lines of src (value k - M/2 at place k) turned by
// the phase o / N per step; frequency f at dst[pos[f]].
__device__ __forceinline__ void phase_fft(const double2* __restrict__ src, double2* __restrict__ dst,
                                          int ld, const GcfFft& p, int o,
                                          const double2* __restrict__ w) {
  const int M = p.M, r = M / 2;
  for (int e = threadIdx.x; e < kGcfLines * M; e += kGcfThreads) {
    const int l = e / M, i = e - l * M, k = i - r;
    const double2 v = src[l * ld + i];
    const int t = k * o;
    dst[l * ld + (k < 0 ? k + M : k)] = o ? zmul(v, __ldg(w + (t < 0 ? t + p.N : t))) : v;
  }
  for (int q = 0; q < p.stages; q++) {
    __syncthreads();
    switch (p.radix[q]) {
      case 4: zstage<4>(dst, ld, p, q, w); break;
      case 2: zstage<2>(dst, ld, p, q, w); break;
      case 3: zstage<3>(dst, ld, p, q, w); break;
      case 5: zstage<5>(dst, ld, p, q, w); break;
      default: zstage<7>(dst, ld, p, q, w); break;
    }
  }
  __syncthreads();
}

__global__ void k_gcf_roots(int N, double2* __restrict__ w) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= N) return;
  double s, c;
  sincospi(2.0 * t / N, &s, &c);
  w[t] = make_double2(c, s);
}

// block (x: group of kGcfLines screen columns, y: plane of the batch): g[plane]
// [ou][sx][jj], rows of M.
__global__ void __launch_bounds__(kGcfThreads)
    k_gcf_first(const GcfPlaneDev* __restrict__ planes, int p0, const __grid_constant__ GcfFft p,
                double t2, const double* __restrict__ taper, const double2* __restrict__ w,
                int64_t plane_stride, double2* __restrict__ g) {
  extern __shared__ __align__(16) double2 sm[];
  const int M = p.M, r = M / 2, ld = M + 1, j0 = blockIdx.x * kGcfLines;
  double2 *src = sm, *dst = sm + kGcfLines * ld;
  const GcfPlaneDev pl = planes[p0 + blockIdx.y];
  const double normer = t2 / (double)r;
  for (int e = threadIdx.x; e < kGcfLines * M; e += kGcfThreads) {
    const int l = e / M, ii = e - l * M, jj = j0 + l;
    double2 v = make_double2(0.0, 0.0);
    if (jj < M) {
      const double x = (double)(ii - r) * normer;
      const double y = (double)(jj - r) * normer;
      const double ph = pl.w * (1.0 - sqrt(1.0 - x * x - y * y));
      double s, c;
      sincos(2.0 * 3.141592653589793238462643383279502884 * ph, &s, &c);
      double tw = 1.0;
      if (taper) tw = taper[ii] * taper[jj];
      v = make_double2(c * tw, -s * tw);
    }
    src[l * ld + ii] = v;
  }
  __syncthreads();
  double2* out = g + blockIdx.y * plane_stride;
  const int S = pl.S;
  for (int ou = 0; ou < GB_OVER; ou++) {
    phase_fft(src, dst, ld, p, ou, w);
    for (int e = threadIdx.x; e < kGcfLines * S; e += kGcfThreads) {
      const int sx = e / kGcfLines, l = e - sx * kGcfLines, a = sx - S / 2;
      if (j0 + l < M)
        out[((int64_t)ou * S + sx) * M + j0 + l] = dst[l * ld + p.pos[a < 0 ? a + M : a]];
    }
    __syncthreads();
  }
}

// block (x: group of kGcfLines lines sx, y: phase ou, z: plane of the batch).
__global__ void __launch_bounds__(kGcfThreads)
    k_gcf_second(const GcfPlaneDev* __restrict__ planes, int p0, const __grid_constant__ GcfFft p,
                 const double* __restrict__ taper, const double2* __restrict__ w,
                 int64_t plane_stride, const double2* __restrict__ g, double2* __restrict__ out64,
                 float2* __restrict__ out32) {
  extern __shared__ __align__(16) double2 sm[];
  const GcfPlaneDev pl = planes[p0 + blockIdx.z];
  const int M = p.M, S = pl.S, ld = M + 1, x0 = blockIdx.x * kGcfLines, ou = blockIdx.y;
  if (x0 >= S) return;
  double2 *src = sm, *dst = sm + kGcfLines * ld;
  const double2* in = g + blockIdx.z * plane_stride + ((int64_t)ou * S + x0) * M;
  for (int e = threadIdx.x; e < kGcfLines * M; e += kGcfThreads) {
    const int l = e / M, i = e - l * M;
    src[l * ld + i] = x0 + l < S ? in[(int64_t)l * M + i] : make_double2(0.0, 0.0);
  }
  // one over the phase's sum: M^2 times the screen's centre, where w has no part
  const double t0 = taper ? taper[M / 2] : 1.0;
  const double inv = 1.0 / ((double)M * M * (t0 * t0));
  __syncthreads();
  for (int ov = 0; ov < GB_OVER; ov++) {
    phase_fft(src, dst, ld, p, ov, w);
    const int64_t o = pl.off + (int64_t)(ou + GB_OVER * ov) * S * S + x0;
    for (int e = threadIdx.x; e < kGcfLines * S; e += kGcfThreads) {
      const int sy = e / kGcfLines, l = e - sy * kGcfLines, a = sy - S / 2;
      if (x0 + l >= S) continue;
      const double2 v = dst[l * ld + p.pos[a < 0 ? a + M : a]];
      const double2 q = make_double2(v.x * inv, v.y * inv);
      if (out64) out64[o + (int64_t)sy * S + l] = q;
      if (out32) out32[o + (int64_t)sy * S + l] = make_float2((float)q.x, (float)q.y);
    }
    __syncthreads();
  }
}

// one block per (plane in batch, phase): sum of real parts of the final
// (fftshift-ed) arena at rows == ou (mod 8), columns == ov (mod 8).
__global__ void k_gcf_sums(const double2* __restrict__ arena, int N, double* __restrict__ sums) {
  const int b = blockIdx.y;
  const int ph = blockIdx.x;  // ou * 8 + ov
  const int ou = ph / GB_OVER, ov = ph % GB_OVER;
  const int n8 = N / GB_OVER;
  double acc = 0.0;
  for (int64_t e = threadIdx.x; e < (int64_t)n8 * n8; e += blockDim.x) {
    const int rf = (int)(e / n8) * GB_OVER + ou;
    const int cf = (int)(e % n8) * GB_OVER + ov;
    acc += arena[(int64_t)b * N * N + (int64_t)shift_idx(rf, N) * N + shift_idx(cf, N)].x;
  }
  __shared__ double red[256];
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if ((int)threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) sums[b * GB_PHASES + ph] = red[0];
}

// dst[off + (ou + 8 ov) S^2 + sy S + sx] =
//   final[(c + sx) 8 + ou][(c + sy) 8 + ov] / sums[ou][ov],  c = smax/2 - S/2
__global__ void k_gcf_extract(const GcfPlaneDev* __restrict__ planes, int p0, int smax, int N,
                              const double2* __restrict__ arena, const double* __restrict__ sums,
                              double2* __restrict__ out64, float2* __restrict__ out32) {
  const int b = blockIdx.y;
  const GcfPlaneDev pl = planes[p0 + b];
  const int S = pl.S;
  const int c = smax / 2 - S / 2;
  const int64_t n = (int64_t)GB_PHASES * S * S;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int phase = (int)(e / ((int64_t)S * S));
    const int rem = (int)(e - (int64_t)phase * S * S);
    const int sy = rem / S, sx = rem - sy * S;
    const int ou = phase % GB_OVER, ov = phase / GB_OVER;
    const int rf = (c + sx) * GB_OVER + ou, cf = (c + sy) * GB_OVER + ov;
    const double2 v = arena[(int64_t)b * N * N + (int64_t)shift_idx(rf, N) * N + shift_idx(cf, N)];
    const double d = sums[b * GB_PHASES + ou * GB_OVER + ov];
    const double2 q = make_double2(v.x / d, v.y / d);
    if (out64) out64[pl.off + e] = q;
    if (out32) out32[pl.off + e] = make_float2((float)q.x, (float)q.y);
  }
}

}  // namespace gb

using namespace gb;

#define GB_CUFFT_TRY(expr)                                                           \
  do {                                                                               \
    cufftResult _r = (expr);                                                         \
    if (_r != CUFFT_SUCCESS) {                                                       \
      gb_set_error(GB_ERR_CUDA, "%s:%d %s: cuFFT error %d", __FILE__, __LINE__, #expr, \
                   (int)_r);                                                         \
      rc = GB_ERR_CUDA;                                                              \
      goto done;                                                                     \
    }                                                                                \
  } while (0)

#define GB_CUDA_GOTO(expr)                                                           \
  do {                                                                               \
    cudaError_t _e = (expr);                                                         \
    if (_e != cudaSuccess) {                                                         \
      gb_set_error(GB_ERR_CUDA, "%s:%d %s: %s", __FILE__, __LINE__, #expr,             \
                   cudaGetErrorString(_e));                                          \
      rc = GB_ERR_CUDA;                                                              \
      goto done;                                                                     \
    }                                                                                \
  } while (0)

// The stages of a transform of length M, or false where a prime factor is above 7.
static bool gcf_factor(int M, GcfFft* p) {
  p->M = M;
  p->N = GB_OVER * M;
  p->stages = 0;
  int rest = M;
  for (int r : {7, 5, 3, 4, 2})
    for (; rest % r == 0; rest /= r) {
      if (p->stages == kGcfStages) return false;
      p->radix[p->stages++] = r;
    }
  if (rest != 1) return false;
  int m = M;
  for (int q = 0; q < p->stages; q++) p->m[q] = m /= p->radix[q];
  for (int f = 0; f < M; f++) {
    int at = 0, v = f;
    for (int q = 0; q < p->stages; v /= p->radix[q++]) at += v % p->radix[q] * p->m[q];
    p->pos[f] = (uint8_t)at;
  }
  return true;
}

// Generation by the pruned transforms.  One allocation: the planes, the roots and
// the work array of a batch of planes (at most about 256 MiB).
static int gcf_pruned(const std::vector<GcfPlaneDev>& hp, const GcfFft& p, double t2,
                      const double* d_taper, double* d_gcf64, float* d_gcf32, cudaStream_t s) {
  const int n_planes = (int)hp.size();
  int smax = 0;
  for (const auto& q : hp) smax = std::max(smax, q.S);
  const int64_t stride = (int64_t)GB_OVER * smax * p.M;
  const int batch = (int)std::clamp<int64_t>(((int64_t)1 << 28) / (stride * 16), 1,
                                             std::min(n_planes, 32768));
  const size_t planes_bytes = (sizeof(GcfPlaneDev) * n_planes + 255) & ~(size_t)255;
  const size_t roots_bytes = sizeof(double2) * p.N;
  unsigned char* d = nullptr;
  int rc = dev_alloc((void**)&d, planes_bytes + roots_bytes + sizeof(double2) * stride * batch,
                     "GCF generation");
  if (rc) return rc;
  GcfPlaneDev* d_planes = (GcfPlaneDev*)d;
  double2* w = (double2*)(d + planes_bytes);
  double2* g = w + p.N;
  const size_t smem = gcf_smem(p.M);
  // the limit is the kernels', not this call's: the same for every support, so that
  // calls of other threads cannot lower it below what this one launches with
  GB_CUDA_GOTO(cudaFuncSetAttribute(k_gcf_first, cudaFuncAttributeMaxDynamicSharedMemorySize, kGcfSmem));
  GB_CUDA_GOTO(cudaFuncSetAttribute(k_gcf_second, cudaFuncAttributeMaxDynamicSharedMemorySize, kGcfSmem));
  GB_CUDA_GOTO(cudaMemcpyAsync(d_planes, hp.data(), sizeof(GcfPlaneDev) * n_planes,
                               cudaMemcpyHostToDevice, s));
  k_gcf_roots<<<(p.N + 255) / 256, 256, 0, s>>>(p.N, w);
  for (int p0 = 0; p0 < n_planes; p0 += batch) {
    const int nb = std::min(batch, n_planes - p0);
    k_gcf_first<<<dim3((p.M + kGcfLines - 1) / kGcfLines, nb), kGcfThreads, smem, s>>>(
        d_planes, p0, p, t2, d_taper, w, stride, g);
    k_gcf_second<<<dim3((smax + kGcfLines - 1) / kGcfLines, GB_OVER, nb), kGcfThreads, smem, s>>>(
        d_planes, p0, p, d_taper, w, stride, g, (double2*)d_gcf64, (float2*)d_gcf32);
    GB_CUDA_GOTO(cudaGetLastError());
  }
  GB_CUDA_GOTO(cudaStreamSynchronize(s));
done:
  cudaFree(d);
  return rc;
}

extern "C" int gb_gcf_generate(int32_t n_planes, const double* w_planes, const int32_t* supports,
                               const int64_t* gcf_offsets, int32_t max_support, double t2,
                               const double* d_taper, double* d_gcf64, float* d_gcf32,
                               void* stream) {
  if (n_planes < 1 || n_planes > GB_MAX_PLANES || !w_planes || !supports || !gcf_offsets ||
      max_support < 2 || max_support > GB_MAX_SUPPORT || (max_support & 1) || !(t2 > 0.0) ||
      (!d_gcf64 && !d_gcf32)) {
    gb_set_error(GB_ERR_ARG, "gb_gcf_generate: bad arguments (max_support must be even, 2..%d)",
                 GB_MAX_SUPPORT);
    return GB_ERR_ARG;
  }
  for (int p = 0; p < n_planes; p++) {
    if (supports[p] < 1 || supports[p] > max_support || gcf_offsets[p] < 0) {
      gb_set_error(GB_ERR_ARG, "gb_gcf_generate: plane %d support %d out of range", p, supports[p]);
      return GB_ERR_ARG;
    }
  }
  cudaStream_t s = (cudaStream_t)stream;
  std::vector<GcfPlaneDev> hp(n_planes);
  for (int p = 0; p < n_planes; p++) hp[p] = GcfPlaneDev{w_planes[p], supports[p], gcf_offsets[p]};
  GcfFft fft;
  if (gcf_factor(max_support, &fft)) return gcf_pruned(hp, fft, t2, d_taper, d_gcf64, d_gcf32, s);
  const int N = GB_OVER * max_support;
  const size_t arena_bytes = (size_t)N * N * sizeof(double2);
  // batch so that the FFT arenas stay within ~1 GiB
  int batch = (int)std::max<size_t>(1, ((size_t)1 << 30) / arena_bytes);
  batch = std::min(batch, n_planes);
  int rc = GB_OK;
  GcfPlaneDev* d_planes = nullptr;
  double2* arena = nullptr;
  double* sums = nullptr;
  cufftHandle plan = 0;
  bool have_plan = false;
  int nfft[2] = {N, N};
  if ((rc = dev_alloc((void**)&d_planes, sizeof(GcfPlaneDev) * n_planes, "GCF generation")) ||
      (rc = dev_alloc((void**)&arena, arena_bytes * batch, "GCF generation")) ||
      (rc = dev_alloc((void**)&sums, sizeof(double) * GB_PHASES * batch, "GCF generation")))
    goto done;
  GB_CUDA_GOTO(cudaMemcpyAsync(d_planes, hp.data(), sizeof(GcfPlaneDev) * n_planes,
                               cudaMemcpyHostToDevice, s));
  GB_CUFFT_TRY(cufftPlanMany(&plan, 2, nfft, nullptr, 1, N * N, nullptr, 1, N * N, CUFFT_Z2Z, batch));
  have_plan = true;
  GB_CUFFT_TRY(cufftSetStream(plan, s));
  for (int p0 = 0; p0 < n_planes; p0 += batch) {
    const int nb = std::min(batch, n_planes - p0);
    GB_CUDA_GOTO(cudaMemsetAsync(arena, 0, arena_bytes * batch, s));
    dim3 blk(32, 8), grd((max_support + 31) / 32, (max_support + 7) / 8, nb);
    k_gcf_screen<<<grd, blk, 0, s>>>(d_planes, p0, max_support, N, t2, d_taper, arena);
    GB_CUDA_GOTO(cudaGetLastError());
    // unused batch slots hold zeros: transforming them is harmless
    GB_CUFFT_TRY(cufftExecZ2Z(plan, (cufftDoubleComplex*)arena, (cufftDoubleComplex*)arena,
                              CUFFT_INVERSE));
    k_gcf_sums<<<dim3(GB_PHASES, nb), 256, 0, s>>>(arena, N, sums);
    GB_CUDA_GOTO(cudaGetLastError());
    k_gcf_extract<<<dim3(64, nb), 256, 0, s>>>(d_planes, p0, max_support, N, arena, sums,
                                              (double2*)d_gcf64, (float2*)d_gcf32);
    GB_CUDA_GOTO(cudaGetLastError());
  }
  GB_CUDA_GOTO(cudaStreamSynchronize(s));
done:
  if (have_plan) cufftDestroy(plan);
  cudaFree(d_planes);
  cudaFree(arena);
  cudaFree(sums);
  return rc;
}

// ---------------------------------------------------------------- GCF choice per w-region
// MS6/programs/Kernel/Config.hs:128-132: the GCF file with the largest w not
// above max(|w0|, |w1|) (maximumBy keeps the last of equal maxima); and
// MS6/programs/Kernel/IO.hs:110-113: conjugate when the region lies mostly at
// negative w (low < -high).
extern "C" int gb_gcf_select(int32_t n_files, const double* w_files, double w0, double w1,
                             int32_t* index, int32_t* conjugate) {
  if (n_files < 1 || !w_files || !index || !conjugate) {
    gb_set_error(GB_ERR_ARG, "gb_gcf_select: bad arguments");
    return GB_ERR_ARG;
  }
  const double w = fabs(w0) > fabs(w1) ? fabs(w0) : fabs(w1);
  int best = -1;
  for (int i = 0; i < n_files; i++)
    if (w_files[i] <= w && (best < 0 || w_files[i] >= w_files[best])) best = i;
  if (best < 0) {
    gb_set_error(GB_ERR_ARG, "gb_gcf_select: no GCF with w <= %g", w);
    return GB_ERR_ARG;
  }
  *index = best;
  *conjugate = w0 < -w1 ? 1 : 0;
  return GB_OK;
}

namespace gb {
template <class C>
__global__ void k_conjugate(C* __restrict__ g, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    g[i].y = -g[i].y;
}
}  // namespace gb

extern "C" int gb_gcf_conjugate_f32(float* d_gcf, int64_t n_complex, void* stream) {
  if (!d_gcf || n_complex < 0) {
    gb_set_error(GB_ERR_ARG, "gb_gcf_conjugate_f32: bad arguments");
    return GB_ERR_ARG;
  }
  if (!n_complex) return GB_OK;
  const int b = (int)std::min<int64_t>((n_complex + 255) / 256, 4096);
  k_conjugate<float2><<<b, 256, 0, (cudaStream_t)stream>>>((float2*)d_gcf, n_complex);
  GB_CUDA_TRY(cudaGetLastError());
  return GB_OK;
}

extern "C" int gb_gcf_conjugate_f64(double* d_gcf, int64_t n_complex, void* stream) {
  if (!d_gcf || n_complex < 0) {
    gb_set_error(GB_ERR_ARG, "gb_gcf_conjugate_f64: bad arguments");
    return GB_ERR_ARG;
  }
  if (!n_complex) return GB_OK;
  const int b = (int)std::min<int64_t>((n_complex + 255) / 256, 4096);
  k_conjugate<double2><<<b, 256, 0, (cudaStream_t)stream>>>((double2*)d_gcf, n_complex);
  GB_CUDA_TRY(cudaGetLastError());
  return GB_OK;
}
