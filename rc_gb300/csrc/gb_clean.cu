// Hogbom CLEAN on the GPU: the minor loop of the imaging major cycle.
//
// Engine form, gb_hogbom_f32 (FP32 residual/model/PSF): per iteration
//   peak   = residual pixel of largest |value| (ties: lowest row-major index)
//   stop   if |peak| < threshold (every later iteration is a no-op)
//   residual -= (gain * peak / psf_peak) * psf shifted so its peak sits on
//               the residual peak (zero outside the PSF)
//   model[peak] += gain * peak
// The whole loop is one cooperative launch (k_clean), which a CUDA graph can
// capture.  What an iteration needs is only the new peak, so the subtraction is
// lazy: the image is cut into 32 x 16 tiles, dealt out to the warps; a tile keeps
// the maximum it had when it was last brought up to date and an upper bound of
// what the components since then can have made of it (|s| times the largest
// |psf| over the part that covers the tile, rounded up, from a table of block
// maxima of the PSF's window that can lie on the image).  After a component the
// next peak is at least what is left at the old one, so only tiles whose bound
// reaches that are brought up to date: a few around the bright sources instead of
// the whole image.  The others take their pending components later, several per
// pass over their pixels (when a tile's bound rises, when the list of components is
// full, at the end), each pixel in the components' order, with unfused arithmetic
// (__fmul_rn / __fsub_rn), so every pixel and every peak is what a numpy float32
// loop computes, bit for bit.
// Per iteration each CTA publishes its best candidate and reads all the others'.
// Reference form, kern_hogbom_model / kern_hogbom_residual: the reference's
// Halide CLEAN (MS6/kernel/cpu/gridding/hogbom.cpp:10-109) restated on the GPU
// in FP64 with its own rules: 12 cycles; the "PSF peak" is the argmax of
// |residual| over the PSF's domain (hogbom.cpp:58); the peak value is the
// absolute value (hogbom.cpp:85-90); the PSF shift is clamped (:99-100); the
// model gets gain*|peak| (:108); the residual returned is the one of the cycle
// at which the threshold was first crossed, else the last (:68-74).
#include <float.h>
#include <limits.h>
#include <math.h>
#include <stddef.h>

#include <algorithm>

#include "gb_common.cuh"
#include "gb_runtime.cuh"

namespace gb {

constexpr int kCleanTile = 32;          // tile width: a lane holds one column of a tile
constexpr int kCleanRows = 16;          // tile height
constexpr int kCleanWarps = 16;         // of a CTA: the first trades candidates, the rest own tiles
constexpr int kCleanOwners = kCleanWarps - 1;
constexpr int kCleanThreads = 32 * kCleanWarps;
constexpr int kCleanPer = 5;            // candidates each lane of a warp reads
constexpr int kCleanCtas = 32 * kCleanPer;  // at most (one per SM)
constexpr int kCleanPending = 512;      // components a tile may lag behind
constexpr int kCleanLag = 4;            // components that an idle warp lets a tile lag behind
constexpr int kCleanPsfBlocks = 16384;  // entries of the PSF's block maxima, at most

__device__ __forceinline__ bool better(float a, int64_t ia, float b, int64_t ib) {
  return a > b || (a == b && ia < ib);
}

// A CTA's best pixel of an iteration: the largest |val| with the lowest
// row-major index (all ones: no pixel).  Each 8-byte word carries the
// iteration, so that a reader sees by itself whether the word is this
// iteration's: no barrier, counter or fence between writer and readers.
struct __align__(16) CleanCand {
  uint64_t val;  // float bits << 32 | iteration + 1
  uint64_t idx;  // index << 24 | (iteration + 1) mod 2^24
};
constexpr uint64_t kCleanNone = (1ull << 40) - 1;

// Start of the caller's work buffer, zeroed before the launch.
struct CleanState {
  uint32_t arrive;     // CTAs that have written their share of psf_max
  int32_t err;         // a bounded wait for the other CTAs ran out
  int32_t iterations;  // iterations that subtracted a component
  int32_t pad;
};
struct CleanWork {
  CleanState st;
  CleanCand cand[2][kCleanCtas];
  float psf_max[kCleanPsfBlocks];
};

// A warp's view of one of its tiles.
struct CleanTile {
  int64_t idx;  // where its maximum was when it was last up to date (-1: no pixel)
  float val;    // that pixel
  float ub;     // no pixel is larger than this now
  int32_t ver;    // components applied
  int32_t exact;  // the maximum still holds
  int32_t x0, y0;
};

struct CleanArgs {
  float* res;
  const float* psf;
  float* model;
  CleanWork* w;
  int nx, ny, pnx, pny, ppx, ppy;
  int ntx, ntiles, local;  // tiles across, in all, and per warp at most
  CleanTile* far_tiles;    // the warps' tiles where shared memory does not hold them, or NULL
  int wx0, wx1, wy0, wy1;  // the PSF's pixels that can lie on the image
  int eb, nbx, nby;        // their blocks of 2^eb x 2^eb pixels
  float gain, threshold;
  int n_iter;
};

struct CleanComp {
  int dx, dy;  // where the PSF's pixel (0, 0) lands
  float s;
};

struct CleanShared {
  CleanComp comp[kCleanPending];
  float val[kCleanWarps];    // the owners' candidates
  int64_t idx[kCleanWarps];  // (-1: none)
  int red[kCleanWarps];
  int stop;
  float peak;  // this iteration's
  int px, py;
};

// One component taken from a tile's column: rows r0 <= r < r1 of it are covered
// by the PSF (all of them in the common case, without a test per row).
__device__ __forceinline__ void clean_subtract(float (&v)[kCleanRows], const float* __restrict__ p,
                                               int pnx, int r0, int r1, float s) {
  float w[kCleanRows];
  if (r0 <= 0 && r1 >= kCleanRows) {
#pragma unroll
    for (int r = 0; r < kCleanRows; r++) w[r] = __ldg(p + (int64_t)r * pnx);
#pragma unroll
    for (int r = 0; r < kCleanRows; r++) v[r] = __fsub_rn(v[r], __fmul_rn(s, w[r]));
  } else {
#pragma unroll
    for (int r = 0; r < kCleanRows; r++)
      w[r] = r >= r0 && r < r1 ? __ldg(p + (int64_t)r * pnx) : 0.f;
#pragma unroll
    for (int r = 0; r < kCleanRows; r++)
      if (r >= r0 && r < r1) v[r] = __fsub_rn(v[r], __fmul_rn(s, w[r]));
  }
}

// A tile brought up to date by its warp: the components [ver, n) applied to its
// pixels and its maximum found again.
// (A call, not inlined at each use; its arguments by value, so that none is
// read back from memory.)
struct CleanImage {
  float* res;
  const float* psf;
  int nx, ny, pnx, pny;
};
__device__ __noinline__ void clean_refresh_call(CleanImage a, const CleanComp* comp, CleanTile* tile,
                                                int n) {
  const int lane = threadIdx.x & 31;
  CleanTile& d = *tile;
  const int x0 = d.x0, y0 = d.y0, ver = d.ver;
  const int rows = min(kCleanRows, a.ny - y0);
  const bool col = x0 + lane < a.nx;
  float* c0 = a.res + (int64_t)y0 * a.nx + x0 + lane;
  float v[kCleanRows];
  if (col && rows == kCleanRows) {
#pragma unroll
    for (int r = 0; r < kCleanRows; r++) v[r] = c0[(int64_t)r * a.nx];
  } else {
#pragma unroll
    for (int r = 0; r < kCleanRows; r++)
      v[r] = col && r < rows ? c0[(int64_t)r * a.nx] : __int_as_float(0x7FC00000);
  }
  bool changed = false;
  for (int c = ver; c < n; c++) {
    const CleanComp q = comp[c];
    const int px = x0 - q.dx, py = y0 - q.dy;  // of the tile in the PSF
    if (!(px < a.pnx && -kCleanTile < px && py < a.pny && -kCleanRows < py)) continue;
    changed = true;
    if ((unsigned)(px + lane) < (unsigned)a.pnx)
      clean_subtract(v, a.psf + (int64_t)py * a.pnx + px + lane, a.pnx, -py, a.pny - py, q.s);
  }
  if (changed) {
    if (col && rows == kCleanRows) {
#pragma unroll
      for (int r = 0; r < kCleanRows; r++) c0[(int64_t)r * a.nx] = v[r];
    } else {
#pragma unroll
      for (int r = 0; r < kCleanRows; r++)
        if (col && r < rows) c0[(int64_t)r * a.nx] = v[r];
    }
  }
  // the largest |v| (fmaxf passes over a NaN), then its first row and column:
  // within a tile those order like the row-major index
  float m = -1.f;
#pragma unroll
  for (int r = 0; r < kCleanRows; r++) m = fmaxf(m, fabsf(v[r]));
  // floats from -1 up order like the integers of their bits
  const int top = __reduce_max_sync(0xffffffffu, m < 0.f ? -1 : __float_as_int(m));
  const float best = __int_as_float(top);
  int row = INT_MAX / 32 - 1;
  float val = 0.f;
#pragma unroll
  for (int r = kCleanRows - 1; r >= 0; r--)
    if (fabsf(v[r]) == best) {
      row = r;
      val = v[r];
    }
  const int at = row * 32 + lane, first = __reduce_min_sync(0xffffffffu, at);
  if (top < 0 ? lane == 0 : at == first) {
    d.idx = top < 0 ? -1 : (int64_t)(y0 + row) * a.nx + x0 + lane;
    d.val = val;
    d.ub = top < 0 ? -1.f : best;
    d.ver = n;
    d.exact = 1;
  }
  __syncwarp();
}

__device__ __forceinline__ void clean_refresh(const CleanArgs& a, const CleanShared& sh,
                                              CleanTile& d, int n) {
  clean_refresh_call(CleanImage{a.res, a.psf, a.nx, a.ny, a.pnx, a.pny}, sh.comp, &d, n);
}

constexpr int kCleanPolls = 1 << 23;  // bound of every wait: seconds

// The Hogbom loop, up to one CTA per SM, cooperative.  An iteration is bound by
// latency: the update of the brightest tiles by their warps (their pixels and
// the PSF over them, one L2 round trip), and a candidate's way through L2 to
// the other CTAs; about 10 of the 8192 tiles are brought up to date for their
// own sake per iteration on a 2048^2 image of 30 sources.  There, with a 2048^2
// PSF, 200 iterations take 1.08 ms (3.59 ms as a launch per iteration that
// updated every tile under the PSF); 256^2, 164 iterations 0.57 ms (2.13 ms);
// 2048^2 with the strong sidelobes of 36 antennas, 135 iterations 0.79 ms (2.43
// ms).  Tiles of 32 x 16: a whole CTA per 64 x 64 tile took 1.94 ms, a warp per
// 32 x 32 tile 1.36 ms, 32 x 8 1.11 ms.  kCleanLag: 16 components 1.20 ms, 8
// 1.12 ms, 4 1.08 ms; without the idle warps' updates 3 ms and more.
__global__ void __launch_bounds__(kCleanThreads, 1) k_clean(const __grid_constant__ CleanArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ CleanShared sh;
  float* psf_max = (float*)smem;
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int ctas = (int)gridDim.x, owners = ctas * kCleanOwners;
  // owner o = (warp - 1) * ctas + block has the tiles o, o + owners, ...: tiles
  // side by side belong to different CTAs
  const int o = (warp - 1) * ctas + (int)blockIdx.x;
  const int nt = warp == 0 || o >= a.ntiles ? 0 : (a.ntiles - o + owners - 1) / owners;
  CleanTile* tiles = (a.far_tiles ? a.far_tiles + (int64_t)blockIdx.x * kCleanOwners * a.local
                                  : (CleanTile*)(psf_max + ((a.nbx * a.nby + 3) & ~3))) +
                     (int64_t)max(warp - 1, 0) * a.local;
  // the block maxima of the PSF's window (NaN pixels aside: they only make NaN
  // pixels), a warp to a block
  for (int b = (int)blockIdx.x + warp * ctas; b < a.nbx * a.nby; b += ctas * kCleanWarps) {
    const int bx = a.wx0 + (b % a.nbx << a.eb), by = a.wy0 + (b / a.nbx << a.eb);
    const int ex = min(bx + (1 << a.eb), a.wx1), ey = min(by + (1 << a.eb), a.wy1);
    float m = 0.f;
    for (int x = bx + lane; x < ex; x += 32)
      for (int y = by; y < ey; y += kCleanRows) {
        float v[kCleanRows];
#pragma unroll
        for (int r = 0; r < kCleanRows; r++)
          v[r] = __ldg(a.psf + (int64_t)min(y + r, ey - 1) * a.pnx + x);
#pragma unroll
        for (int r = 0; r < kCleanRows; r++) m = fmaxf(m, fabsf(v[r]));
      }
    const int wm = __reduce_max_sync(0xffffffffu, __float_as_int(m));
    if (lane == 0) a.w->psf_max[b] = __int_as_float(wm);
  }
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    atomicAdd(&a.w->st.arrive, 1u);
  }
  for (int k = lane; k < nt; k += 32) {
    const int t = o + k * owners;
    tiles[k].x0 = t % a.ntx * kCleanTile;
    tiles[k].y0 = t / a.ntx * kCleanRows;
    tiles[k].ver = 0;
  }
  __syncwarp();
  for (int k = 0; k < nt; k++) clean_refresh(a, sh, tiles[k], 0);
  if (tid == 0) {
    uint32_t v = 0;
    for (int p = 0; p < kCleanPolls && v < (uint32_t)ctas; p++)
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(&a.w->st.arrive) : "memory");
    sh.stop = v < (uint32_t)ctas;
    if (sh.stop) atomicExch(&a.w->st.err, 1);
  }
  __syncthreads();
  if (sh.stop) return;
  for (int b = tid; b < a.nbx * a.nby; b += kCleanThreads) psf_max[b] = __ldcg(&a.w->psf_max[b]);
  const float psf_peak = __ldg(a.psf + (int64_t)a.ppy * a.pnx + a.ppx);
  __syncthreads();
  int n = 0;        // components in the list
  int done = 0;     // iterations that subtracted one
  float lb = -1.f;  // the peak is at least this
  for (int it = 0; it < a.n_iter; it++) {
    int lag = -1;  // the warp's tile furthest behind, if by kCleanLag or more
    if (warp > 0) {
      // tiles that may hold the peak, largest bound first, until every other
      // one's bound is below the largest maximum found
      for (;;) {
        // bounds and maxima are -1, or not negative: their bits order like they
        int e = -1, f = -1, ek = -1, fk = -1, behind = kCleanLag - 1, lk = -1;
        for (int k = lane; k < nt; k += 32) {
          const CleanTile& d = tiles[k];
          const int u = d.ub < 0.f ? -1 : __float_as_int(d.ub);
          if (d.exact) {
            if (u >= 0 && (u > e || (u == e && d.idx < tiles[ek].idx))) {
              e = u;
              ek = k;
            }
          } else if (u > f) {
            f = u;
            fk = k;
          }
          if (n - d.ver > behind) {
            behind = n - d.ver;
            lk = k;
          }
        }
        const int be = __reduce_max_sync(0xffffffffu, e), bf = __reduce_max_sync(0xffffffffu, f);
        const int bl = lb < 0.f ? -1 : __float_as_int(lb);
        // a bound that only equals the best may hide an equal pixel before it
        if (bf >= 0 && bf >= max(be, bl)) {
          const int src = __ffs(__ballot_sync(0xffffffffu, f == bf)) - 1;
          clean_refresh(a, sh, tiles[__shfl_sync(0xffffffffu, fk, src)], n);
          continue;
        }
        unsigned tie = __ballot_sync(0xffffffffu, e == be);
        if (be < 0 || be < bl) {
          if (lane == 0) sh.idx[warp] = -1;
        } else {
          int64_t idx = -1;
          int bk = -1;
          while (tie) {  // mostly one lane
            const int k = __shfl_sync(0xffffffffu, ek, __ffs(tie) - 1);
            tie &= tie - 1;
            const int64_t i = tiles[k].idx;
            if (idx < 0 || i < idx) {
              idx = i;
              bk = k;
            }
          }
          if (lane == 0) {
            sh.idx[warp] = idx;
            sh.val[warp] = tiles[bk].val;
          }
        }
        const unsigned late = __ballot_sync(0xffffffffu, lk >= 0);
        if (late) lag = __shfl_sync(0xffffffffu, lk, __ffs(late) - 1);
        break;
      }
    }
    __syncthreads();
    if (warp > 0) {
      // while the candidates are traded: the tile that is furthest behind
      if (lag >= 0) clean_refresh(a, sh, tiles[lag], n);
    } else {
      float val = 0.f;
      int64_t idx = -1;
      if (lane > 0 && lane < kCleanWarps) {
        val = sh.val[lane];
        idx = sh.idx[lane];
      }
#pragma unroll
      for (int q = 8; q > 0; q >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, val, q);
        const int64_t oi = __shfl_xor_sync(0xffffffffu, idx, q);
        if (oi >= 0 && (idx < 0 || better(fabsf(ov), oi, fabsf(val), idx))) {
          val = ov;
          idx = oi;
        }
      }
      CleanCand* cand = a.w->cand[it & 1];
      const uint32_t tag = (uint32_t)(it + 1);
      if (lane == 0) {
        const uint64_t wv = (uint64_t)__float_as_uint(val) << 32 | tag;
        const uint64_t wi = (idx < 0 ? kCleanNone : (uint64_t)idx) << 24 | (tag & 0xFFFFFFu);
        asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(cand + blockIdx.x),
                     "l"(wv), "l"(wi)
                     : "memory");
      }
      val = 0.f;
      uint64_t best = kCleanNone;
      bool ok = true;
      // all of a lane's candidates are read at once, until all are there
      uint64_t cv[kCleanPer], ci[kCleanPer];
      for (int p = 0;; p++) {
        bool all = true;
#pragma unroll
        for (int i = 0; i < kCleanPer; i++)
          asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];"
                       : "=l"(cv[i]), "=l"(ci[i])
                       : "l"(cand + min(lane + 32 * i, ctas - 1))
                       : "memory");
#pragma unroll
        for (int i = 0; i < kCleanPer; i++)
          all = all && (uint32_t)cv[i] == tag && ((uint32_t)ci[i] & 0xFFFFFFu) == (tag & 0xFFFFFFu);
        if (__all_sync(0xffffffffu, all)) break;
        if (p == kCleanPolls) {
          ok = false;
          break;
        }
      }
#pragma unroll
      for (int i = 0; i < kCleanPer; i++) {
        const float v = __uint_as_float((uint32_t)(cv[i] >> 32));
        const uint64_t x = ci[i] >> 24;
        if (x != kCleanNone &&
            (best == kCleanNone || better(fabsf(v), (int64_t)x, fabsf(val), (int64_t)best))) {
          val = v;
          best = x;
        }
      }
#pragma unroll
      for (int q = 16; q > 0; q >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, val, q);
        const uint64_t oi = __shfl_xor_sync(0xffffffffu, best, q);
        if (oi != kCleanNone &&
            (best == kCleanNone || better(fabsf(ov), (int64_t)oi, fabsf(val), (int64_t)best))) {
          val = ov;
          best = oi;
        }
      }
      if (lane == 0) {
        const bool stop = !ok || best == kCleanNone || fabsf(val) < a.threshold || psf_peak == 0.f;
        if (!ok) atomicExch(&a.w->st.err, 1);
        int py, px;
        if (best >> 32) {
          py = (int)(best / (uint64_t)a.nx);
          px = (int)(best % (uint64_t)a.nx);
        } else {
          py = (int)((uint32_t)best / (uint32_t)a.nx);
          px = (int)((uint32_t)best - (uint32_t)py * (uint32_t)a.nx);
        }
        sh.stop = stop;
        sh.peak = val;
        sh.px = px;
        sh.py = py;
        if (!stop)
          sh.comp[n] = CleanComp{px - a.ppx, py - a.ppy,
                                 __fdiv_rn(__fmul_rn(a.gain, val), psf_peak)};
      }
    }
    __syncthreads();
    if (sh.stop) break;
    const CleanComp q = sh.comp[n];
    if (blockIdx.x == 0 && tid == 0) {
      float* m = a.model + (int64_t)sh.py * a.nx + sh.px;
      *m = __fadd_rn(*m, __fmul_rn(a.gain, sh.peak));
    }
    n++;
    done++;
    // the peak's own pixel after the subtraction: the next peak is no smaller
    lb = fabsf(__fsub_rn(sh.peak, __fmul_rn(q.s, psf_peak)));
    if (!(lb >= 0.f)) lb = -1.f;  // not a number: no bound
    const float as = fabsf(q.s);
    for (int k = lane; k < nt; k += 32) {
      CleanTile& d = tiles[k];
      const int x0 = d.x0 - q.dx, y0 = d.y0 - q.dy;  // of the tile in the PSF
      if (!(x0 < a.pnx && -kCleanTile < x0 && y0 < a.pny && -kCleanRows < y0)) continue;
      const int bx0 = (max(x0, a.wx0) - a.wx0) >> a.eb, by0 = (max(y0, a.wy0) - a.wy0) >> a.eb;
      const int bx1 = (min(x0 + kCleanTile, a.wx1) - 1 - a.wx0) >> a.eb;
      const int by1 = (min(y0 + kCleanRows, a.wy1) - 1 - a.wy0) >> a.eb;
      const float m = fmaxf(fmaxf(psf_max[by0 * a.nbx + bx0], psf_max[by0 * a.nbx + bx1]),
                            fmaxf(psf_max[by1 * a.nbx + bx0], psf_max[by1 * a.nbx + bx1]));
      // rounded up like the pixels' own products and differences at worst
      const float u = __fadd_ru(fmaxf(d.ub, 0.f), __fmul_ru(as, m));
      d.ub = u <= FLT_MAX ? u : __int_as_float(0x7F800000);
      d.exact = 0;
    }
    __syncwarp();
    if (n == kCleanPending) {
      for (int k = 0; k < nt; k++) clean_refresh(a, sh, tiles[k], n);
      for (int k = lane; k < nt; k += 32) tiles[k].ver = 0;
      n = 0;
      __syncthreads();  // the list is reused
    }
  }
  for (int k = 0; k < nt; k++)
    if (tiles[k].ver < n) clean_refresh(a, sh, tiles[k], n);
  if (blockIdx.x == 0 && tid == 0) a.w->st.iterations = done;
}

// ---------------------------------------------------------------- reference form (FP64)
struct RefPeak {
  double absv;
  int64_t idx;
};

// argmax of |res| over x < wx, y < wy (row-major index into a buffer of row
// length nx), first index on ties: one block, written to *out
__global__ void __launch_bounds__(1024) k_ref_argmax(const double* __restrict__ res, int nx,
                                                     int wx, int wy, RefPeak* out) {
  __shared__ double s_v[1024];
  __shared__ int64_t s_i[1024];
  double best = -1.0;
  int64_t bi = INT64_MAX;
  for (int64_t e = threadIdx.x; e < (int64_t)wx * wy; e += blockDim.x) {
    const int x = (int)(e % wx), y = (int)(e / wx);
    const int64_t i = (int64_t)y * nx + x;
    const double a = fabs(res[i]);
    if (a > best || (a == best && i < bi)) {
      best = a;
      bi = i;
    }
  }
  s_v[threadIdx.x] = best;
  s_i[threadIdx.x] = bi;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) {
      const double a = s_v[threadIdx.x + o];
      const int64_t i = s_i[threadIdx.x + o];
      if (a > s_v[threadIdx.x] || (a == s_v[threadIdx.x] && i < s_i[threadIdx.x])) {
        s_v[threadIdx.x] = a;
        s_i[threadIdx.x] = i;
      }
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = RefPeak{s_v[0], s_i[0]};
}

// one reference cycle's update; peaks[0] = the "PSF peak", peaks[1 + c] = cycle c's peak
__global__ void k_ref_cycle(double* __restrict__ res, int nx, int ny,
                            const double* __restrict__ psf, int pnx, int pny,
                            const RefPeak* __restrict__ peaks, int c, double gain,
                            double threshold, double* __restrict__ model, int32_t* under) {
  if (*under) return;
  const RefPeak pk = peaks[1 + c], pp = peaks[0];
  if (pk.absv < threshold) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *under = 1;
    return;
  }
  const int peakX = (int)(pk.idx % nx), peakY = (int)(pk.idx / nx);
  const int ppx = (int)(pp.idx % nx), ppy = (int)(pp.idx / nx);
  const int dx = min(max(peakX - ppx, -pnx), nx), dy = min(max(peakY - ppy, -pny), ny);
  const double s = gain * pk.absv / pp.absv;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < (int64_t)nx * ny;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int x = (int)(e % nx), y = (int)(e / nx);
    const int qx = x - dx, qy = y - dy;
    const double pv = (qx >= 0 && qx < pnx && qy >= 0 && qy < pny) ? psf[(int64_t)qy * pnx + qx]
                                                                    : 0.0;
    res[e] = res[e] - s * pv;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    const int cx = min(max(peakX, 0), nx - 1), cy = min(max(peakY, 0), ny - 1);
    model[(int64_t)cy * nx + cx] += gain * pk.absv;
  }
}

}  // namespace gb

using namespace gb;

namespace {
constexpr size_t kCleanSmem = 200 * 1024;  // of the 227 KB a CTA may have

// The work buffer holds 16-byte records: its first 16-byte boundary.
CleanWork* clean_work(void* d_work) {
  return (CleanWork*)(((uintptr_t)d_work + 15) & ~(uintptr_t)15);
}

// The state, and a record per tile (used where the tiles do not fit the CTAs'
// shared memory; a warp's share is rounded up).
int64_t clean_work_bytes(int32_t nx, int32_t ny) {
  const int64_t ntx = (nx + (int64_t)kCleanTile - 1) / kCleanTile;
  const int64_t nty = (ny + (int64_t)kCleanRows - 1) / kCleanRows;
  return 16 + (int64_t)sizeof(CleanWork) + (ntx * nty + kCleanCtas * kCleanOwners) * (int64_t)sizeof(CleanTile);
}
}  // namespace

extern "C" int gb_hogbom_f32(float* d_residual, int32_t nx, int32_t ny, const float* d_psf,
                             int32_t pnx, int32_t pny, int32_t psf_peak_x, int32_t psf_peak_y,
                             float gain, float threshold, int32_t n_iter, float* d_model,
                             void* d_work, int64_t work_bytes, void* stream) {
  if (!d_residual || !d_psf || !d_model || !d_work || nx < 1 || ny < 1 || pnx < 1 || pny < 1 ||
      psf_peak_x < 0 || psf_peak_x >= pnx || psf_peak_y < 0 || psf_peak_y >= pny || n_iter < 0 ||
      work_bytes < clean_work_bytes(nx, ny)) {
    gb_set_error(GB_ERR_ARG, "gb_hogbom_f32: bad arguments (work needs %lld bytes)",
                 (long long)(nx > 0 && ny > 0 ? clean_work_bytes(nx, ny) : 0));
    return GB_ERR_ARG;
  }
  const int64_t ntx = (nx + (int64_t)kCleanTile - 1) / kCleanTile;
  const int64_t nty = (ny + (int64_t)kCleanRows - 1) / kCleanRows;
  if (ntx * nty > INT32_MAX / 2) {
    gb_set_error(GB_ERR_CAPACITY, "gb_hogbom_f32: more than 2^30 image tiles");
    return GB_ERR_CAPACITY;
  }
  cudaStream_t s = (cudaStream_t)stream;
  CleanArgs a;
  a.w = clean_work(d_work);
  GB_CUDA_TRY(cudaMemsetAsync(a.w, 0, offsetof(CleanWork, psf_max), s));
  if (n_iter == 0) return GB_OK;
  a.res = d_residual;
  a.psf = d_psf;
  a.model = d_model;
  a.nx = nx;
  a.ny = ny;
  a.pnx = pnx;
  a.pny = pny;
  a.ppx = psf_peak_x;
  a.ppy = psf_peak_y;
  a.gain = gain;
  a.threshold = threshold;
  a.n_iter = n_iter;
  a.ntx = (int)ntx;
  a.ntiles = (int)(ntx * nty);
  // A component lies within the image, so only the part of the PSF less than the
  // image's size away from its peak can: of a small image's large PSF a few blocks,
  // not a table that its few CTAs would take milliseconds for (64^2, PSF 4096^2, one
  // iteration: 8.7 ms with all of it, 32 us so; 256^2, PSF 4096^2, 20 iterations:
  // 1109 and 97 us).
  a.wx0 = std::max(0, psf_peak_x - (nx - 1));
  a.wx1 = (int)std::min<int64_t>(pnx, (int64_t)psf_peak_x + nx);
  a.wy0 = std::max(0, psf_peak_y - (ny - 1));
  a.wy1 = (int)std::min<int64_t>(pny, (int64_t)psf_peak_y + ny);
  auto blocks = [&](int n) { return (int64_t)((n + (1ll << a.eb) - 1) >> a.eb); };
  for (a.eb = 5; blocks(a.wx1 - a.wx0) * blocks(a.wy1 - a.wy0) > kCleanPsfBlocks; a.eb++) {}
  a.nbx = (int)blocks(a.wx1 - a.wx0);
  a.nby = (int)blocks(a.wy1 - a.wy0);
  const size_t table = sizeof(float) * (size_t)((a.nbx * a.nby + 3) & ~3);
  GB_CUDA_TRY(cudaFuncSetAttribute((const void*)k_clean, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)kCleanSmem));
  void* args[] = {&a};
  const int64_t want = (ntx * nty + kCleanOwners - 1) / kCleanOwners;
  // The CTAs wait for one another, so all must fit at once.  A process may have fewer
  // multiprocessors than the device (a partition of it): a grid that is refused for
  // that is halved, down to one CTA.
  for (int grid = (int)std::min<int64_t>({want, (int64_t)sm_count(), (int64_t)kCleanCtas});;
       grid = (grid + 1) / 2) {
    const int64_t owners = (int64_t)grid * kCleanOwners;
    a.local = (int)((ntx * nty + owners - 1) / owners);
    const size_t own = sizeof(CleanTile) * (size_t)a.local * kCleanOwners;
    a.far_tiles = table + own > kCleanSmem ? (CleanTile*)(a.w + 1) : nullptr;
    const cudaError_t e =
        cudaLaunchCooperativeKernel((const void*)k_clean, dim3(grid), dim3(kCleanThreads), args,
                                    a.far_tiles ? table : table + own, s);
    if (e != cudaErrorCooperativeLaunchTooLarge || grid == 1) {
      GB_CUDA_TRY(e);
      return GB_OK;
    }
    (void)cudaGetLastError();  // not the next call's
  }
}

extern "C" int gb_hogbom_work_bytes(int32_t nx, int32_t ny, int64_t* out) {
  if (!out || nx < 1 || ny < 1) {
    gb_set_error(GB_ERR_ARG, "gb_hogbom_work_bytes: bad arguments");
    return GB_ERR_ARG;
  }
  *out = clean_work_bytes(nx, ny);
  return GB_OK;
}

extern "C" int gb_hogbom_iterations(const void* d_work, int32_t* out, void* stream) {
  if (!d_work || !out) {
    gb_set_error(GB_ERR_ARG, "gb_hogbom_iterations: NULL argument");
    return GB_ERR_ARG;
  }
  CleanState st;
  GB_CUDA_TRY(cudaMemcpyAsync(&st, clean_work(const_cast<void*>(d_work)), sizeof(st), cudaMemcpyDeviceToHost,
                              (cudaStream_t)stream));
  GB_CUDA_TRY(cudaStreamSynchronize((cudaStream_t)stream));
  *out = st.iterations;
  if (st.err) {
    gb_set_error(GB_ERR_TIMEOUT, "gb_hogbom_f32: a wait for the other CTAs did not complete in time");
    return GB_ERR_TIMEOUT;
  }
  return GB_OK;
}

// ---------------------------------------------------------------- reference ABI
namespace {
constexpr int kRefCycles = 12;  // MS6/kernel/cpu/gridding/hogbom.cpp:4

int check_img(const buffer_t* b, const char* who, const char* name) {
  if (!b || !b->host || b->elem_size != 8 || b->extent[0] < 1 || b->extent[1] < 1 ||
      b->stride[0] != 1 || (b->extent[1] > 1 && b->stride[1] != b->extent[0])) {
    gb_set_error(GB_ERR_ARG, "%s: %s must be a dense 2-D double image", who, name);
    return GB_ERR_ARG;
  }
  return GB_OK;
}

// shared body: runs the 12 cycles on device copies; returns the model and the
// residual of the threshold cycle (or the last)
int ref_clean(double gain, double threshold, buffer_t* psf, buffer_t* res, buffer_t* model,
              buffer_t* res_out, const char* who) {
  int rc;
  if ((rc = check_img(psf, who, "psf")) || (rc = check_img(res, who, "res"))) return rc;
  buffer_t* out = model ? model : res_out;
  if ((rc = check_img(out, who, "output"))) return rc;
  const int nx = res->extent[0], ny = res->extent[1];
  const int pnx = psf->extent[0], pny = psf->extent[1];
  if (out->extent[0] != nx || out->extent[1] != ny) {
    gb_set_error(GB_ERR_ARG, "%s: output must match the residual's extent", who);
    return GB_ERR_ARG;
  }
  cudaStream_t s;
  if ((rc = stage_stream(&s))) return rc;
  void *d_res, *d_psf, *d_model, *d_aux;
  const size_t nres = (size_t)nx * ny * 8, npsf = (size_t)pnx * pny * 8;
  if ((rc = stage_buffer(0, nres, &d_res)) || (rc = stage_buffer(1, npsf, &d_psf)) ||
      (rc = stage_buffer(2, nres, &d_model)) ||
      (rc = stage_buffer(3, sizeof(RefPeak) * (kRefCycles + 1) + 16, &d_aux)))
    return rc;
  RefPeak* peaks = (RefPeak*)d_aux;
  int32_t* under = (int32_t*)(peaks + kRefCycles + 1);
  GB_CUDA_TRY(cudaMemcpyAsync(d_res, res->host, nres, cudaMemcpyHostToDevice, s));
  GB_CUDA_TRY(cudaMemcpyAsync(d_psf, psf->host, npsf, cudaMemcpyHostToDevice, s));
  if (model)
    GB_CUDA_TRY(cudaMemcpyAsync(d_model, model->host, nres, cudaMemcpyHostToDevice, s));
  else
    GB_CUDA_TRY(cudaMemsetAsync(d_model, 0, nres, s));
  GB_CUDA_TRY(cudaMemsetAsync(under, 0, sizeof(int32_t), s));
  // "PSF peak": argmax |res| over the PSF's domain (hogbom.cpp:57-61)
  k_ref_argmax<<<1, 1024, 0, s>>>((const double*)d_res, nx, std::min(pnx, nx), std::min(pny, ny),
                                  peaks);
  GB_CUDA_TRY(cudaGetLastError());
  const int blocks = (int)std::min<int64_t>(((int64_t)nx * ny + 255) / 256, sm_count() * 8);
  // Once a cycle's peak is under the threshold it neither subtracts nor adds
  // to the model and sets `under`, which makes every later cycle a no-op: the
  // residual left is the one of the crossing cycle (hogbom.cpp:68-74).
  for (int c = 0; c < kRefCycles; c++) {
    k_ref_argmax<<<1, 1024, 0, s>>>((const double*)d_res, nx, nx, ny, peaks + 1 + c);
    GB_CUDA_TRY(cudaGetLastError());
    k_ref_cycle<<<blocks, 256, 0, s>>>((double*)d_res, nx, ny, (const double*)d_psf, pnx, pny,
                                       peaks, c, gain, threshold, (double*)d_model, under);
    GB_CUDA_TRY(cudaGetLastError());
  }
  if (model)
    GB_CUDA_TRY(cudaMemcpyAsync(model->host, d_model, nres, cudaMemcpyDeviceToHost, s));
  else
    GB_CUDA_TRY(cudaMemcpyAsync(res_out->host, d_res, nres, cudaMemcpyDeviceToHost, s));
  GB_CUDA_TRY(cudaStreamSynchronize(s));
  return GB_OK;
}
}  // namespace

// replaces kern_hogbom_model (MS6/kernel/cpu/gridding/hogbom.cpp:128,
// bound at MS6/programs/Kernel/Cleaning.hs:22-32): model accumulates in place
extern "C" int kern_hogbom_model(double gain, double threshold, buffer_t* psf, buffer_t* res,
                                 buffer_t* model) {
  return ref_clean(gain, threshold, psf, res, model, nullptr, "kern_hogbom_model");
}

// replaces kern_hogbom_residual (hogbom.cpp:129, Cleaning.hs:35-44)
extern "C" int kern_hogbom_residual(double gain, double threshold, buffer_t* psf, buffer_t* res,
                                    buffer_t* residual) {
  return ref_clean(gain, threshold, psf, res, nullptr, residual, "kern_hogbom_residual");
}
