// Visibility plan: w-plane assignment, FP64 index math, and the sort / bin of
// footprint pieces by (grid tile, period) that feeds the FP32 tiled kernels.
//
// It replaces the reference's host-side binning (MS6/programs/Kernel/
// Binning.hs:34-181, a scalar Haskell pass per visibility) and the NVIDIA
// gridder's host std::sort (MS6/kernel/nvidia/gridder/binsort.cpp:6-35) with
// a counting sort on the GPU:
//   1. k_plan_count: per visibility, plane + index math (FP64), then a
//      histogram of pieces per (tile, period rank) and of visibilities per tile;
//   2. an exclusive scan of both;
//   3. k_plan_items, twice (count, write): work items, the record ranges of one
//      tile and one thread-group class, cut by a cost model;
//   4. k_plan_fill: 16-byte records scattered into their bins;
//   5. bundle_items: items longest first, bundles of them for the persistent
//      kernels, longest first.
// The host reads back once, between counting and writing items, to size the
// arrays.  1.17 M visibilities on a 4096^2 grid take 0.84 ms, of which the kernels
// 0.28 ms (k_plan_count 110 us, its FP64 index math); with the scan, the items and
// the bundles on the host 2.55 ms.  4.18 M: 1.04 ms (2.88), 4.18 M on 8192^2 1.25 ms
// (6.39).
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "gb_common.cuh"
#include "gb_plan.cuh"
#include "gb_runtime.cuh"

namespace gb {

// What the plan's later kernels need of a visibility: its corner pixel and
// phase (x < 0: not kept), so that the FP64 index math runs once.
struct VisCell {
  int32_t x, yp;  // yp = y | phase << 24 (a grid has at most 2^22 rows)
};

constexpr int kMaxRanks = 64;  // distinct periods

// Counters of k_plan_count (the first four), k_rank_sums and k_plan_items, and
// the classes' first items.
struct PlanCounts {
  unsigned long long kept, taps, recs, paired, tiles;
  unsigned long long rank[kMaxRanks];  // pieces per period rank
  int32_t class_first[kMaxClasses + 1];
};

// +1 at hist[key] for every active lane: one atomic per distinct key.  Returns
// the lane's place among the key's lanes, in lane order, after what was there.
__device__ __forceinline__ int32_t warp_count(int32_t* __restrict__ hist, int64_t key) {
  const unsigned act = __activemask(), peers = __match_any_sync(act, key);
  const int lane = threadIdx.x & 31, leader = __ffs(peers) - 1;
  int32_t first = 0;
  if (lane == leader) first = atomicAdd(&hist[key], __popc(peers));
  first = __shfl_sync(act, first, leader);
  return first + __popc(peers & ((1u << lane) - 1u));
}

__global__ void __launch_bounds__(256)
    k_plan_count(PlanDev P, const PlaneInfo* __restrict__ pl, const int32_t* __restrict__ plane_in,
                 int32_t* __restrict__ plane_out, VisCell* __restrict__ cells, int32_t n_planes,
                 double w_lo, double w_hi, int32_t T, int32_t ntx, int32_t nper,
                 int32_t* __restrict__ hist, int32_t* __restrict__ vis_hist,
                 PlanCounts* __restrict__ cnt) {
  unsigned long long sum[4] = {0, 0, 0, 0};  // kept, taps, recs, paired
  const int64_t ntiles = (int64_t)ntx * ((P.ext_y + T - 1) / T);
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < P.n_vis;
       t += (int64_t)gridDim.x * blockDim.x) {
    const double* r = P.uvw + t * P.uvw_stride;
    int32_t p = plane_in ? plane_in[t] : w_plane(r[2], w_lo, w_hi, n_planes);
    if (p >= n_planes) p = -1;
    plane_out[t] = p;
    VisIndex ix;
    ix.keep = false;
    PlaneInfo q;
    if (p >= 0) {
      q = pl[p];
      ix = vis_index(r[0], r[1], P.scale, P.grid_size, q.S, P.margin, 0, 0, P.ext_x, P.ext_y);
    }
    cells[t] = ix.keep ? VisCell{ix.x0, ix.y0 | ix.phase << 24} : VisCell{-1, 0};
    // skipped visibilities go last
    warp_count(vis_hist, ix.keep ? (int64_t)(ix.y0 / T) * ntx + ix.x0 / T : ntiles);
    if (!ix.keep) continue;
    sum[0]++;
    sum[1] += (unsigned long long)q.S * q.S;
    for (int oy = 0; oy < q.S; oy += q.P) {
      const int64_t row = (int64_t)((ix.y0 + oy) / T) * ntx;
      for (int ox = 0; ox < q.S; ox += q.P) {
        warp_count(hist, (row + (ix.x0 + ox) / T) * nper + q.rank);
        sum[2]++;
        // degridding pairs the taps of a piece whose rows, GCF rows and GCF
        // offset are all even (the same rule the kernels apply per record)
        const int wx = min(q.P, q.S - ox), wy = min(q.P, q.S - oy);
        if (((wx | q.S | (int)((q.gcf_off + ox) & 1)) & 1) == 0)
          sum[3] += (unsigned long long)wx * wy;
      }
    }
  }
  __shared__ unsigned long long s_sum[8][4];  // per warp
#pragma unroll
  for (int k = 0; k < 4; k++) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum[k] += __shfl_xor_sync(0xffffffffu, sum[k], o);
    if ((threadIdx.x & 31) == 0) s_sum[threadIdx.x >> 5][k] = sum[k];
  }
  __syncthreads();
  if (threadIdx.x < 4) {
    unsigned long long all = 0;
    for (int w = 0; w < 8; w++) all += s_sum[w][threadIdx.x];
    if (all) atomicAdd(&cnt->kept + threadIdx.x, all);
  }
}

// Pieces per period rank (keys run rank-fastest within a tile).
__global__ void __launch_bounds__(256) k_rank_sums(const int32_t* __restrict__ hist, int64_t nkeys,
                                                   int nper, PlanCounts* __restrict__ cnt) {
  __shared__ unsigned long long s_rank[kMaxRanks];
  for (int r = threadIdx.x; r < nper; r += blockDim.x) s_rank[r] = 0;
  __syncthreads();
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nkeys;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int32_t v = hist[i];
    if (v) atomicAdd(&s_rank[i % nper], (unsigned long long)v);
  }
  __syncthreads();
  for (int r = threadIdx.x; r < nper; r += blockDim.x)
    if (s_rank[r]) atomicAdd(&cnt->rank[r], s_rank[r]);
}

// ---------------------------------------------------------------- exclusive scan
// out[i] = in[0] + .. + in[i - 1] for i = 0 .. n, modulo 2^32: sums per block of
// kScanKeys keys, their scan by one block, the keys' scan with those.
constexpr int kScanThreads = 512, kScanPer = 8, kScanKeys = kScanThreads * kScanPer;

// Exclusive scan over the block of each thread's value; *total the sum.
__device__ __forceinline__ uint32_t block_scan(uint32_t v, uint32_t* total) {
  __shared__ uint32_t warp_sum[kScanThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t a = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += a;
  }
  __syncthreads();  // warp_sum of an earlier call is read
  if (lane == 31) warp_sum[warp] = inc;
  __syncthreads();
  uint32_t before = 0, all = 0;
#pragma unroll
  for (int w = 0; w < kScanThreads / 32; w++) {
    if (w < warp) before += warp_sum[w];
    all += warp_sum[w];
  }
  *total = all;
  return before + inc - v;
}

__global__ void __launch_bounds__(kScanThreads)
    k_scan_sums(const int32_t* __restrict__ in, int64_t n, uint32_t* __restrict__ sums) {
  const int64_t i0 = (int64_t)blockIdx.x * kScanKeys;
  uint32_t v = 0;
#pragma unroll
  for (int k = 0; k < kScanPer; k++) {
    const int64_t i = i0 + k * kScanThreads + threadIdx.x;
    if (i < n) v += (uint32_t)in[i];
  }
  uint32_t total;
  block_scan(v, &total);
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_top(uint32_t* __restrict__ sums, int nb) {
  uint32_t carry = 0;
  for (int b = 0; b < nb; b += kScanThreads) {
    const int i = b + threadIdx.x;
    const uint32_t v = i < nb ? sums[i] : 0u;
    uint32_t total;
    const uint32_t e = block_scan(v, &total);
    if (i < nb) sums[i] = carry + e;
    carry += total;
  }
}

__global__ void __launch_bounds__(kScanThreads)
    k_scan_keys32(const int32_t* __restrict__ in, int64_t n, const uint32_t* __restrict__ sums,
                  int32_t* __restrict__ out) {
  const int64_t i0 = (int64_t)blockIdx.x * kScanKeys + (int64_t)threadIdx.x * kScanPer;
  uint32_t v[kScanPer], sum = 0;
#pragma unroll
  for (int k = 0; k < kScanPer; k++) {
    v[k] = i0 + k < n ? (uint32_t)in[i0 + k] : 0u;
    sum += v[k];
  }
  uint32_t total, e = block_scan(sum, &total) + sums[blockIdx.x];
#pragma unroll
  for (int k = 0; k < kScanPer; k++) {
    if (i0 + k <= n) out[i0 + k] = (int32_t)e;
    e += v[k];
  }
}

static int64_t scan_blocks(int64_t n) { return n / kScanKeys + 1; }  // out has n + 1 entries

// sums: scan_blocks(n) words of scratch.
static int scan_keys(const int32_t* in, int64_t n, int32_t* out, uint32_t* sums, cudaStream_t s) {
  const int nb = (int)scan_blocks(n);
  k_scan_sums<<<nb, kScanThreads, 0, s>>>(in, n, sums);
  k_scan_top<<<1, kScanThreads, 0, s>>>(sums, nb);
  k_scan_keys32<<<nb, kScanThreads, 0, s>>>(in, n, sums, out);
  GB_CUDA_TRY(cudaGetLastError());
  return GB_OK;
}

// ---------------------------------------------------------------- items
// How the items are cut: the classes' period ranks (consecutive: group width
// grows with the period), the cost of a record and of an item, and per rank the
// split-row stride residue of degridding.
struct ItemRule {
  int nper, nclass;
  int lo[kMaxClasses], hi[kMaxClasses];
  float fixed[kMaxClasses];
  float rec[kMaxRanks];       // cost of a record
  double per_cta[kMaxRanks];  // the same over the items a CTA runs side by side
  int16_t period[kMaxRanks];
  int8_t residue[kMaxRanks];
  double pieces;  // items wanted per unit of total cost: bundles per CTA x CTAs
};

// Writes the items (where `items` is given, from index `at` on) of one tile's records
// of class c; returns how many.  An item is closed when its cost reaches cmax.  By one
// thread; or by a warp, all of whose lanes walk the same way: items of one rank alone are
// alike from the first record of one on, so the warp counts them by a division and
// writes them side by side.
template <bool kWarp>
__device__ __forceinline__ int cut_items(const ItemRule& R, const int32_t* __restrict__ offs,
                                         int64_t tile, int ntx, int c, float cmax, int64_t at,
                                         Item* __restrict__ items, float* __restrict__ costs) {
  const int64_t k0 = tile * R.nper;
  const int lane = threadIdx.x & 31;
  const float fixed = R.fixed[c];
  float cost = fixed;
  int32_t start = offs[k0 + R.lo[c]], in_item = 0;
  int64_t top_taps = 0;
  int n = 0, top = -1, pmax = 0;
  auto write = [&](int64_t i, int32_t first, int32_t records, int p, int rank, float item_cost) {
    Item it;
    it.start = first;
    it.count = records;
    it.tile_x = (int16_t)(tile % ntx);
    it.tile_y = (int16_t)(tile / ntx);
    it.pmax = (int16_t)p;
    it.cls = item_cls_with_residue((int16_t)c, R.residue[rank]);
    items[i] = it;
    costs[i] = item_cost;
  };
  auto close = [&]() {
    if (items && (!kWarp || lane == 0)) write(at + n, start, in_item, pmax, top, cost);
    n++;
    start += in_item;
    in_item = 0;
    cost = fixed;
    top_taps = 0;
    pmax = 0;
  };
  for (int r = R.lo[c]; r < R.hi[c]; r++) {
    int32_t pos = offs[k0 + r];
    const int32_t end = offs[k0 + r + 1];
    const float rc = R.rec[r], per = 1.f / rc;
    int32_t alike0 = -1;  // where the last item that began with this rank did
    while (pos < end) {
      if (kWarp && !in_item) {
        if (alike0 >= 0) {  // the one before is of this rank alone: so are the next m
          const int32_t recs = pos - alike0, m = (end - pos) / recs;
          float item_cost = fixed;
          for (int32_t k = 0; k < recs && m > 0;) {  // its cost, step by step
            const int32_t take = min(max((int32_t)fminf((cmax - item_cost) * per, 2e9f), 1), recs - k);
            item_cost += (float)take * rc;
            k += take;
          }
          if (items)
            for (int i = lane; i < m; i += 32)
              write(at + n + i, pos + i * recs, recs, R.period[r], r, item_cost);
          n += m;
          pos += m * recs;
          start = pos;
          alike0 = -1;
          if (m > 0) continue;
        }
        alike0 = pos;
      }
      const float room = fminf((cmax - cost) * per, 2e9f);
      const int32_t take = min(max((int32_t)room, 1), end - pos);
      const int64_t t = (int64_t)take * R.period[r] * R.period[r];
      if (t > top_taps) {  // the stage stride goes by the largest run
        top_taps = t;
        top = r;
      }
      pmax = R.period[r];
      in_item += take;
      cost += (float)take * rc;
      pos += take;
      if (cost >= cmax) close();
    }
  }
  if (in_item) close();
  return n;
}

constexpr int kItemThreads = 128;
// Items from which a warp cuts them (counting and writing, us): from 128 / 64 / 32 / 16 a
// core-heavy 1e6 of 29 planes on 1024^2 31 and 63 / 21 and 36 / 21 and 35 / 26 and 38, 1e5
// of 31 planes on 256^2 37 and 76 / 42 and 75 / 58 and 90 / 69 and 105.
constexpr float kWarpItems = 64.f;

// The items of each (class, tile): counted (per class, tile-fastest), or with
// `items` written from first[] on.  cmax: the larger of four times an item's fixed
// cost and an even share of all the work.
// A thread to a (class, tile): most are empty or give an item or a few.  But a
// core-heavy array puts much of its work into a few tiles, each of hundreds or
// thousands of items: those are left for the block's warps.  A plan of 1e6 visibilities
// of support 8, all in one tile: 0.66 ms, with a thread to each tile 4.6 ms (on host
// threads 2.3 ms); 8e6: 1.4 ms, 4.8 and 11.6; 1e6 of a core-heavy array on 256^2: 0.79 ms,
// 2.9 and 1.8.  Every lane in step over the ranks of all tiles took 10 us longer where
// the tiles are sparse (39 -> 49 us on 16384^2, 31 ranks).
__global__ void __launch_bounds__(kItemThreads)
    k_plan_items(const __grid_constant__ ItemRule R, int64_t ntiles, int32_t ntx,
                 const int32_t* __restrict__ offs, PlanCounts* __restrict__ cnt,
                 int32_t* __restrict__ count, const int32_t* __restrict__ first,
                 Item* __restrict__ items, float* __restrict__ costs) {
  __shared__ float s_tau;
  __shared__ bool s_over;
  __shared__ int s_dense;
  __shared__ int32_t s_entry[kItemThreads];
  if (threadIdx.x == 0) {
    double total = 0;
    for (int r = 0; r < R.nper; r++) total += (double)cnt->rank[r] * R.per_cta[r];
    s_tau = (float)(total / R.pieces);
    s_over = cnt->recs >= (unsigned long long)INT32_MAX;  // refused by the host: offs wrapped
    s_dense = 0;
  }
  __syncthreads();
  const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int c = (int)(e / ntiles);
  bool used = false;
  if (c < R.nclass) {
    const int64_t tile = e - c * ntiles, k0 = tile * R.nper;
    const int32_t b0 = offs[k0 + R.lo[c]], b1 = offs[k0 + R.hi[c]];
    used = c == 0 && offs[k0 + R.nper] != offs[k0];
    int n = 0;
    if (b1 != b0 && !s_over) {
      const float cmax = fmaxf(4.f * R.fixed[c], s_tau);
      if ((float)(b1 - b0) * R.rec[R.lo[c]] >= kWarpItems * (cmax - R.fixed[c]))
        s_entry[atomicAdd(&s_dense, 1)] = threadIdx.x;
      else
        n = cut_items<false>(R, offs, tile, ntx, c, cmax, items ? first[e] : 0, items, costs);
    }
    if (!items) count[e] = n;
  }
  // (the dense ones' counts after the zeros above)
  const int used_here = __syncthreads_count(used);
  if (!items && threadIdx.x == 0 && used_here)
    atomicAdd(&cnt->tiles, (unsigned long long)used_here);
  for (int k = threadIdx.x >> 5; k < s_dense; k += kItemThreads / 32) {
    const int64_t d = blockIdx.x * (int64_t)blockDim.x + s_entry[k];
    const int dc = (int)(d / ntiles);
    const int n = cut_items<true>(R, offs, d - dc * ntiles, ntx, dc, fmaxf(4.f * R.fixed[dc], s_tau),
                                  items ? first[d] : 0, items, costs);
    if (!items && (threadIdx.x & 31) == 0) count[d] = n;
  }
}

// The classes' first items, from the scan of their counts.
__global__ void k_plan_classes(const int32_t* __restrict__ first, int64_t ntiles, int nclass,
                               PlanCounts* __restrict__ cnt) {
  if (threadIdx.x <= nclass) cnt->class_first[threadIdx.x] = first[threadIdx.x * ntiles];
}

// offs, vis_offs: the scan of both histograms one after the other; the cursors
// are the same arrays, zeroed again.
__global__ void k_plan_fill(PlanDev P, const PlaneInfo* __restrict__ pl,
                            const VisCell* __restrict__ cells, int32_t T, int32_t ntx, int32_t nper,
                            const int32_t* __restrict__ offs, int32_t* __restrict__ cursor,
                            Rec* __restrict__ recs, const int32_t* __restrict__ vis_offs,
                            int32_t* __restrict__ vis_cursor, int32_t* __restrict__ order) {
  const int64_t ntiles = (int64_t)ntx * ((P.ext_y + T - 1) / T);
  const uint32_t vis0 = (uint32_t)vis_offs[0];
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < P.n_vis;
       t += (int64_t)gridDim.x * blockDim.x) {
    const VisCell cell = cells[t];
    const bool keep = cell.x >= 0;
    const int x0 = cell.x, y0 = cell.yp & 0xFFFFFF, phase = cell.yp >> 24;
    const int64_t vt = keep ? (int64_t)(y0 / T) * ntx + x0 / T : ntiles;
    order[(uint32_t)vis_offs[vt] - vis0 + (uint32_t)warp_count(vis_cursor, vt)] = (int32_t)t;
    if (!keep) continue;
    const PlaneInfo q = pl[P.plane[t]];
    const int64_t gbase = q.gcf_off + (int64_t)phase * q.S * q.S;
    for (int oy = 0; oy < q.S; oy += q.P) {
      const int Y0 = y0 + oy, ty = Y0 / T;
      const int wy = min(q.P, q.S - oy);
      for (int ox = 0; ox < q.S; ox += q.P) {
        const int X0 = x0 + ox, tx = X0 / T;
        const int wx = min(q.P, q.S - ox);
        // lanes with the same bin take consecutive places in lane order:
        // neighbouring samples of a baseline, which a warp holds side by side,
        // stay neighbours in the bin, where the gridder sums the taps that
        // consecutive pieces put on one pixel
        const int64_t key = ((int64_t)ty * ntx + tx) * nper + q.rank;
        const int32_t pos = offs[key] + warp_count(cursor, key);
        Rec rc;
        rc.vis = (int32_t)t;
        rc.gcf = (uint32_t)(gbase + (int64_t)oy * q.S + ox);
        rc.xl = (uint8_t)(X0 - tx * T);
        rc.yl = (uint8_t)(Y0 - ty * T);
        rc.wx = (uint8_t)wx;
        rc.wy = (uint8_t)wy;
        rc.xm = (uint8_t)(X0 % q.P);
        rc.ym = (uint8_t)(Y0 % q.P);
        rc.pm1 = (uint8_t)(q.P - 1);
        rc.sm1 = (uint8_t)(q.S - 1);
        recs[pos] = rc;
      }
    }
  }
}

// ---------------------------------------------------------------- bundles
// Items sorted by cost within their (class, grid) bucket, quantised to kLevels
// levels of the largest cost (the longest-first heuristic needs no finer
// order), groups of G of them as bundles, bundles sorted likewise.
constexpr int kLevels = 1024;

struct Bucket {
  int32_t first, count, first_bundle, G;
};

__global__ void k_cost_max(const float* __restrict__ cost, int n, int* __restrict__ top) {
  float m = 0.f;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    m = fmaxf(m, cost[i]);
  const int w = __reduce_max_sync(0xffffffffu, __float_as_int(m));
  if ((threadIdx.x & 31) == 0) atomicMax(top, w);
}

__device__ __forceinline__ int cost_level(float cost, const int* top) {
  const float m = __int_as_float(*top);
  const int l = m > 0.f ? (int)(cost / m * (kLevels - 1)) : 0;
  return kLevels - 1 - min(max(l, 0), kLevels - 1);  // largest first
}

__device__ __forceinline__ int64_t item_key(const Item& it, int grid, int ngrid, int level) {
  return ((int64_t)item_class(it.cls) * ngrid + grid) * kLevels + level;
}

// grids: the items' grid slots, or NULL (slot 0).
__global__ void k_item_levels(const Item* __restrict__ items, const float* __restrict__ cost,
                              const int16_t* __restrict__ grids, int n, int ngrid,
                              const int* __restrict__ top, int32_t* __restrict__ hist) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n)
    warp_count(hist, item_key(items[i], grids ? grids[i] : 0, ngrid, cost_level(cost[i], top)));
}

__global__ void k_item_place(const Item* __restrict__ items, const float* __restrict__ cost,
                             const int16_t* __restrict__ grids, int n, int ngrid,
                             const int* __restrict__ top, const int32_t* __restrict__ offs,
                             int32_t* __restrict__ cursor, Item* __restrict__ out,
                             int32_t* __restrict__ levels) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int level = cost_level(cost[i], top);
  const int64_t key = item_key(items[i], grids ? grids[i] : 0, ngrid, level);
  const int pos = offs[key] + warp_count(cursor, key);
  out[pos] = items[i];
  levels[pos] = level;
}

__device__ __forceinline__ int find_bucket(const Bucket* __restrict__ b, int n, int bundle) {
  int lo = 0, hi = n - 1;  // the last bucket whose first bundle is not after it
  while (lo < hi) {
    const int m = (lo + hi + 1) / 2;
    if (b[m].first_bundle <= bundle)
      lo = m;
    else
      hi = m - 1;
  }
  return lo;
}

// Counts the bundles' levels, or with `out` writes them in level order.
__global__ void k_bundles(const Bucket* __restrict__ buckets, int nbuckets, int ngrid, int n,
                          const int32_t* __restrict__ levels, int32_t* __restrict__ hist,
                          const int32_t* __restrict__ offs, Bundle* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int k = find_bucket(buckets, nbuckets, i);
  const Bucket b = buckets[k];
  const int at = (i - b.first_bundle) * b.G, level = levels[b.first + at];
  const int place = warp_count(hist, level);
  if (!out) return;
  Bundle q;
  q.first_item = b.first + at;
  q.n_items = (int16_t)min(b.G, b.count - at);
  q.cls = (int16_t)(k / ngrid);
  q.grid = k % ngrid;
  q.pad = 0;
  out[offs[level] + place] = q;
}

int count_bundles(const std::vector<int>& counts, const ClassInfo* cls, int ngrid) {
  int64_t n = 0;
  for (size_t k = 0; k < counts.size(); k++) {
    const int G = cls[k / ngrid].G;
    n += (counts[k] + G - 1) / G;
  }
  return (int)n;
}

int bundle_items(const Item* items, const float* cost, const int16_t* grids, int n,
                 const std::vector<int>& counts, const ClassInfo* cls, int ngrid, Item* out,
                 Bundle* bundles, cudaStream_t s) {
  if (n == 0) return GB_OK;
  const int nb = (int)counts.size();
  std::vector<Bucket> hb(nb);
  int first = 0, fb = 0;
  for (int k = 0; k < nb; k++) {
    hb[k] = Bucket{first, counts[k], fb, cls[k / ngrid].G};
    first += counts[k];
    fb += (counts[k] + hb[k].G - 1) / hb[k].G;
  }
  const int64_t keys = (int64_t)nb * kLevels;
  // scratch: top | item histogram | bundle histogram (zeroed), their scans, the
  // items' levels, scan sums, buckets
  const int64_t zero = 1 + keys + kLevels;
  const int64_t words = 2 * zero + 3 + n + scan_blocks(keys) + 4 * (int64_t)nb;
  int32_t* d = nullptr;
  int rc = dev_alloc((void**)&d, sizeof(int32_t) * words, "plan bundles");
  if (rc) return rc;
  int *top = d, *hist = top + 1, *bhist = hist + keys;
  int *offs = d + zero, *boffs = offs + keys + 1, *levels = boffs + kLevels + 1;
  uint32_t* sums = (uint32_t*)(levels + n);
  Bucket* db = (Bucket*)(sums + scan_blocks(keys));
  const int ib = (n + 255) / 256, bb = (fb + 255) / 256;
  auto run = [&]() -> int {
    GB_CUDA_TRY(cudaMemsetAsync(d, 0, sizeof(int32_t) * zero, s));
    GB_CUDA_TRY(cudaMemcpyAsync(db, hb.data(), sizeof(Bucket) * nb, cudaMemcpyHostToDevice, s));
    k_cost_max<<<std::min(ib, sm_count()), 256, 0, s>>>(cost, n, top);
    k_item_levels<<<ib, 256, 0, s>>>(items, cost, grids, n, ngrid, top, hist);
    if ((rc = scan_keys(hist, keys, offs, sums, s))) return rc;
    GB_CUDA_TRY(cudaMemsetAsync(hist, 0, sizeof(int32_t) * keys, s));
    k_item_place<<<ib, 256, 0, s>>>(items, cost, grids, n, ngrid, top, offs, hist, out, levels);
    k_bundles<<<bb, 256, 0, s>>>(db, nb, ngrid, fb, levels, bhist, nullptr, nullptr);
    if ((rc = scan_keys(bhist, kLevels, boffs, sums, s))) return rc;
    GB_CUDA_TRY(cudaMemsetAsync(bhist, 0, sizeof(int32_t) * kLevels, s));
    k_bundles<<<bb, 256, 0, s>>>(db, nb, ngrid, fb, levels, bhist, boffs, bundles);
    GB_CUDA_TRY(cudaGetLastError());
    GB_CUDA_TRY(cudaStreamSynchronize(s));
    return GB_OK;
  };
  rc = run();
  cudaFree(d);
  return rc;
}

__global__ void k_plan_export(PlanDev P, const int32_t* __restrict__ supports,
                              int32_t* __restrict__ out5) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < P.n_vis;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int32_t p = P.plane[t];
    int32_t* o = out5 + 5 * t;
    if (p < 0) {
      o[0] = o[1] = o[2] = 0;
      o[3] = p;
      o[4] = 0;
      continue;
    }
    const double* r = P.uvw + t * P.uvw_stride;
    const VisIndex ix = vis_index(r[0], r[1], P.scale, P.grid_size, supports[p], P.margin, 0, 0,
                                  P.ext_x, P.ext_y);
    o[0] = ix.x0;
    o[1] = ix.y0;
    o[2] = ix.phase;
    o[3] = p;
    o[4] = ix.keep ? 1 : 0;
  }
}

// Thread-group width for a period: the smallest power of two L >= 64 (and
// <= NT) holding P^2 taps in at most two rounds; NT otherwise.
static int class_width(int P, int NT) {
  for (int L = 64; L <= NT; L *= 2)
    if (P * P <= 2 * L) return L;
  return NT;
}

static int blocks_for(int64_t n, int threads) {
  int64_t b = (n + threads - 1) / threads;
  const int64_t cap = (int64_t)sm_count() * 32;
  if (b > cap) b = cap;
  return (int)(b < 1 ? 1 : b);
}

}  // namespace gb

void gb_plan::release_raw() {
  cudaFree(d_raw_items);
  d_raw_items = nullptr;
  d_raw_cost = nullptr;
}

namespace gb {

static void free_plan(gb_plan* p) {
  if (!p) return;
  cudaFree(p->d_tables);
  cudaFree(p->d_recs);
  cudaFree(p->d_items);
  p->release_raw();
  p->df.release();
  delete p;
}

template <class T>
static int dalloc(T** p, size_t n) {
  void* q = nullptr;
  const int rc = dev_alloc(&q, sizeof(T) * (n ? n : 1), "plan");
  *p = (T*)q;
  return rc;
}

// Modelled shared-memory wavefronts per pair that degridding's split-row stage
// costs a sub-warp of SW lanes reading SW consecutive pairs (row-major, rows
// of w2 pairs) with rows r (mod 16) float2 apart: the largest number of
// addresses on one 8-byte bank pair (of 16), averaged over where the run
// starts in its row, per pair of the run.
static double split_stage_cost(int w2, int r, int SW) {
  double sum = 0;
  for (int t0 = 0; t0 < w2; t0++) {
    int cnt[16] = {0};
    for (int l = 0; l < SW; l++) {
      const int t = t0 + l, j = t / w2, i = t - j * w2;
      cnt[(j * r + i) & 15]++;
    }
    sum += *std::max_element(cnt, cnt + 16);
  }
  return sum / w2 / SW;
}

// Sub-warp width of degridding for a class's largest period (the kernel's rule).
static int degrid_subwarp(int pmax) { return pmax <= 8 ? 8 : pmax <= 16 ? 16 : 32; }

static int build_plan(gb_plan* P, const gb_geometry* geo, int64_t n_vis, const double* d_uvw,
                      int64_t uvw_stride, const int32_t* d_plane_in, cudaStream_t s) {
  int rc;
  const int np = geo->n_planes;
  // ---- per-plane pieces, periods, classes
  P->planes.resize(np);
  std::vector<int> periods;
  for (int p = 0; p < np; p++) {
    PlaneInfo& q = P->planes[p];
    q.S = geo->supports[p];
    q.k = (q.S + P->pcap - 1) / P->pcap;
    q.P = (q.S + q.k - 1) / q.k;
    // an even support is cut into even-width pieces (the last one narrower),
    // so degridding can take every piece's taps in pairs
    if (q.k > 1 && !(q.S & 1) && (q.P & 1) && q.P < P->pcap) q.P++;
    q.gcf_off = geo->gcf_offsets[p];
    P->gcf_len = std::max<int64_t>(P->gcf_len, q.gcf_off + (int64_t)GB_PHASES * q.S * q.S);
    periods.push_back(q.P);
    if (q.gcf_off + (int64_t)GB_PHASES * q.S * q.S > (int64_t)UINT32_MAX) {
      gb_set_error(GB_ERR_CAPACITY, "GCF array exceeds 2^32 complex elements");
      return GB_ERR_CAPACITY;
    }
  }
  std::sort(periods.begin(), periods.end());
  periods.erase(std::unique(periods.begin(), periods.end()), periods.end());
  const int nper = (int)periods.size();
  for (auto& q : P->planes)
    q.rank = (int)(std::lower_bound(periods.begin(), periods.end(), q.P) - periods.begin());
  // classes by group width, ascending
  std::vector<int> widths;
  for (int pp : periods) widths.push_back(class_width(pp, P->NT));
  std::vector<int> cls_w = widths;
  std::sort(cls_w.begin(), cls_w.end());
  cls_w.erase(std::unique(cls_w.begin(), cls_w.end()), cls_w.end());
  P->n_classes = (int)cls_w.size();
  if (P->n_classes > kMaxClasses) {
    gb_set_error(GB_ERR_CAPACITY, "too many thread-group classes");
    return GB_ERR_CAPACITY;
  }
  std::vector<int> rank_cls(nper);
  for (int r = 0; r < nper; r++)
    rank_cls[r] = (int)(std::lower_bound(cls_w.begin(), cls_w.end(), widths[r]) - cls_w.begin());
  const int smem_cap = tiled_max_smem();
  for (int c = 0; c < P->n_classes; c++) {
    ClassInfo& ci = P->cls[c];
    ci.L = cls_w[c];
    ci.pmax = 0;
    for (int r = 0; r < nper; r++)
      if (rank_cls[r] == c) ci.pmax = std::max(ci.pmax, periods[r]);
    ci.A = P->T + ci.pmax - 1;
    const size_t per_group = group_bytes(ci.A, ci.L);
    int G = P->NT / ci.L;
    while (G > 0 && (size_t)G * per_group > (size_t)smem_cap) G--;
    if (G == 0) {
      gb_set_error(GB_ERR_CAPACITY,
                   "tile %d with period %d needs %zu B of shared memory (limit %d)", P->T,
                   ci.pmax, per_group, smem_cap);
      return GB_ERR_CAPACITY;
    }
    ci.G = G;
  }
  P->smem_grid = tiled_smem_grid(P->cls, P->n_classes, P->NT);
  P->smem_degrid = tiled_smem_degrid(P->cls, P->n_classes, P->NT);
  P->ctas_per_sm_grid = tiled_ctas_per_sm(P, true);
  for (int st = 0; st < 3; st++) P->ctas_per_sm_degrid[st] = tiled_ctas_per_sm(P, false, st);

  // ---- device tables
  {
    size_t bytes = 0;
    auto place = [&](size_t n) {
      const size_t at = bytes;
      bytes += (n + 255) & ~(size_t)255;
      return at;
    };
    const size_t plane = place(sizeof(int32_t) * n_vis), order = place(sizeof(int32_t) * n_vis);
    const size_t sup = place(sizeof(int32_t) * np), offs = place(sizeof(int64_t) * np);
    const size_t planes = place(sizeof(PlaneInfo) * np), queue = place(sizeof(int32_t) * 3);
    if ((rc = dalloc(&P->d_tables, bytes))) return rc;
    P->d_plane = (int32_t*)(P->d_tables + plane);
    P->d_order = (int32_t*)(P->d_tables + order);
    P->d_supports = (int32_t*)(P->d_tables + sup);
    P->d_offsets = (int64_t*)(P->d_tables + offs);
    P->d_planes = (PlaneInfo*)(P->d_tables + planes);
    P->d_queue = (int32_t*)(P->d_tables + queue);
  }
  // [0], [1]: work-queue heads of the grid and degrid kernels; [2]: device
  // error word (a TMA stage completion not seen in time)
  GB_CUDA_TRY(cudaMemsetAsync(P->d_queue, 0, 3 * sizeof(int32_t), s));
  GB_CUDA_TRY(cudaMemcpyAsync(P->d_supports, geo->supports, sizeof(int32_t) * np,
                              cudaMemcpyHostToDevice, s));
  GB_CUDA_TRY(cudaMemcpyAsync(P->d_offsets, geo->gcf_offsets, sizeof(int64_t) * np,
                              cudaMemcpyHostToDevice, s));
  GB_CUDA_TRY(cudaMemcpyAsync(P->d_planes, P->planes.data(), sizeof(PlaneInfo) * np,
                              cudaMemcpyHostToDevice, s));
  PlanDev& D = P->dev;
  D.n_vis = n_vis;
  D.uvw = d_uvw;
  D.uvw_stride = uvw_stride;
  D.plane = P->d_plane;
  D.order = P->d_order;
  D.supports = P->d_supports;
  D.gcf_offsets = P->d_offsets;
  D.scale = geo->scale;
  D.grid_size = geo->grid_size;
  D.margin = geo->margin;
  D.ext_x = geo->ext_x;
  D.ext_y = geo->ext_y;
  D.pitch = geo->pitch;

  // ---- histogram
  P->ntx = (geo->ext_x + P->T - 1) / P->T;
  P->nty = (geo->ext_y + P->T - 1) / P->T;
  const int64_t nkeys = (int64_t)P->ntx * P->nty * nper;
  if (nkeys >= (int64_t)INT32_MAX) {
    gb_set_error(GB_ERR_CAPACITY, "too many (tile, period) bins");
    return GB_ERR_CAPACITY;
  }
  // per-visibility order: one bucket per tile (the footprint corner's) and a
  // last one for the visibilities no kernel grids; both histograms lie one
  // after the other and are scanned together
  const int64_t ntiles = (int64_t)P->ntx * P->nty, nvkeys = ntiles + 1, all = nkeys + nvkeys;
  const int64_t nci = ntiles * P->n_classes;
  const int64_t nsums = std::max(scan_blocks(all), scan_blocks(nci));
  // scratch: counters and histograms (zeroed), their scan, the items' counts and
  // scan, scan sums, the visibilities' cells
  const size_t cnt_bytes = (sizeof(PlanCounts) + 255) & ~(size_t)255;
  const size_t words = (size_t)(all + (all + 1) + nci + (nci + 1) + nsums + 1) & ~(size_t)1;
  unsigned char* d = nullptr;
  if ((rc = dalloc(&d, cnt_bytes + sizeof(int32_t) * words + sizeof(VisCell) * n_vis))) return rc;
  struct Tmp {
    void* p;
    ~Tmp() { cudaFree(p); }
  } tmp{d};
  PlanCounts* d_cnt = (PlanCounts*)d;
  int32_t* d_hist = (int32_t*)(d + cnt_bytes);
  int32_t* d_vhist = d_hist + nkeys;
  int32_t* d_offs = d_hist + all;
  int32_t* d_icount = d_offs + all + 1;
  int32_t* d_ifirst = d_icount + nci;
  uint32_t* d_sums = (uint32_t*)(d_ifirst + nci + 1);
  VisCell* d_cells = (VisCell*)(d_hist + words);
  GB_CUDA_TRY(cudaMemsetAsync(d, 0, cnt_bytes + sizeof(int32_t) * all, s));
  if (n_vis > 0) {
    const int blocks = std::min(blocks_for(n_vis, 256), sm_count() * 8);
    k_plan_count<<<blocks, 256, 0, s>>>(
        D, P->d_planes, d_plane_in, P->d_plane, d_cells, np, geo->w_low, geo->w_high, P->T, P->ntx,
        nper, d_hist, d_vhist, d_cnt);
    k_rank_sums<<<blocks_for(nkeys, 4096), 256, 0, s>>>(d_hist, nkeys, nper, d_cnt);
    GB_CUDA_TRY(cudaGetLastError());
  }
  if ((rc = scan_keys(d_hist, all, d_offs, d_sums, s))) return rc;

  // cost model, in thread-group steps: a piece of period P costs ceil(P^2/L)
  // tap rounds plus one for its record; an item adds zeroing + flush of its
  // A x A accumulator.
  ItemRule R{};
  R.nper = nper;
  R.nclass = P->n_classes;
  for (int c = 0; c < P->n_classes; c++) {
    const ClassInfo& ci = P->cls[c];
    R.lo[c] = nper;
    R.fixed[c] = (float)(2 * ((ci.A * ci.A + ci.L - 1) / ci.L));
  }
  for (int r = 0; r < nper; r++) {
    const int c = rank_cls[r];
    const ClassInfo& ci = P->cls[c];
    R.rec[r] = (float)((periods[r] * periods[r] + ci.L - 1) / ci.L + 1);
    R.per_cta[r] = (double)R.rec[r] / ci.G;
    R.period[r] = (int16_t)periods[r];
    R.lo[c] = std::min(R.lo[c], r);
    R.hi[c] = std::max(R.hi[c], r + 1);
    // split-row stride residue: the one that minimises the modelled stage cost
    // of pieces of this period (they pair P / 2 taps per row when P is even); an
    // item takes that of its largest run, which comes within 1 % of minimising
    // over all of its runs on the benchmark workloads
    R.residue[r] = -1;
    const int SW = degrid_subwarp(ci.pmax);
    double bc = 0;
    for (int m = 0; m < 16 && !(periods[r] & 1); m++) {
      const double c2 = split_stage_cost(periods[r] / 2, m, SW);
      if (R.residue[r] < 0 || c2 < bc) {
        R.residue[r] = (int8_t)m;
        bc = c2;
      }
    }
  }
  R.pieces = (double)P->bpc * std::max(1, sm_count() * std::max(1, P->ctas_per_sm_grid));
  const int iblocks = (int)((nci + kItemThreads - 1) / kItemThreads);
  k_plan_items<<<iblocks, kItemThreads, 0, s>>>(R, ntiles, P->ntx, d_offs, d_cnt, d_icount, nullptr, nullptr,
                                       nullptr);
  GB_CUDA_TRY(cudaGetLastError());
  if ((rc = scan_keys(d_icount, nci, d_ifirst, d_sums, s))) return rc;
  k_plan_classes<<<1, 32, 0, s>>>(d_ifirst, ntiles, P->n_classes, d_cnt);
  GB_CUDA_TRY(cudaGetLastError());
  PlanCounts cnt;
  GB_CUDA_TRY(cudaMemcpyAsync(&cnt, d_cnt, sizeof(cnt), cudaMemcpyDeviceToHost, s));
  GB_CUDA_TRY(cudaStreamSynchronize(s));
  P->kept = (int64_t)cnt.kept;
  P->taps = (int64_t)cnt.taps;
  P->n_recs = (int64_t)cnt.recs;
  P->taps_paired = (int64_t)cnt.paired;
  P->tiles_used = (int64_t)cnt.tiles;
  if (P->n_recs >= (int64_t)INT32_MAX) {
    gb_set_error(GB_ERR_CAPACITY, "more than 2^31 footprint pieces");
    return GB_ERR_CAPACITY;
  }
  const int n_items = cnt.class_first[P->n_classes];
  P->class_items.clear();
  for (int c = 0; c < P->n_classes; c++)
    P->class_items.push_back(cnt.class_first[c + 1] - cnt.class_first[c]);

  // ---- records and items
  // (the raw costs lie behind the raw items, the bundles behind the items)
  unsigned char* raw = nullptr;
  if ((rc = dalloc(&P->d_recs, P->n_recs)) ||
      (rc = dalloc(&raw, (sizeof(Item) + sizeof(float)) * n_items)))
    return rc;
  P->d_raw_items = (Item*)raw;
  P->d_raw_cost = (float*)(P->d_raw_items + n_items);
  GB_CUDA_TRY(cudaMemsetAsync(d_hist, 0, sizeof(int32_t) * all, s));  // reused as cursors
  if (n_vis > 0)
    k_plan_fill<<<blocks_for(n_vis, 256), 256, 0, s>>>(D, P->d_planes, d_cells, P->T, P->ntx, nper,
                                                       d_offs, d_hist, P->d_recs, d_offs + nkeys,
                                                       d_vhist, P->d_order);
  k_plan_items<<<iblocks, kItemThreads, 0, s>>>(R, ntiles, P->ntx, d_offs, d_cnt, nullptr, d_ifirst,
                                       P->d_raw_items, P->d_raw_cost);
  GB_CUDA_TRY(cudaGetLastError());
  // a batch member's items go into the batch's own tables instead
  P->n_items = n_items;
  if (P->own_work) {
    P->n_bundles = count_bundles(P->class_items, P->cls, 1);
    unsigned char* work = nullptr;
    if ((rc = dalloc(&work, sizeof(Item) * n_items + sizeof(Bundle) * P->n_bundles))) return rc;
    P->d_items = (Item*)work;
    P->d_bundles = (Bundle*)(P->d_items + n_items);
    if ((rc = bundle_items(P->d_raw_items, P->d_raw_cost, nullptr, n_items, P->class_items, P->cls,
                           1, P->d_items, P->d_bundles, s)))
      return rc;
    P->release_raw();
  } else {
    GB_CUDA_TRY(cudaStreamSynchronize(s));
  }
  return GB_OK;
}

}  // namespace gb

using namespace gb;

extern "C" int gb_plan_create(const gb_geometry* geo, int64_t n_vis, const double* d_uvw,
                              int64_t uvw_stride, const int32_t* d_plane, void* stream,
                              gb_plan** out) {
  return gb::plan_create(geo, n_vis, d_uvw, uvw_stride, d_plane, stream, true, out);
}

int gb::plan_create(const gb_geometry* geo, int64_t n_vis, const double* d_uvw,
                    int64_t uvw_stride, const int32_t* d_plane, void* stream, bool own_work,
                    gb_plan** out) {
  if (!out) {
    gb_set_error(GB_ERR_ARG, "gb_plan_create: NULL out");
    return GB_ERR_ARG;
  }
  *out = nullptr;
  if (!geo || n_vis < 0 || n_vis > (int64_t)INT32_MAX || (n_vis > 0 && !d_uvw) ||
      uvw_stride < 3 || geo->n_planes < 1 || geo->n_planes > GB_MAX_PLANES || !geo->supports ||
      !geo->gcf_offsets || geo->ext_x <= 0 || geo->ext_y <= 0 || geo->pitch < geo->ext_x ||
      !(geo->scale == geo->scale)) {
    gb_set_error(GB_ERR_ARG, "gb_plan_create: bad geometry or arguments");
    return GB_ERR_ARG;
  }
  int smax = 0;
  for (int p = 0; p < geo->n_planes; p++) {
    const int S = geo->supports[p];
    if (S < 1 || S > GB_MAX_SUPPORT || geo->gcf_offsets[p] < 0) {
      gb_set_error(GB_ERR_ARG, "gb_plan_create: plane %d support %d / offset out of range", p, S);
      return GB_ERR_ARG;
    }
    smax = std::max(smax, S);
  }
  // defaults: the measured best on the benchmark workloads (tile 24 with
  // 256 threads; pieces up to 40 x 40, so supports up to 40 stay whole and a
  // CTA's accumulators still let four CTAs share an SM)
  const int T = geo->tile ? geo->tile : 24;
  const int NT = geo->threads ? geo->threads : 256;
  const int cap = geo->period_cap ? geo->period_cap : (40 * 40 <= 8 * NT ? 40 : 32);
  const int bpc = geo->bundles_per_cta ? geo->bundles_per_cta : 4;
  if (T < 8 || T > 128 || (NT != 128 && NT != 256 && NT != 512) || cap < 8 || cap > 64 ||
      cap * cap > 8 * NT || bpc < 1 || bpc > 64 || geo->ext_x > 32767 * T ||
      geo->ext_y > 32767 * T) {
    gb_set_error(GB_ERR_ARG, "gb_plan_create: unsupported tuning tile=%d threads=%d cap=%d", T, NT,
                 cap);
    return GB_ERR_ARG;
  }
  int device = 0;
  GB_CUDA_TRY(cudaGetDevice(&device));
  gb_plan* P = new gb_plan();
  P->own_work = own_work;
  P->device = device;
  P->T = T;
  P->NT = NT;
  P->pcap = cap;
  P->bpc = bpc;
  P->n_planes = geo->n_planes;
  P->max_support = smax;
  P->supports.assign(geo->supports, geo->supports + geo->n_planes);
  P->gcf_offsets.assign(geo->gcf_offsets, geo->gcf_offsets + geo->n_planes);
  const int rc = build_plan(P, geo, n_vis, d_uvw, uvw_stride, d_plane, (cudaStream_t)stream);
  if (rc) {
    free_plan(P);
    return rc;
  }
  *out = P;
  return GB_OK;
}

extern "C" int gb_plan_destroy(gb_plan* plan) {
  free_plan(plan);
  return GB_OK;
}

extern "C" int gb_plan_stats(const gb_plan* P, int64_t* st) {
  if (!P || !st) {
    gb_set_error(GB_ERR_ARG, "gb_plan_stats: NULL argument");
    return GB_ERR_ARG;
  }
  st[0] = P->kept;
  st[1] = P->taps;
  st[2] = P->n_items;
  st[3] = P->tiles_used;
  st[4] = P->T;
  st[5] = P->max_support;
  st[6] = P->NT;
  return GB_OK;
}

extern "C" int gb_plan_set_stage(gb_plan* P, int32_t stage) {
  if (!P || stage < GB_STAGE_AUTO || stage > GB_STAGE_ROWS) {
    gb_set_error(GB_ERR_ARG, "gb_plan_set_stage: bad argument");
    return GB_ERR_ARG;
  }
  P->stage_pref = stage;
  return GB_OK;
}

extern "C" int gb_plan_device_status(gb_plan* P, int32_t* out2, void* stream) {
  if (!P || !out2) {
    gb_set_error(GB_ERR_ARG, "gb_plan_device_status: NULL argument");
    return GB_ERR_ARG;
  }
  int32_t err = 0;
  cudaStream_t s = (cudaStream_t)stream;
  GB_CUDA_TRY(cudaMemcpyAsync(&err, P->d_queue + 2, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
  GB_CUDA_TRY(cudaMemsetAsync(P->d_queue + 2, 0, sizeof(int32_t), s));
  GB_CUDA_TRY(cudaStreamSynchronize(s));
  out2[0] = err;
  out2[1] = P->last_stage;
  if (err) {
    gb_set_error(GB_ERR_TIMEOUT, "degridding: a TMA stage did not complete in time");
    return GB_ERR_TIMEOUT;
  }
  return GB_OK;
}

extern "C" int gb_plan_export_index(const gb_plan* P, int32_t* d_out5, void* stream) {
  if (!P || !d_out5) {
    gb_set_error(GB_ERR_ARG, "gb_plan_export_index: NULL argument");
    return GB_ERR_ARG;
  }
  if (P->dev.n_vis == 0) return GB_OK;
  k_plan_export<<<blocks_for(P->dev.n_vis, 256), 256, 0, (cudaStream_t)stream>>>(
      P->dev, P->d_supports, d_out5);
  GB_CUDA_TRY(cudaGetLastError());
  return GB_OK;
}

extern "C" int gb_grid_f64(gb_plan* P, const double* d_vis, const double* d_gcf, double* d_grid,
                           void* stream) {
  if (!P || (P->dev.n_vis && (!d_vis || !d_gcf)) || !d_grid) {
    gb_set_error(GB_ERR_ARG, "gb_grid_f64: NULL argument");
    return GB_ERR_ARG;
  }
  if (P->dev.n_vis == 0) return GB_OK;
  return launch_grid_plain64(P, d_vis, d_gcf, d_grid, (cudaStream_t)stream);
}

extern "C" int gb_degrid_f64(gb_plan* P, const double* d_gcf, const double* d_grid, double* d_pred,
                             int32_t mode, void* stream) {
  if (!P || (P->dev.n_vis && (!d_pred || !d_gcf || !d_grid)) || (mode != 0 && mode != 1)) {
    gb_set_error(GB_ERR_ARG, "gb_degrid_f64: bad argument");
    return GB_ERR_ARG;
  }
  if (P->dev.n_vis == 0) return GB_OK;
  return launch_degrid_plain64(P, d_gcf, d_grid, d_pred, mode, P->df, (cudaStream_t)stream);
}

// The FP64 pair under its forward / backward names (see gb_grid_forward).
extern "C" int gb_grid_forward_f64(gb_plan* P, const double* d_gcf, const double* d_vis,
                                   double* d_grid, void* stream) {
  return gb_grid_f64(P, d_vis, d_gcf, d_grid, stream);
}

extern "C" int gb_grid_backward_f64(gb_plan* P, const double* d_gcf, const double* d_grid_grad,
                                    double* d_vis_grad, void* stream) {
  return gb_degrid_f64(P, d_gcf, d_grid_grad, d_vis_grad, 0, stream);
}

extern "C" int gb_degrid_forward_f64(gb_plan* P, const double* d_gcf, const double* d_grid,
                                     double* d_pred, void* stream) {
  return gb_degrid_f64(P, d_gcf, d_grid, d_pred, 0, stream);
}

extern "C" int gb_degrid_backward_f64(gb_plan* P, const double* d_gcf,
                                      const double* d_pred_grad, double* d_grid_grad,
                                      void* stream) {
  return gb_grid_f64(P, d_pred_grad, d_gcf, d_grid_grad, stream);
}
