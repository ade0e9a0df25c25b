// k_nn.cu -- nearest-neighbour data association (CorrespondenceFinderNN,
// correspondencefindernn.cpp:44-97) on the device.
//
// The reference asks FLANN's randomized kd-tree (approximate, 16 checks) for
// the nearest current point within the squared radius in the 6-D space
// (p, s n).  Here the search is exact: the current cloud is bucketed in a
// uniform grid over xyz (cell h); a query searches a box of cells around its
// own whose half-width doubles (1, 2, 4, ... cells) and stops once the lower
// bound on the xyz distance to anything outside the box -- a lower bound of the
// 6-D distance -- exceeds the best squared distance found (or the radius).  Ties
// keep the lowest current index, as the oracle's exhaustive scan does, so the
// order of a cell's points is free.
//
//   k_nn_bounds    bounding box of the current cloud
//   k_nn_count     per current point: its cell, its rank in the cell
//   (CUB scan of the cell counts: the first point of every cell)
//   k_nn_scatter   positions, scaled normals and indices in cell order
//   k_nn_query     eight lanes per reference point: transform, the boxes up to
//                  kNNNear cells, the reference's gates; match[i] = current
//                  index or -1
//   k_nn_far       the points that need a wider search, a CTA each
//   k_nn_pairs     ordered compaction into (ref, cur) pairs
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstring>

#include <cub/device/device_scan.cuh>

#include "common.cuh"
#include "kernels.hpp"

namespace nicp {

constexpr int kNNThreads = 256;
// Box half-width (cells, a power of two) up to which eight lanes search before
// a CTA takes over: 2 against 4 measured 1.10 / 1.41 ms per 10-iteration
// alignment at 320x240 (cells of 0.7 of the mean spacing, see nn_plan).  Both
// are from rooms of that size; the result does not depend on them.
constexpr int kNNNear = 2;
constexpr int kNNFarBlocks = 4 * 148;  // CTAs of the wide search: about what fits at once
constexpr int kRuns = 4;               // runs of points in flight per group of lanes

__device__ __forceinline__ int cell_coord(float v, float origin, float inv_h) {
  return (int)fminf(fmaxf(floorf((v - origin) * inv_h), -1e8f), 1e8f);
}

// Six keys (float_key: minima of x, y, z, then maxima) over the finite points;
// box comes filled with ~0 (minima) and 0 (maxima).
__global__ void __launch_bounds__(256) k_nn_bounds(const float4 *__restrict__ pts, const int *__restrict__ count,
                                                   unsigned *__restrict__ box) {
  const int n = *count;
  unsigned lo[3] = {~0u, ~0u, ~0u}, hi[3] = {0u, 0u, 0u};
  for (int j = blockIdx.x * 256 + threadIdx.x; j < n; j += gridDim.x * 256) {
    const float4 p = pts[j];
    const float v[3] = {p.x, p.y, p.z};
    if (!(isfinite(p.x) && isfinite(p.y) && isfinite(p.z))) continue;
#pragma unroll
    for (int a = 0; a < 3; a++) {
      lo[a] = min(lo[a], float_key(v[a]));
      hi[a] = max(hi[a], float_key(v[a]));
    }
  }
#pragma unroll
  for (int a = 0; a < 3; a++) {
    lo[a] = __reduce_min_sync(0xffffffffu, lo[a]);
    hi[a] = __reduce_max_sync(0xffffffffu, hi[a]);
  }
  if ((threadIdx.x & 31) == 0) {
#pragma unroll
    for (int a = 0; a < 3; a++) {
      atomicMin(box + a, lo[a]);
      atomicMax(box + 3 + a, hi[a]);
    }
  }
}

__global__ void __launch_bounds__(256) k_nn_count(const float4 *__restrict__ pts, int n, NNGrid g,
                                                  int *__restrict__ cells, int *__restrict__ cell_of,
                                                  int *__restrict__ rank) {
  const int j = blockIdx.x * 256 + threadIdx.x;
  if (j >= n) return;
  const float4 p = pts[j];
  const int cx = min(max(cell_coord(p.x, g.origin[0], g.inv_h), 0), g.dim[0] - 1);
  const int cy = min(max(cell_coord(p.y, g.origin[1], g.inv_h), 0), g.dim[1] - 1);
  const int cz = min(max(cell_coord(p.z, g.origin[2], g.inv_h), 0), g.dim[2] - 1);
  const int c = (cz * g.dim[1] + cy) * g.dim[0] + cx;
  cell_of[j] = c;
  rank[j] = atomicAdd(cells + c, 1);
}

// (x, y, z, index) and the normal scaled by nscale (_model2linear,
// correspondencefindernn.cpp:13-27): two 128-bit loads per candidate.
__global__ void __launch_bounds__(256) k_nn_scatter(const float4 *__restrict__ pts, const float4 *__restrict__ nrm,
                                                    int n, float nscale, const int *__restrict__ first,
                                                    const int *__restrict__ cell_of, const int *__restrict__ rank,
                                                    float4 *__restrict__ feat) {
  const int j = blockIdx.x * 256 + threadIdx.x;
  if (j >= n) return;
  const float4 p = pts[j], q = nrm[j];
  const int at = first[cell_of[j]] + rank[j];
  feat[2 * (size_t)at] = make_float4(p.x, p.y, p.z, __int_as_float(j));
  feat[2 * (size_t)at + 1] = make_float4(fm(nscale, q.x), fm(nscale, q.y), fm(nscale, q.z), 0.0f);
}

struct NNExchange {
  float bd[kNNThreads / 32];
  int best[kNNThreads / 32], at[kNNThreads / 32];
};

// A reference point moved by the transform (Tg: rows 0..2, the aligner's
// _T.inverse()), and the nearest current point found so far.
struct NNSearch {
  float3 p, sn, rn;
  float rn2, bd;
  int best, at;

  __device__ __forceinline__ void start(const NNQuery &a, float4 p0, float4 n0) {
    float Tg[12];
#pragma unroll
    for (int k = 0; k < 12; k++) Tg[k] = a.Tg ? a.Tg[k] : a.state->Tgate[k];
    p = xform_point(Tg, p0);
    // sR = T.linear() * nscale, then sR * n
    float sR[12];
#pragma unroll
    for (int r = 0; r < 3; r++) {
#pragma unroll
      for (int c = 0; c < 3; c++) sR[r * 4 + c] = fm(Tg[r * 4 + c], a.nscale);
      sR[r * 4 + 3] = 0.0f;
    }
    sn = xform_normal(sR, n0);
    rn = xform_normal(Tg, n0);
    rn2 = dot3x(rn.x, rn.y, rn.z, rn.x, rn.y, rn.z);
    best = at = -1;
    bd = a.sq;  // a candidate must be closer
  }
  // False where the gates reject whatever is found (no normal, unless they
  // are demoted), or where nothing is at a distance below the radius (a
  // position or normal that is not finite).
  __device__ __forceinline__ bool needed(const NNQuery &a) const {
    return (a.demoted || rn2 != 0.0f) && isfinite(p.x) && isfinite(p.y) && isfinite(p.z) && isfinite(sn.x) &&
           isfinite(sn.y) && isfinite(sn.z);
  }
  __device__ __forceinline__ void visit(const NNQuery &a, int s) {
    take(a.feat[2 * (size_t)s], a.feat[2 * (size_t)s + 1], s);
  }
  __device__ __forceinline__ void take(float4 c, float4 m, int s) {
    const float e0 = fsb(p.x, c.x), e1 = fsb(p.y, c.y), e2 = fsb(p.z, c.z);
    const float e3 = fsb(sn.x, m.x), e4 = fsb(sn.y, m.y), e5 = fsb(sn.z, m.z);
    float d = fm(e0, e0);
    d = fa(d, fm(e1, e1));
    d = fa(d, fm(e2, e2));
    d = fa(d, fm(e3, e3));
    d = fa(d, fm(e4, e4));
    d = fa(d, fm(e5, e5));
    const int j = __float_as_int(c.w);
    if (d < bd || (d == bd && best >= 0 && j < best)) {
      best = j;
      bd = d;
      at = s;
    }
  }
  // the lanes of `mask` all take the best one's: smallest distance, then lowest index
  __device__ __forceinline__ void agree(unsigned mask) {
    const float d = __uint_as_float(__reduce_min_sync(mask, __float_as_uint(bd)));
    const bool mine = bd == d && best >= 0;
    const unsigned j = __reduce_min_sync(mask, mine ? (unsigned)best : ~0u);
    const unsigned who = __ballot_sync(mask, mine && (unsigned)best == j) & mask;
    const int from = __shfl_sync(mask, at, who ? __ffs(who) - 1 : (int)(threadIdx.x & 31));
    bd = d;
    best = who ? (int)j : -1;
    at = who ? from : -1;
  }
  // xyz distance to the cells of index c along an axis, rounded down
  __device__ __forceinline__ float gap(const NNGrid &g, int axis, float v, int c) const {
    const float o = v - g.origin[axis];
    return fmaxf(0.0f, fmaxf((float)c * g.h - o, o - (float)(c + 1) * g.h) - g.slack[axis]);
  }
  // the run [s0, s1) of `feat` that holds the cells c0..c1 of a row whose y
  // and z lie sqrt(g2) away, without the ends that are out of reach
  __device__ __forceinline__ void run(const NNQuery &a, int cz, int cy, int c0, int c1, float g2, int &s0,
                                      int &s1) const {
    const NNGrid &g = a.grid;
    const float reach = sqrtf(fmaxf(0.0f, bd * 1.0001f - g2)) + g.slack[0];
    c0 = max(max(c0, 0), cell_coord(p.x - reach, g.origin[0], g.inv_h) - 1);
    c1 = min(min(c1, g.dim[0] - 1), cell_coord(p.x + reach, g.origin[0], g.inv_h) + 1);
    if (c0 > c1) return;
    const int *row = a.first + (size_t)(cz * g.dim[1] + cy) * g.dim[0];
    s0 = row[c0];
    s1 = row[c1 + 1];
  }
  // G lanes (sub 0..G-1 of `mask`) search together a box of cells around the
  // query's own that doubles (kdone: already searched, or -1) until it holds
  // everything within the best distance (true) or would pass klimit (false):
  // each lane looks up the run of one row, then all lanes go through the runs.
  // Every lane leaves with the best of all: smallest distance, then lowest
  // index.
  // With kWarps > 1 (G = 32) the warps of a CTA take turns at the rows and
  // exchange their best, in `x`, after each box.
  template <int G, int kWarps>
  __device__ __forceinline__ bool search(const NNQuery &a, int sub, unsigned mask, int kdone, int klimit,
                                         NNExchange *x) {
    const int first_row = kWarps > 1 ? G * (int)(threadIdx.x >> 5) : 0;
    const NNGrid &g = a.grid;
    const int qx = cell_coord(p.x, g.origin[0], g.inv_h), qy = cell_coord(p.y, g.origin[1], g.inv_h),
              qz = cell_coord(p.z, g.origin[2], g.inv_h);
    const float loose = fmaxf(g.slack[0], fmaxf(g.slack[1], g.slack[2]));
    // the box that holds the whole grid
    const int kcover = max(max(max(abs(qx), abs(g.dim[0] - 1 - qx)), max(abs(qy), abs(g.dim[1] - 1 - qy))),
                           max(abs(qz), abs(g.dim[2] - 1 - qz)));
    for (int k = kdone < 0 ? 1 : 2 * kdone;; k *= 2) {
      if (k > klimit) return false;
      k = min(k, kcover);
      const int z0 = max(qz - k, 0), z1 = min(qz + k, g.dim[2] - 1), y0 = max(qy - k, 0),
                y1 = min(qy + k, g.dim[1] - 1);
      const int ny = max(y1 - y0 + 1, 0), rows = ny * max(z1 - z0 + 1, 0);
      const int ends = kdone < 0 ? 1 : 2;  // the box before has been searched: a row's two ends
      for (int r0 = first_row; r0 < rows * ends; r0 += G * kWarps) {
        const int r = r0 + sub;
        int s0 = 0, s1 = 0;
        if (r < rows * ends) {
          const int row = r / ends, cz = z0 + row / ny, cy = y0 + row % ny;
          const float gz = gap(g, 2, p.z, cz), gy = gap(g, 1, p.y, cy), g2 = gz * gz + gy * gy;
          const bool whole = max(abs(cz - qz), abs(cy - qy)) > kdone;
          if (g2 <= bd * 1.0001f && !(whole && r % ends))
            run(a, cz, cy, whole || r % ends == 0 ? qx - k : qx + kdone + 1,
                whole || r % ends ? qx + k : qx - kdone - 1, g2, s0, s1);
        }
        unsigned todo = __ballot_sync(mask, s0 < s1) & mask;
        while (todo) {  // kRuns runs at a time: their loads are in flight together
          int at0[kRuns], end[kRuns], most = 0;
#pragma unroll
          for (int u = 0; u < kRuns; u++) {
            const int l = todo ? __ffs(todo) - 1 : (int)(threadIdx.x & 31);
            const int e0 = __shfl_sync(mask, s0, l), e1 = __shfl_sync(mask, s1, l);
            at0[u] = e0 + sub;
            end[u] = todo ? e1 : e0;
            most = max(most, end[u] - e0);
            todo &= todo - 1;  // (0 stays 0)
          }
          for (int done = 0; done < most; done += G) {
            float4 c[kRuns], m[kRuns];
#pragma unroll
            for (int u = 0; u < kRuns; u++) {
              const size_t s = 2 * (size_t)(at0[u] + done);
              if (at0[u] + done < end[u]) {
                c[u] = a.feat[s];
                m[u] = a.feat[s + 1];
              }
            }
#pragma unroll
            for (int u = 0; u < kRuns; u++)
              if (at0[u] + done < end[u]) take(c[u], m[u], at0[u] + done);
          }
        }
        agree(mask);
      }
      if (kWarps > 1) {
        const int wid = threadIdx.x >> 5;
        __syncthreads();  // (the exchange before has been read)
        if (sub == 0) {
          x->bd[wid] = bd;
          x->best[wid] = best;
          x->at[wid] = at;
        }
        __syncthreads();
        const int w = min(sub, kWarps - 1);
        bd = x->bd[w];
        best = x->best[w];
        at = x->at[w];
        agree(mask);
      }
      // (what lies outside the box is more than k h away from the query's
      // nearer side of its cell, so at least k h - rounding from the query)
      const float lb = (float)k * g.h - loose;
      if (k >= kcover || (lb > 0.0f && lb * lb > bd * 1.0001f)) return true;
      kdone = k;
    }
  }
  // the gates (correspondencefindernn.cpp:80-93): the match or -1
  __device__ __forceinline__ int gate(const NNQuery &a) const {
    if (best < 0) return -1;
    const float4 cn = a.cur_nrm[best], cp = a.cur_pts[best];
    const float cn2 = dot3x(cn.x, cn.y, cn.z, cn.x, cn.y, cn.z);
    if (!a.demoted && (rn2 == 0.0f || cn2 == 0.0f)) return -1;
    const float dx = fsb(p.x, cp.x), dy = fsb(p.y, cp.y), dz = fsb(p.z, cp.z);
    if (dot3x(dx, dy, dz, dx, dy, dz) > a.sq) return -1;
    if (isnan(cn.x) || isnan(cn.y) || isnan(cn.z) || isnan(rn.x) || isnan(rn.y) || isnan(rn.z)) return -1;
    if (!a.demoted && dot3x(rn.x, rn.y, rn.z, cn.x, cn.y, cn.z) < a.cos_thr) return -1;
    return best;
  }
};

// Eight lanes per reference point; what is not settled within kNNNear cells
// goes to k_nn_far.
// The kernel is bound by the round trips to the runs and candidates it visits,
// so the work is in visiting fewer, and several at a time: a reference point
// that the gates reject whatever it finds is not searched; the candidate that
// the point had in the loop's previous iteration (`near`) gives a bound to
// start from; rows of cells and ends of rows beyond the best distance are
// skipped, and a row's cells are one run of `feat` (first[] of empty cells
// included).  One thread per point, shell by shell, over cells of 50 points
// took 1.7 ms per query at 320x240 (75 k points, a quarter of them with a
// normal: the others searched the whole radius in vain); now 65 us, and 22 us
// for k_nn_far.
__global__ void __launch_bounds__(kNNThreads) k_nn_query(NNQuery a) {
  __shared__ int hits;
  const int sub = threadIdx.x & 7;
  const unsigned mask = 0xffu << (threadIdx.x & 24);
  const int i = blockIdx.x * (kNNThreads / 8) + (threadIdx.x >> 3);
  const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  const float4 p0 = i < a.nr ? a.ref_pts[i] : zero, n0 = i < a.nr ? a.ref_nrm[i] : zero;
  if (threadIdx.x == 0) hits = 0;
  chain();
  __syncthreads();
  if (i < a.nr) {
    NNSearch q;
    q.start(a, p0, n0);
    bool settled = true;
    if (q.needed(a)) {
      if (a.seeded) {
        const int s = a.near[i];
        if (s >= 0) q.visit(a, s);
      }
      settled = q.search<8, 1>(a, sub, mask, -1, kNNNear, nullptr);
    }
    if (sub == 0) {
      a.near[i] = q.at;
      if (settled) {
        const int m = q.gate(a);
        a.match[i] = m;
        if (m >= 0) atomicAdd(&hits, 1);
      } else {
        a.far[atomicAdd(a.far_count, 1)] = i;
      }
    }
  }
  __syncthreads();
  // (kNNBlock is a multiple of the points of a CTA)
  if (threadIdx.x == 0 && hits) atomicAdd(a.block_hits + blockIdx.x * (kNNThreads / 8) / kNNBlock, hits);
}

// The points whose nearest neighbour lies further away (seen in one view
// only, or where no neighbour has a like normal): a CTA per point.
__global__ void __launch_bounds__(kNNThreads) k_nn_far(NNQuery a) {
  __shared__ NNExchange x;
  chain();
  const int n = *a.far_count;
  for (int w = blockIdx.x; w < n; w += gridDim.x) {
    const int i = a.far[w];
    NNSearch q;
    q.start(a, a.ref_pts[i], a.ref_nrm[i]);
    const int seed = a.near[i];
    if (seed >= 0) q.visit(a, seed);
    q.search<32, kNNThreads / 32>(a, threadIdx.x & 31, 0xffffffffu, kNNNear, INT_MAX, &x);
    if (threadIdx.x == 0) {
      const int m = q.gate(a);
      a.near[i] = q.at;
      a.match[i] = m;
      if (m >= 0) atomicAdd(a.block_hits + i / kNNBlock, 1);
    }
  }
}

// (ref, cur) pairs in reference-index order: a CTA adds the hits of the query
// CTAs before its own, then places its matches by ballots.
// (match and block_hits are written by k_nn_far while this chained kernel
// waits for it: no __restrict__, which would promise the compiler that they
// do not change and let it load them early, or through the read-only path.)
__global__ void __launch_bounds__(kNNBlock) k_nn_pairs(const int *match, int n, const int *block_hits, int32_t *pairs,
                                                       int *num_pairs, int *far_count, int *next_hits) {
  constexpr int kWarps = kNNBlock / 32;
  __shared__ int part[kWarps], hits[kWarps];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  chain();
  int before = 0;
  for (int q = threadIdx.x; q < (int)blockIdx.x; q += kNNBlock) before += block_hits[q];
  before = __reduce_add_sync(0xffffffffu, before);
  const int i = blockIdx.x * kNNBlock + threadIdx.x;
  const int m = i < n ? match[i] : -1;
  const unsigned ok = __ballot_sync(0xffffffffu, m >= 0);
  if (lane == 0) {
    part[wid] = before;
    hits[wid] = __popc(ok);
  }
  __syncthreads();
  int base = 0, own = 0;
#pragma unroll
  for (int w = 0; w < kWarps; w++) {
    base += part[w] + (w < wid ? hits[w] : 0);
    own += part[w] + hits[w];
  }
  if (m >= 0) {
    const size_t at = (size_t)base + __popc(ok & ((1u << lane) - 1u));
    pairs[2 * at] = i;
    pairs[2 * at + 1] = m;
  }
  if (threadIdx.x == 0) {
    next_hits[blockIdx.x] = 0;  // for the next query
    if (blockIdx.x == gridDim.x - 1) {
      *num_pairs = own;
      *far_count = 0;
    }
  }
}

int launch_nn_bounds(const float4 *pts, const int *count, int capacity, unsigned *box, cudaStream_t s) {
  cudaMemsetAsync(box, 0xff, 3 * sizeof(unsigned), s);
  cudaMemsetAsync(box + 3, 0, 3 * sizeof(unsigned), s);
  const int blocks = capacity < 1 ? 1 : (capacity + 2047) / 2048;
  k_nn_bounds<<<blocks, 256, 0, s>>>(pts, count, box);
  return cudaGetLastError() == cudaSuccess ? 0 : 1;
}
float nn_key_float(unsigned key) {
  const unsigned u = (key & 0x80000000u) ? (key & 0x7fffffffu) : ~key;
  float f;
  memcpy(&f, &u, sizeof(f));
  return f;
}

size_t nn_temp_bytes(size_t cells) {
  size_t b = 0;
  cub::DeviceScan::ExclusiveSum(nullptr, b, (const int *)nullptr, (int *)nullptr, (int)cells + 1);
  return b;
}

int launch_nn_build(const NNBuild &b, cudaStream_t s) {
  const int n = b.nc;
  if (n <= 0) return 0;
  const int blocks = (n + 255) / 256;
  const size_t ncells = (size_t)b.grid.dim[0] * b.grid.dim[1] * b.grid.dim[2];
  cudaMemsetAsync(b.cells, 0, 4 * (ncells + 1), s);
  cudaMemsetAsync(b.far_count, 0, b.zero_bytes, s);
  k_nn_count<<<blocks, 256, 0, s>>>(b.cur_pts, n, b.grid, b.cells, b.cell_of, b.rank);
  size_t tb = b.temp_bytes;
  if (cub::DeviceScan::ExclusiveSum(b.temp, tb, b.cells, b.first, (int)ncells + 1, s) != cudaSuccess) return 1;
  k_nn_scatter<<<blocks, 256, 0, s>>>(b.cur_pts, b.cur_nrm, n, b.nscale, b.first, b.cell_of, b.rank, b.feat);
  return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

int launch_nn_correspond(const NNQuery &q, int32_t *pairs, int *num_pairs, bool chained, cudaStream_t s) {
  const int n = q.nr;
  if (n <= 0 || q.nc <= 0) {
    cudaMemsetAsync(num_pairs, 0, sizeof(int), s);
    return cudaGetLastError() == cudaSuccess ? 0 : 1;
  }
  const int blocks = (n + kNNBlock - 1) / kNNBlock;
  launch(chained, k_nn_query, (n + kNNThreads / 8 - 1) / (kNNThreads / 8), kNNThreads, 0, s, q);
  launch(true, k_nn_far, std::min(blocks, kNNFarBlocks), kNNThreads, 0, s, q);
  launch(true, k_nn_pairs, blocks, kNNBlock, 0, s, q.match, n, q.block_hits, pairs, num_pairs, q.far_count,
         q.next_hits);
  return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

}  // namespace nicp
