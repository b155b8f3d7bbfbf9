// GPU cell-list neighbour search emitting the reference's sorted neighbour lists as CSR,
// and the sliced-ELL copy the bond kernels stream.
//
// Same result as buildNeighborList (src/pd/PdCorrespondenceSkeleton.cpp:95-129), element
// for element: tolerance 64 eps max(delta, max|x|) (:30-39), cells of width delta + 2 tol,
// the 27 surrounding cells searched, a candidate kept when sqrt(dx^2+dy^2+dz^2) <= delta+tol
// with the reference's operation order and IEEE rounding (no FMA contraction), each row in
// ascending index order. Because correctly rounded sqrt is monotone, the test
// RN(sqrt(s)) <= r is replaced by the equivalent s <= s*, s* the largest double whose
// rounded root does not exceed r (found once on the host).
//
// Device passes: |x| max reduction; cell coordinates and their bounding box; counting sort
// of points into a dense cell grid; the matches of every point counted; an exclusive scan
// gives row_ptr; the matches written in ascending order.
//
// The search runs a block per cell, or several (k_nb_cell): the points of the 27 cells around it are sorted by
// index once for all of its points, so a row's matches come out in order by ballot compaction and no row is
// sorted by itself. Distances are decided in FP32, in units of the cell width and relative to a point of the
// cell, outside a margin of 2e-5 of the squared radius (ten times their error), and by the exact test within it;
// chunks of 32 candidates whose bounding box lies beyond the radius are skipped. Where the points are too
// sparse or too dense for that (fewer than kMinCellPoints a cell on average, or more than kMaxCandidates around
// one), a warp per point searches the cells and bitonic-sorts its row (k_nb_count, k_nb_fill).
// 250,000 jittered points, horizon 4.015 h, on a B200: count 275 us, fill 395 us (1390 and 2565 per point); both
// issue-bound (73 %), about a third of it sorting and placing the candidates of the 5,096 cells.
#include "vpd_bond.cuh"  // bcast2

#include <algorithm>
#include <cfloat>
#include <climits>
#include <cmath>
#include <vector>

namespace vpd {

// ------------------------------------------------------------------ exclusive scan
constexpr int kScanThreads = 256;
constexpr int kScanItems = 4;
constexpr int kScanTile = kScanThreads * kScanItems;

int64_t scan_tmp_elems(int64_t n) { return (n + kScanTile - 1) / kScanTile + 1; }

// Exclusive scan across a block of kScanThreads threads; *total gets the block sum.
__device__ int64_t block_exclusive_scan(int64_t v, int64_t *total) {
  __shared__ int64_t warp_sums[kScanThreads / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int64_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int64_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o)
      x += y;
  }
  if (lane == 31)
    warp_sums[wid] = x;
  __syncthreads();
  if (wid == 0) {
    int64_t w = lane < kScanThreads / 32 ? warp_sums[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o)
        w += y;
    }
    if (lane < kScanThreads / 32)
      warp_sums[lane] = w;
  }
  __syncthreads();
  const int64_t excl = x - v + (wid > 0 ? warp_sums[wid - 1] : 0);
  *total = warp_sums[kScanThreads / 32 - 1];
  __syncthreads();
  return excl;
}

__global__ void k_scan_reduce(const int32_t *in, int64_t n, int64_t *sums) {
  const int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
  int64_t s = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k)
    if (base + k < n)
      s += in[base + k];
  int64_t total;
  block_exclusive_scan(s, &total);
  if (threadIdx.x == 0)
    sums[blockIdx.x] = total;
}

// Single block: exclusive scan of the per-tile sums in place; sums[nb] = grand total.
__global__ void k_scan_top(int64_t *sums, int64_t nb) {
  int64_t carry = 0;
  for (int64_t base = 0; base < nb; base += kScanTile) {
    int64_t v[kScanItems];
    int64_t local = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
      const int64_t idx = base + (int64_t)threadIdx.x * kScanItems + k;
      v[k] = idx < nb ? sums[idx] : 0;
      local += v[k];
    }
    int64_t total;
    int64_t run = block_exclusive_scan(local, &total) + carry;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
      const int64_t idx = base + (int64_t)threadIdx.x * kScanItems + k;
      if (idx < nb)
        sums[idx] = run;
      run += v[k];
    }
    carry += total;
  }
  if (threadIdx.x == 0)
    sums[nb] = carry;
}

__global__ void k_scan_apply(const int32_t *in, int64_t n, const int64_t *sums, int64_t nb,
                             int64_t *out) {
  const int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
  int64_t v[kScanItems];
  int64_t local = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    v[k] = base + k < n ? in[base + k] : 0;
    local += v[k];
  }
  int64_t total;
  int64_t run = block_exclusive_scan(local, &total) + sums[blockIdx.x];
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    if (base + k < n)
      out[base + k] = run;
    run += v[k];
  }
  if (blockIdx.x == 0 && threadIdx.x == 0)
    out[n] = sums[nb];
}

int scan_exclusive_i32(const int32_t *in, int64_t n, int64_t *out, int64_t *tmp,
                       cudaStream_t s) {
  const int64_t nb = (n + kScanTile - 1) / kScanTile;
  if (nb == 0) {
    VPD_CUDA(cudaMemsetAsync(out, 0, sizeof(int64_t), s));
    return VPD_OK;
  }
  k_scan_reduce<<<(unsigned)nb, kScanThreads, 0, s>>>(in, n, tmp);
  k_scan_top<<<1, kScanThreads, 0, s>>>(tmp, nb);
  k_scan_apply<<<(unsigned)nb, kScanThreads, 0, s>>>(in, n, tmp, nb, out);
  VPD_CUDA(cudaGetLastError());
  return VPD_OK;
}

// ------------------------------------------------------------------ neighbour kernels
// reduce words: [0] max row length, [1] flags (1: non-finite coordinate, 2: a row beyond its buffer), [2..4] min
// coordinate, [5..7] max coordinate (order_key), [8..11] of the cells (k_cell_load).
constexpr int kReduceWords = 12;

// Doubles as integers of the same order (a finite number and its key determine each other).
__host__ __device__ __forceinline__ long long order_key(long long bits) {
  return bits < 0 ? bits ^ 0x7fffffffffffffffll : bits;
}
static double key_value(unsigned long long key) {
  const long long bits = order_key((long long)key);
  double v;
  memcpy(&v, &bits, sizeof v);
  return v;
}

__global__ void __launch_bounds__(256) k_bounds(const double4 *xv, int64_t n, unsigned long long *red) {
  long long lo[3] = {LLONG_MAX, LLONG_MAX, LLONG_MAX}, hi[3] = {LLONG_MIN, LLONG_MIN, LLONG_MIN};
  bool bad = false;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const double4 p = xv[i];
    const double c[3] = {p.x, p.y, p.z};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      bad = bad || !isfinite(c[d]);
      const long long k = order_key(__double_as_longlong(c[d]));
      lo[d] = k < lo[d] ? k : lo[d];
      hi[d] = k > hi[d] ? k : hi[d];
    }
  }
  __shared__ long long s_lo[8][3], s_hi[8][3];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const long long a = __shfl_xor_sync(0xffffffffu, lo[d], o);
      const long long b = __shfl_xor_sync(0xffffffffu, hi[d], o);
      lo[d] = a < lo[d] ? a : lo[d];
      hi[d] = b > hi[d] ? b : hi[d];
    }
    if (lane == 0)
      s_lo[warp][d] = lo[d], s_hi[warp][d] = hi[d];
  }
  const bool any = __syncthreads_or(bad);
  if (threadIdx.x < 3) {
    const int d = threadIdx.x;
    long long a = s_lo[0][d], b = s_hi[0][d];
    for (int w = 1; w < 8; ++w)
      a = s_lo[w][d] < a ? s_lo[w][d] : a, b = s_hi[w][d] > b ? s_hi[w][d] : b;
    atomicMin((long long *)red + 2 + d, a);
    atomicMax((long long *)red + 5 + d, b);
  }
  if (any && threadIdx.x == 0)
    atomicOr(&red[1], 1ull);
}

__device__ __forceinline__ long long cell_coord(double x, double cw) {
  return (long long)floor(__ddiv_rn(x, cw));
}

struct GridDev {
  long long lo0, lo1, lo2, d0, d1, d2;
};

__global__ void k_cell_assign(const double4 *xv, int64_t n, double cw, GridDev g, long long *cc, int32_t *cell_of,
                              int32_t *count) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n)
    return;
  const double4 p = xv[i];
  const long long x = cell_coord(p.x, cw), y = cell_coord(p.y, cw), z = cell_coord(p.z, cw);
  cc[3 * i] = x, cc[3 * i + 1] = y, cc[3 * i + 2] = z;
  const long long c = ((x - g.lo0) * g.d1 + (y - g.lo1)) * g.d2 + (z - g.lo2);
  cell_of[i] = (int32_t)c;
  atomicAdd(&count[c], 1);
}

__global__ void k_cell_scatter(const int32_t *cell_of, int64_t n, const int64_t *cell_start,
                               int32_t *cursor, int32_t *sorted) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n)
    return;
  const int32_t c = cell_of[i];
  sorted[cell_start[c] + atomicAdd(&cursor[c], 1)] = (int32_t)i;
}

// |xj - xi|^2 in the reference's order ((a0 a0 + a1 a1) + a2 a2), every operation rounded.
__device__ __forceinline__ bool within(const double4 &pj, const double4 &pi, double dist2_max) {
  const double a0 = __dsub_rn(pj.x, pi.x), a1 = __dsub_rn(pj.y, pi.y), a2 = __dsub_rn(pj.z, pi.z);
  const double s = __dadd_rn(__dadd_rn(__dmul_rn(a0, a0), __dmul_rn(a1, a1)), __dmul_rn(a2, a2));
  return s <= dist2_max;
}

static __device__ __noinline__ bool within_exact(const double4 *xv, int32_t j, int32_t i, double dist2_max) {
  return within(xv[j], xv[i], dist2_max);
}

constexpr int kNbWarps = 8;

// One warp per point: number of neighbours.
__global__ void k_nb_count(const double4 *xv, int64_t n, const long long *cc, GridDev g,
                           const int64_t *cell_start, const int32_t *sorted, double dist2_max,
                           int32_t *len, unsigned long long *red) {
  const int lane = threadIdx.x & 31;
  const int64_t i = (int64_t)blockIdx.x * kNbWarps + (threadIdx.x >> 5);
  if (i >= n)
    return;
  const double4 pi = xv[i];
  const long long c0 = cc[3 * i] - g.lo0, c1 = cc[3 * i + 1] - g.lo1, c2 = cc[3 * i + 2] - g.lo2;
  int cnt = 0;
  for (int dx = -1; dx <= 1; ++dx) {
    const long long x0 = c0 + dx;
    if (x0 < 0 || x0 >= g.d0)
      continue;
    for (int dy = -1; dy <= 1; ++dy) {
      const long long x1 = c1 + dy;
      if (x1 < 0 || x1 >= g.d1)
        continue;
      for (int dz = -1; dz <= 1; ++dz) {
        const long long x2 = c2 + dz;
        if (x2 < 0 || x2 >= g.d2)
          continue;
        const long long cell = (x0 * g.d1 + x1) * g.d2 + x2;
        const int64_t end = cell_start[cell + 1];
        for (int64_t p = cell_start[cell] + lane; p < end; p += 32) {
          const int32_t j = sorted[p];
          if (j != i && within(xv[j], pi, dist2_max))
            ++cnt;
        }
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
  if (lane == 0) {
    len[i] = cnt;
    atomicMax(&red[0], (unsigned long long)cnt);
  }
}

// One warp per point: gather matches into shared memory, bitonic sort, write the row.
__global__ void k_nb_fill(const double4 *xv, int64_t n, const long long *cc, GridDev g,
                          const int64_t *cell_start, const int32_t *sorted, double dist2_max,
                          const int64_t *row_ptr, int32_t *col, int cap,
                          unsigned long long *red) {
  extern __shared__ int32_t nb_smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t i = (int64_t)blockIdx.x * (blockDim.x >> 5) + warp;
  if (i >= n)
    return;
  int32_t *buf = nb_smem + (size_t)warp * cap;
  const double4 pi = xv[i];
  const long long c0 = cc[3 * i] - g.lo0, c1 = cc[3 * i + 1] - g.lo1, c2 = cc[3 * i + 2] - g.lo2;
  const unsigned lt = (1u << lane) - 1u;
  int cnt = 0;
  for (int dx = -1; dx <= 1; ++dx) {
    const long long x0 = c0 + dx;
    if (x0 < 0 || x0 >= g.d0)
      continue;
    for (int dy = -1; dy <= 1; ++dy) {
      const long long x1 = c1 + dy;
      if (x1 < 0 || x1 >= g.d1)
        continue;
      for (int dz = -1; dz <= 1; ++dz) {
        const long long x2 = c2 + dz;
        if (x2 < 0 || x2 >= g.d2)
          continue;
        const long long cell = (x0 * g.d1 + x1) * g.d2 + x2;
        const int64_t start = cell_start[cell], end = cell_start[cell + 1];
        for (int64_t base = start; base < end; base += 32) {
          const int64_t p = base + lane;
          bool keep = false;
          int32_t j = 0;
          if (p < end) {
            j = sorted[p];
            keep = j != i && within(xv[j], pi, dist2_max);
          }
          const unsigned mask = __ballot_sync(0xffffffffu, keep);
          const int slot = cnt + __popc(mask & lt);
          if (keep && slot < cap)
            buf[slot] = j;
          cnt += __popc(mask);
        }
      }
    }
  }
  if (cnt > cap) {  // cannot happen when cap >= the count pass's maximum; reported, not written
    if (lane == 0)
      atomicOr(&red[1], 2ull);
    return;
  }
  int width = 32;
  while (width < cnt)
    width <<= 1;
  for (int t = cnt + lane; t < width; t += 32)
    buf[t] = INT_MAX;
  __syncwarp();
  for (int k = 2; k <= width; k <<= 1)
    for (int jj = k >> 1; jj > 0; jj >>= 1) {
      for (int t = lane; t < width; t += 32) {
        const int partner = t ^ jj;
        if (partner > t) {
          const int32_t a = buf[t], b = buf[partner];
          const bool ascending = (t & k) == 0;
          if ((a > b) == ascending) {
            buf[t] = b;
            buf[partner] = a;
          }
        }
      }
      __syncwarp();
    }
  int32_t *row = col + row_ptr[i];
  for (int t = lane; t < cnt; t += 32)
    row[t] = buf[t];
}

// ------------------------------------------------------------------ search by cell
constexpr int kMaxCandidates = 4096;  // 99 KB of shared memory
// Points per cell from which on a block per cell (38 ns each) is quicker than a warp per point (11, 5.5 and 2.8 ns a point in
// bodies, plates and lines of 1M points, which look into 27, 9 and 3 cells), by the number of directions with more
// than one cell. Lists of 1M points, milliseconds, by cell | by point: 3, 5.7 and 11.7 points a cell of a body 14.1 | 11.3,
// 8.9 | 12.2 and 6.2 | 13.2, 6 and 9 of a plate 6.9 | 5.7 and 5.4 | 6.0, 9 and 20 of a line 3.8 | 3.0 and 2.5 | 3.6.
constexpr int kMinCellPoints[4] = {1, 14, 8, 5};
constexpr int kCellThreads = 256;

// The nine runs of `sorted` that hold the points of the 27 cells around cell c (the three along the last
// dimension are consecutive): run k of lane k < 9.
struct CellRun {
  int64_t begin;
  int count;
};
__device__ __forceinline__ CellRun cell_run(int64_t c, const GridDev &g, const int64_t *cell_start, int k) {
  const long long c2 = c % g.d2, c1 = (c / g.d2) % g.d1, c0 = c / (g.d2 * g.d1);
  const long long x0 = c0 + k / 3 - 1, x1 = c1 + k % 3 - 1;
  if (k >= 9 || x0 < 0 || x0 >= g.d0 || x1 < 0 || x1 >= g.d1)
    return {0, 0};
  const long long row = (x0 * g.d1 + x1) * g.d2;
  const long long lo = c2 > 0 ? c2 - 1 : 0, hi = c2 + 1 < g.d2 ? c2 + 1 : g.d2 - 1;
  const int64_t b = cell_start[row + lo];
  return {b, (int)(cell_start[row + hi + 1] - b)};
}

// load[0] the most candidates of any cell that holds points; of cells with up to kMaxCandidates, load[1] the most
// points, load[2] the most pairs (points times candidates) and load[3] all pairs.
__global__ void k_cell_load(int64_t ncells, GridDev g, const int64_t *cell_start, unsigned long long *load) {
  const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  unsigned total = 0, points = 0;
  if (c < ncells && cell_start[c + 1] > cell_start[c]) {
    for (int k = 0; k < 9; ++k)
      total += (unsigned)cell_run(c, g, cell_start, k).count;
    if (total <= kMaxCandidates)
      points = (unsigned)(cell_start[c + 1] - cell_start[c]);
  }
  const unsigned pairs = points * total;  // below 2^24
  total = __reduce_max_sync(0xffffffffu, total), points = __reduce_max_sync(0xffffffffu, points);
  const unsigned most = __reduce_max_sync(0xffffffffu, pairs), sum = __reduce_add_sync(0xffffffffu, pairs);
  if ((threadIdx.x & 31) == 0 && total) {
    atomicMax(load, (unsigned long long)total);
    atomicMax(load + 1, (unsigned long long)points);
    atomicMax(load + 2, (unsigned long long)most);
    atomicAdd(load + 3, (unsigned long long)sum);
  }
}

// Blocks per cell: one, unless the busiest cell has more than twice its share of the pairs of one block per SM (a body of
// a few cells, or a cluster among sparse points); each block then searches for some of the cell's points, 32 or more, and
// sorts the candidates again. The two calls that build the list, microseconds, a block per cell | so: 3,375 points in one
// cell 9938 | 467, 2,744 points in eight cells 5376 | 442 (3200 both with a warp per point and allocations in the calls).
// At most 65,536 blocks in all: those without points end at once, but each takes its nanoseconds.
static int cell_blocks(const unsigned long long *load, int64_t ncells) {
  const unsigned long long share = std::max(load[3] / 148, 32 * load[0]);
  const unsigned long long wanted = std::min(load[2] / share, (load[1] + 31) / 32);
  return (int)std::max(1ull, std::min(wanted, (unsigned long long)(65536 / ncells)));
}

// Ascending bitonic sort of `width` (a power of two, at least 32) shared-memory ints by the whole block.
__device__ __forceinline__ void block_sort(int32_t *a, int width) {
  for (int k = 2; k <= width; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int t = threadIdx.x; t < width / 2; t += kCellThreads) {
        const int lo = 2 * t - (t & (j - 1)), hi = lo + j;
        const int32_t x = a[lo], y = a[hi];
        if ((x > y) == ((lo & k) == 0))
          a[lo] = y, a[hi] = x;
      }
      __syncthreads();
    }
}

// Sorts the `total` distinct ints of a (lowest `lo`) by setting their bits in `bits` (words 32-bit words, range of the
// values at most 32 words) and listing the set bits: a fraction of the comparisons' work where the indices around a
// cell lie close together, as those of a lattice do.
__device__ __forceinline__ void block_sort_bits(int32_t *a, int total, int32_t lo, uint32_t *bits, int words) {
  __shared__ int s_warp[kCellThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int w = threadIdx.x; w < words; w += kCellThreads)
    bits[w] = 0u;
  __syncthreads();
  for (int t = threadIdx.x; t < total; t += kCellThreads) {
    const uint32_t b = (uint32_t)(a[t] - lo);
    atomicOr(bits + (b >> 5), 1u << (b & 31));
  }
  __syncthreads();
  const int per = (words + kCellThreads - 1) / kCellThreads;
  const int w0 = min(words, (int)threadIdx.x * per), w1 = min(words, w0 + per);
  int mine = 0;
  for (int w = w0; w < w1; ++w)
    mine += __popc(bits[w]);
  int incl = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o)
      incl += y;
  }
  if (lane == 31)
    s_warp[warp] = incl;
  __syncthreads();
  int pos = incl - mine;
  for (int k = 0; k < warp; ++k)
    pos += s_warp[k];
  for (int w = w0; w < w1; ++w)
    for (uint32_t m = bits[w]; m; m &= m - 1)
      a[pos++] = lo + 32 * w + (__ffs(m) - 1);
  __syncthreads();
}

__device__ __forceinline__ float warp_min(float v) {
  float r;
  asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ float warp_max(float v) {
  float r;
  asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}

struct CellSearch {
  double inv_width, dist2_max;
  float r2lo, r2hi;  // (radius / cell width)^2 less and plus the margin
};

// gridDim.y blocks per cell (blockIdx.x). FILL: the rows of the cell's points into col; else their lengths into len (and
// the largest to *longest).
template <bool FILL>
__global__ void __launch_bounds__(kCellThreads) k_nb_cell(const double4 *xv, GridDev g, const int64_t *cell_start,
                                                          const int32_t *sorted, CellSearch cs, int width,
                                                          const int64_t *row_ptr, int32_t *col, int32_t *len,
                                                          unsigned long long *longest) {
  extern __shared__ __align__(16) unsigned char s_cell[];
  float4 *cand = reinterpret_cast<float4 *>(s_cell);  // position relative to the cell's first point, index
  int32_t *index = reinterpret_cast<int32_t *>(cand + width);
  int32_t *own = index + width;                             // the cell's points, in ascending order
  float *box = reinterpret_cast<float *>(own + width);      // per 32 candidates: lowest x, y, z, highest x, y, z
  __shared__ int64_t s_begin[9];
  __shared__ int s_off[10], s_lo, s_hi;
  const int64_t c = blockIdx.x, first = cell_start[c], last = cell_start[c + 1];
  // this block's share of the cell's points (in ascending order): pairs of points for every warp
  constexpr int kPairs = 2 * (kCellThreads / 32);
  const int points = (int)(last - first);
  const int share = ((points + (int)gridDim.y - 1) / (int)gridDim.y + kPairs - 1) / kPairs * kPairs;
  const int q0 = (int)blockIdx.y * share, q1 = min(points, q0 + share);
  if (q0 >= q1)
    return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x < 32) {
    const CellRun r = cell_run(c, g, cell_start, lane);
    int off = r.count;
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, off, o);
      if (lane >= o)
        off += y;
    }
    if (lane < 9)
      s_begin[lane] = r.begin, s_off[lane + 1] = off;
    if (lane == 0)
      s_off[0] = 0;
  }
  __syncthreads();
  const int total = s_off[9];
  int w2 = 32;
  while (w2 < total)
    w2 <<= 1;
  for (int k = 0; k < 9; ++k)
    for (int t = s_off[k] + threadIdx.x; t < s_off[k + 1]; t += kCellThreads)
      index[t] = sorted[s_begin[k] + (t - s_off[k])];
  for (int t = total + threadIdx.x; t < w2; t += kCellThreads)
    index[t] = INT_MAX;
  int o2 = 32;
  while (o2 < (int)(last - first))
    o2 <<= 1;
  for (int t = threadIdx.x; t < o2; t += kCellThreads)
    own[t] = t < last - first ? sorted[first + t] : INT_MAX;
  if (threadIdx.x == 0)
    s_lo = INT_MAX, s_hi = 0;
  __syncthreads();
  int lo = INT_MAX, hi = 0;
  for (int t = threadIdx.x; t < total; t += kCellThreads)
    lo = min(lo, index[t]), hi = max(hi, index[t]);
  lo = __reduce_min_sync(0xffffffffu, lo), hi = __reduce_max_sync(0xffffffffu, hi);
  if (lane == 0)
    atomicMin(&s_lo, lo), atomicMax(&s_hi, hi);
  __syncthreads();
  const int words = (s_hi - s_lo) / 32 + 1;
  if (words <= 4 * width) {  // the candidates' positions are not there yet: 16 bytes each
    block_sort_bits(index, total, s_lo, reinterpret_cast<uint32_t *>(cand), words);
    block_sort_bits(own, points, s_lo, reinterpret_cast<uint32_t *>(cand), words);
  } else {
    block_sort(index, w2);
    block_sort(own, o2);
  }
  const double4 ref = xv[sorted[first]];
  for (int t = total + threadIdx.x; t < min(width, (total + 31) & ~31); t += kCellThreads)
    cand[t] = make_float4(1.0e18f, 1.0e18f, 1.0e18f, __int_as_float(-1));
  for (int t = threadIdx.x; t < total; t += kCellThreads) {
    const double4 p = xv[index[t]];
    cand[t] = make_float4((float)((p.x - ref.x) * cs.inv_width), (float)((p.y - ref.y) * cs.inv_width),
                          (float)((p.z - ref.z) * cs.inv_width), __int_as_float(index[t]));
  }
  __syncthreads();
  const int chunks = (total + 31) / 32;
  for (int k = warp; k < chunks; k += kCellThreads / 32) {
    const float4 p = cand[min(32 * k + lane, total - 1)];
    const float lo[3] = {warp_min(p.x), warp_min(p.y), warp_min(p.z)};
    const float hi[3] = {warp_max(p.x), warp_max(p.y), warp_max(p.z)};
    if (lane < 6)
      box[6 * k + lane] = lane == 0 ? lo[0] : lane == 1 ? lo[1] : lane == 2 ? lo[2] : lane == 3 ? hi[0] : lane == 4 ? hi[1] : hi[2];
  }
  __syncthreads();
  // two points of the cell at a time, consecutive in index, over the chunks near either: one read of a candidate
  // and packed FP32 arithmetic for both
  const unsigned lt = (1u << lane) - 1u;
  int most = 0;
  for (int q = q0 + 2 * warp; q < q1; q += kPairs) {
    int32_t i[2];
    float x[2], y[2], z[2];
    int32_t *row[2];
    int cnt[2] = {0, 0};
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      i[h] = own[min(q + h, q1 - 1)];
      const double4 pi = xv[i[h]];
      x[h] = (float)((pi.x - ref.x) * cs.inv_width), y[h] = (float)((pi.y - ref.y) * cs.inv_width);
      z[h] = (float)((pi.z - ref.z) * cs.inv_width);
      row[h] = FILL ? col + row_ptr[i[h]] : nullptr;
    }
    const float2 nx = make_float2(-x[0], -x[1]), ny = make_float2(-y[0], -y[1]), nz = make_float2(-z[0], -z[1]);
    for (int k0 = 0; k0 < chunks; k0 += 32) {
      bool near = false;
      if (k0 + lane < chunks) {
        const float *b = box + 6 * (k0 + lane);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float dx = fmaxf(fmaxf(b[0] - x[h], x[h] - b[3]), 0.0f), dy = fmaxf(fmaxf(b[1] - y[h], y[h] - b[4]), 0.0f),
                      dz = fmaxf(fmaxf(b[2] - z[h], z[h] - b[5]), 0.0f);
          near = near || dx * dx + dy * dy + dz * dz <= cs.r2hi;
        }
      }
      for (unsigned m = __ballot_sync(0xffffffffu, near); m; m &= m - 1) {
        const int t = 32 * (k0 + __ffs(m) - 1) + lane;
        const float4 p = cand[t];  // (past the last candidate: one far away)
        const int32_t j = __float_as_int(p.w);
        const float2 dx = __fadd2_rn(bcast2(p.x), nx), dy = __fadd2_rn(bcast2(p.y), ny), dz = __fadd2_rn(bcast2(p.z), nz);
        const float2 s = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
        bool keep[2] = {s.x < cs.r2lo, s.y < cs.r2lo};
        const bool near0 = !keep[0] && s.x <= cs.r2hi, near1 = !keep[1] && s.y <= cs.r2hi;
        if (__any_sync(0xffffffffu, near0 || near1)) {  // rare: out of line, by a uniform branch
          if (near0)
            keep[0] = within_exact(xv, j, i[0], cs.dist2_max);
          if (near1)
            keep[1] = within_exact(xv, j, i[1], cs.dist2_max);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const bool k = keep[h] && j != i[h];
          if (FILL) {
            const unsigned hit = __ballot_sync(0xffffffffu, k);
            if (k && q + h < q1)
              row[h][cnt[h] + __popc(hit & lt)] = j;
            cnt[h] += __popc(hit);
          } else {
            cnt[h] += k;
          }
        }
      }
    }
    if (!FILL)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int total_h = __reduce_add_sync(0xffffffffu, cnt[h]);
        if (lane == 0)
          len[i[h]] = total_h;
        most = max(most, total_h);
      }
  }
  if (!FILL && lane == 0 && most > 0)
    atomicMax(longest, (unsigned long long)most);
}

// Shared memory of k_nb_cell for `candidates` points around a cell.
static int cell_width(int candidates) {
  int w = 32;
  while (w < candidates)
    w <<= 1;
  return w;
}
static size_t cell_smem(int width) {
  return (size_t)width * (sizeof(float4) + 2 * sizeof(int32_t)) + (size_t)(width / 32) * 6 * sizeof(float);
}

template <bool FILL>
static int launch_cells(const double4 *xv, const NeighborGrid &grid, const NeighborScratch &scr, const int64_t *row_ptr,
                        int32_t *col, cudaStream_t s) {
  const GridDev g{grid.lo[0], grid.lo[1], grid.lo[2], grid.dims[0], grid.dims[1], grid.dims[2]};
  const double inv = 1.0 / grid.cell_width, r2 = grid.dist2_max * inv * inv;
  const CellSearch cs{inv, grid.dist2_max, (float)(r2 * (1.0 - 2.0e-5)), (float)(r2 * (1.0 + 2.0e-5))};
  const int width = cell_width(grid.candidates);
  const size_t smem = cell_smem(width);
  // the largest search's amount, whatever this one's: the attribute is the function's, and another thread's call may
  // set it between this one's and its launch
  VPD_CUDA(cudaFuncSetAttribute(k_nb_cell<FILL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)cell_smem(kMaxCandidates)));
  const dim3 blocks((unsigned)grid.ncells, (unsigned)grid.cell_blocks);
  k_nb_cell<FILL><<<blocks, kCellThreads, smem, s>>>(xv, g, scr.cell_start, scr.sorted, cs, width, row_ptr, col, scr.len,
                                                     scr.reduce);
  VPD_CUDA(cudaGetLastError());
  return VPD_OK;
}

// ------------------------------------------------------------------ host orchestration
template <typename T> static int scratch(NeighborScratch &scr, T **p, int64_t count) {
  return workspace_alloc(reinterpret_cast<void **>(p), sizeof(T) * (size_t)std::max<int64_t>(count, 1), scr.stream);
}

int neighbor_scratch_alloc(NeighborScratch &scr, int64_t n, cudaStream_t s) {
  scr.stream = s;
  int rc;
  if ((rc = scratch(scr, &scr.cell_coords, 3 * n)) || (rc = scratch(scr, &scr.cell_of, n)) ||
      (rc = scratch(scr, &scr.sorted, n)) || (rc = scratch(scr, &scr.len, n)) ||
      (rc = scratch(scr, &scr.reduce, kReduceWords)))
    return rc;
  return VPD_OK;
}

int neighbor_scratch_alloc_cells(NeighborScratch &scr, int64_t ncells) {
  const int64_t tmp = std::max(scan_tmp_elems(ncells), scan_tmp_elems(0)) + 8;
  int rc;
  if ((rc = scratch(scr, &scr.cell_count, ncells + 1)) || (rc = scratch(scr, &scr.cell_start, ncells + 1)) ||
      (rc = scratch(scr, &scr.scan_tmp, tmp)))
    return rc;
  return VPD_OK;
}

void neighbor_scratch_free(NeighborScratch &scr) {
  void *const all[] = {scr.cell_coords, scr.cell_of,    scr.sorted,     scr.len,
                       scr.reduce,      scr.cell_count, scr.cell_start, scr.scan_tmp};
  for (void *p : all)
    workspace_free(p, scr.stream);
  scr = NeighborScratch{};
}

static unsigned grid_for(int64_t n, int threads) {
  return (unsigned)std::max<int64_t>(1, std::min<int64_t>((n + threads - 1) / threads, 148 * 16));
}

int neighbor_count(const double4 *xv, int64_t n, double horizon, int64_t *row_ptr,
                   NeighborGrid &grid, NeighborScratch &scr, cudaStream_t s) {
  if (!(horizon > 0.0))
    return set_error(VPD_ERR_INVALID, "PD horizon must be positive.");
  if (n <= 0 || n > INT32_MAX)
    return set_error(VPD_ERR_INVALID, "neighbour search needs 1 <= n < 2^31 points");
  unsigned long long init[kReduceWords] = {0, 0,
                                           (unsigned long long)LLONG_MAX, (unsigned long long)LLONG_MAX,
                                           (unsigned long long)LLONG_MAX, (unsigned long long)LLONG_MIN,
                                           (unsigned long long)LLONG_MIN, (unsigned long long)LLONG_MIN, 0, 0, 0, 0};
  VPD_CUDA(cudaMemcpyAsync(scr.reduce, init, sizeof init, cudaMemcpyHostToDevice, s));
  k_bounds<<<grid_for(n, 256), 256, 0, s>>>(xv, n, scr.reduce);
  unsigned long long red[kReduceWords];
  VPD_CUDA(cudaMemcpyAsync(red, scr.reduce, sizeof red, cudaMemcpyDeviceToHost, s));
  VPD_CUDA(cudaStreamSynchronize(s));
  if (red[1])
    return set_error(VPD_ERR_NONFINITE, "Nonfinite PD coordinate.");
  double low[3], high[3], maxabs = 0.0;
  for (int d = 0; d < 3; ++d) {
    low[d] = key_value(red[2 + d]), high[d] = key_value(red[5 + d]);
    maxabs = std::max(maxabs, std::max(std::fabs(low[d]), std::fabs(high[d])));
  }
  const double scale = std::max(horizon, maxabs);
  grid.tolerance = 64.0 * DBL_EPSILON * scale;
  grid.radius = horizon + grid.tolerance;
  grid.cell_width = horizon + 2.0 * grid.tolerance;
  double s2 = grid.radius * grid.radius;
  while (std::sqrt(std::nextafter(s2, INFINITY)) <= grid.radius)
    s2 = std::nextafter(s2, INFINITY);
  while (std::sqrt(s2) > grid.radius)
    s2 = std::nextafter(s2, 0.0);
  grid.dist2_max = s2;

  // the cells of the extreme coordinates bound all cells (cell_coord does not decrease with x)
  double cells = 1.0;
  for (int d = 0; d < 3; ++d) {
    grid.lo[d] = (long long)std::floor(low[d] / grid.cell_width);
    grid.dims[d] = (long long)std::floor(high[d] / grid.cell_width) - grid.lo[d] + 1;
    cells *= (double)grid.dims[d];
  }
  if (cells > (double)kMaxCells)
    return set_error(VPD_ERR_CAPACITY, "neighbour cell grid exceeds 2^28 cells; the points are "
                                       "too spread out relative to the horizon");
  grid.ncells = grid.dims[0] * grid.dims[1] * grid.dims[2];
  if (!scr.cell_count) {
    int rc = neighbor_scratch_alloc_cells(scr, grid.ncells);
    if (rc)
      return rc;
  }
  const GridDev g{grid.lo[0], grid.lo[1], grid.lo[2], grid.dims[0], grid.dims[1], grid.dims[2]};
  VPD_CUDA(cudaMemsetAsync(scr.cell_count, 0, sizeof(int32_t) * (size_t)(grid.ncells + 1), s));
  const unsigned pb = (unsigned)((n + 255) / 256);
  k_cell_assign<<<pb, 256, 0, s>>>(xv, n, grid.cell_width, g, scr.cell_coords, scr.cell_of, scr.cell_count);
  int rc = scan_exclusive_i32(scr.cell_count, grid.ncells, scr.cell_start, scr.scan_tmp, s);
  if (rc)
    return rc;
  VPD_CUDA(cudaMemsetAsync(scr.cell_count, 0, sizeof(int32_t) * (size_t)(grid.ncells + 1), s));
  k_cell_scatter<<<pb, 256, 0, s>>>(scr.cell_of, n, scr.cell_start, scr.cell_count, scr.sorted);
  // the search by cell needs a few points a cell, candidates that fit shared memory, and a cell width whose
  // reciprocal and square are ordinary numbers
  grid.candidates = 0;
  const int directions = (grid.dims[0] > 1) + (grid.dims[1] > 1) + (grid.dims[2] > 1);
  if (grid.ncells * kMinCellPoints[directions] <= n && grid.cell_width > 1.0e-100 && grid.cell_width < 1.0e100) {
    k_cell_load<<<(unsigned)((grid.ncells + 255) / 256), 256, 0, s>>>(grid.ncells, g, scr.cell_start, scr.reduce + 8);
    VPD_CUDA(cudaMemcpyAsync(red, scr.reduce, sizeof red, cudaMemcpyDeviceToHost, s));
    VPD_CUDA(cudaStreamSynchronize(s));
    if (red[8] <= (unsigned long long)kMaxCandidates)
      grid.candidates = (int)red[8], grid.cell_blocks = cell_blocks(red + 8, grid.ncells);
  }
  if (grid.candidates) {
    if ((rc = launch_cells<false>(xv, grid, scr, nullptr, nullptr, s)))
      return rc;
  } else {
    const unsigned wb = (unsigned)((n + kNbWarps - 1) / kNbWarps);
    k_nb_count<<<wb, 32 * kNbWarps, 0, s>>>(xv, n, scr.cell_coords, g, scr.cell_start, scr.sorted,
                                            grid.dist2_max, scr.len, scr.reduce);
  }
  // reuse the cell scan scratch when large enough, else the row scan needs its own
  int64_t *tmp = scr.scan_tmp;
  int64_t *own = nullptr;
  if (scan_tmp_elems(n) > std::max(scan_tmp_elems(grid.ncells), scan_tmp_elems(0)) + 8) {
    if ((rc = scratch(scr, &own, scan_tmp_elems(n))))
      return rc;
    tmp = own;
  }
  rc = scan_exclusive_i32(scr.len, n, row_ptr, tmp, s);
  VPD_CUDA(cudaMemcpyAsync(red, scr.reduce, sizeof red, cudaMemcpyDeviceToHost, s));
  VPD_CUDA(cudaStreamSynchronize(s));
  workspace_free(own, s);
  if (rc)
    return rc;
  grid.max_len = (int)red[0];
  if (grid.max_len > kMaxRow)
    return set_error(VPD_ERR_CAPACITY, "a point has more than 8192 neighbours");
  return VPD_OK;
}

int neighbor_fill(const double4 *xv, int64_t n, const int64_t *row_ptr, int32_t *col,
                  const NeighborGrid &grid, const NeighborScratch &scr, cudaStream_t s) {
  if (grid.candidates) {  // the rows have the counted lengths: nothing to report
    const int rc = launch_cells<true>(xv, grid, scr, row_ptr, col, s);
    if (rc)
      return rc;
    VPD_CUDA(cudaStreamSynchronize(s));
    return VPD_OK;
  }
  int cap = 32;
  while (cap < grid.max_len)
    cap <<= 1;
  const int warps = std::max(1, std::min(8, (48 * 1024) / (cap * 4)));
  const size_t smem = (size_t)warps * cap * sizeof(int32_t);
  const GridDev g{grid.lo[0], grid.lo[1], grid.lo[2], grid.dims[0], grid.dims[1], grid.dims[2]};
  const unsigned blocks = (unsigned)((n + warps - 1) / warps);
  k_nb_fill<<<blocks, 32 * warps, smem, s>>>(xv, n, scr.cell_coords, g, scr.cell_start,
                                             scr.sorted, grid.dist2_max, row_ptr, col, cap,
                                             scr.reduce);
  VPD_CUDA(cudaGetLastError());
  unsigned long long red[kReduceWords];
  VPD_CUDA(cudaMemcpyAsync(red, scr.reduce, sizeof red, cudaMemcpyDeviceToHost, s));
  VPD_CUDA(cudaStreamSynchronize(s));
  if (red[1] & 2ull)
    return set_error(VPD_ERR_CAPACITY, "neighbour row exceeded its buffer");
  return VPD_OK;
}

// ------------------------------------------------------------------ sliced ELL
__global__ void k_sell_width(const int64_t *row_ptr, int64_t n, int64_t nslices, int32_t *len,
                             int32_t *width32) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= nslices * 32)
    return;
  int l = 0;
  if (i < n) {
    l = (int)(row_ptr[i + 1] - row_ptr[i]);
    len[i] = l;
  }
  int m = l;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const int y = __shfl_xor_sync(0xffffffffu, m, o);
    m = y > m ? y : m;
  }
  if ((threadIdx.x & 31) == 0)
    width32[i >> 5] = 32 * m;
}

__global__ void k_sell_fill(const int64_t *row_ptr, const int32_t *col, int64_t n,
                            int64_t nslices, const int64_t *slice_off, int32_t *sell) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= nslices * 32)
    return;
  const int64_t sl = i >> 5;
  const int lane = (int)(i & 31);
  const int width = (int)((slice_off[sl + 1] - slice_off[sl]) >> 5);
  const int l = i < n ? (int)(row_ptr[i + 1] - row_ptr[i]) : 0;
  const int32_t self = i < n ? (int32_t)i : 0;
  int32_t *out = sell + slice_off[sl] + lane;
  for (int k = 0; k < width; ++k)
    out[32 * k] = k < l ? col[row_ptr[i] + k] : self;
}

int build_sell(const int64_t *row_ptr, const int32_t *col, int64_t n, int32_t **len_out,
               int64_t **slice_off_out, int32_t **sell_out, int64_t *sell_total,
               cudaStream_t s) {
  const int64_t nslices = (n + 31) / 32;
  int32_t *len = nullptr, *width32 = nullptr, *sell = nullptr;
  int64_t *slice_off = nullptr, *tmp = nullptr;
  VPD_CUDA(cudaMalloc(&len, sizeof(int32_t) * (size_t)(nslices * 32)));
  VPD_CUDA(cudaMemsetAsync(len, 0, sizeof(int32_t) * (size_t)(nslices * 32), s));
  VPD_CUDA(cudaMalloc(&width32, sizeof(int32_t) * (size_t)nslices));
  VPD_CUDA(cudaMalloc(&slice_off, sizeof(int64_t) * (size_t)(nslices + 1)));
  VPD_CUDA(cudaMalloc(&tmp, sizeof(int64_t) * (size_t)scan_tmp_elems(nslices)));
  const unsigned blocks = (unsigned)((nslices * 32 + 255) / 256);
  k_sell_width<<<blocks, 256, 0, s>>>(row_ptr, n, nslices, len, width32);
  int rc = scan_exclusive_i32(width32, nslices, slice_off, tmp, s);
  if (rc)
    return rc;
  int64_t total = 0;
  VPD_CUDA(cudaMemcpyAsync(&total, slice_off + nslices, sizeof total, cudaMemcpyDeviceToHost, s));
  VPD_CUDA(cudaStreamSynchronize(s));
  VPD_CUDA(cudaMalloc(&sell, sizeof(int32_t) * (size_t)std::max<int64_t>(total, 32)));
  k_sell_fill<<<blocks, 256, 0, s>>>(row_ptr, col, n, nslices, slice_off, sell);
  VPD_CUDA(cudaGetLastError());
  VPD_CUDA(cudaStreamSynchronize(s));
  cudaFree(width32);
  cudaFree(tmp);
  *len_out = len;
  *slice_off_out = slice_off;
  *sell_out = sell;
  *sell_total = total;
  return VPD_OK;
}

}  // namespace vpd
