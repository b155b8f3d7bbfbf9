// Module-level entry points of libvpd_gpu.so: the reference's C++ module functions on
// caller-owned device arrays in the reference's point-major layout (Tensor3 row-major,
// neighbour lists as CSR), and the VUMAT plugin entry vumat_adapter_call evaluated on the GPU.
// The bond sums run eight threads per point, the pointwise kernels one.
#include "vpd_math.cuh"
#include "vpd_step.cuh"
#include "vpd_umma.cuh"  // smem_u32

#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

namespace vpd {

__global__ void k_pack_positions(const double *pos, int64_t n, double4 *xv) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n)
    xv[i] = make_double4(pos[3 * i], pos[3 * i + 1], pos[3 * i + 2], 0.0);
}

// ------------------------------------------------------------------ CSR bond sums
// A row's bonds are dealt out to 1, 2, 4 or 8 lanes, whose partial sums a fixed shuffle tree joins. Many lanes read a
// long row's neighbour indices as consecutive words and fill the GPU where points are few; with one lane per row the
// lanes of a warp share the lines of short rows, and neighbouring rows of a regular lattice gather consecutive points.
// The next bond's index is read before the current bond's gathers are used. What bounds the sums is L1 (90 to 96 % of
// its throughput at 154,000 jittered points): the gathers of 32 bonds touch about eight lines a load in any arrangement
// tried.
constexpr int kRowThreads = 256;

// Bodies below kLargeBody points take eight lanes a row. From there on the lanes follow the mean row length, which
// only the device knows without a synchronisation: a grid has threads for four lanes per row, from kTwoLaneGrid on for
// two; threads of fewer lanes than that end at once (3 to 10 % of a call over short rows at 1M points), those of more pass
// over two rows (5 to 10 % over long ones at 154,000 to 315,000). Calls on lattices, microseconds,
// one lane always | eight always | now: 250,000 points with 4 bonds each, deformation 18 | 47 | 19, damage 14 | 40 | 15,
// with 28, 38 | 87 | 36 and 73 | 88 | 53; 1M points with 6, 61 | 200 | 63 and 52 | 163 | 52, with 118,
// 548 | 770 | 533 and 1210 | 838 | 651; 108,000 points with 229, 198 | 133 | 122 and 394 | 169 | 164; the force sum of
// 1M points with 6, eight always | now, 263 | 145.
// With packed records (calls over long rows) eight lanes serve up to 100,000 points, in the shape tensors up to 500,000:
// damage of 50,000 points with 109 bonds, four | eight lanes 47 | 41, of 82,000 with 230, 135 | 124, of 108,000 with 229,
// 156 | 152; shape tensors of 154,000 with 230, 158 | 145, of 250,000 with 239, 205 | 205, of 1M with 245, 665 | 723.
constexpr int64_t kLargeBody = 60000, kLargePackedBody = 100000, kLargePackedShapes = 500000;
constexpr int64_t kShortRowBody = 150000, kTwoLaneGrid = 500000;
__device__ __forceinline__ int row_lanes(int64_t n, const int64_t *row_ptr) {
  const int64_t bonds = __ldg(row_ptr + n) - __ldg(row_ptr);
  if (n < kShortRowBody)
    return bonds < 24 * n ? 2 : 4;
  return bonds < 20 * n ? 1 : (bonds < 64 * n ? 2 : 4);
}
// launch(LARGE, blocks): the sums' kernels come in both forms, LARGE from large_body points on.
template <typename F> static void launch_rows(int64_t n, int64_t large_body, F &&launch) {
  const bool large = n >= large_body;
  const int64_t lanes = !large ? 8 : (n < kTwoLaneGrid ? 4 : 2);
  const unsigned blocks = (unsigned)((n * lanes + kRowThreads - 1) / kRowThreads);
  if (large)
    launch(std::true_type{}, blocks);
  else
    launch(std::false_type{}, blocks);
}

// Calls pass(lanes, thread) for the calling thread's passes over the rows; whole warps make the same passes.
template <int LANES, typename F> __device__ __forceinline__ void row_passes(int64_t n, F &&pass) {
  const int64_t thread = (int64_t)blockIdx.x * kRowThreads + threadIdx.x, threads = (int64_t)gridDim.x * kRowThreads;
  for (int64_t t = thread; (t & ~int64_t(31)) < n * LANES; t += threads)
    pass(std::integral_constant<int, LANES>{}, t);
}
template <bool LARGE, typename F>
__device__ __forceinline__ void row_passes(int64_t n, const int64_t *row_ptr, F &&pass) {
  if (!LARGE) {
    pass(std::integral_constant<int, 8>{}, (int64_t)blockIdx.x * kRowThreads + threadIdx.x);
    return;
  }
  const int lanes = row_lanes(n, row_ptr);
  if (lanes == 1)
    row_passes<1>(n, pass);
  else if (lanes == 2)
    row_passes<2>(n, pass);
  else
    row_passes<4>(n, pass);
}

// The sum over a row's lanes, in every lane.
template <int LANES> __device__ __forceinline__ double row_sum(double v) {
#pragma unroll
  for (int o = LANES / 2; o > 0; o >>= 1)
    v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Thread t's row; a thread past the end takes an empty one, so that whole warps take part in the shuffles.
struct RowPoint {
  int64_t i, begin, end;
  int lane;
  bool valid;
};
template <int LANES> __device__ __forceinline__ RowPoint row_point(int64_t n, const int64_t *row_ptr, int64_t t) {
  const int64_t k = t / LANES;
  RowPoint r;
  r.valid = k < n;
  r.i = r.valid ? k : 0;
  r.begin = r.valid ? row_ptr[k] : 0, r.end = r.valid ? row_ptr[k + 1] : 0;
  r.lane = (int)t & (LANES - 1);
  return r;
}

// Calls bond(q, j) for the calling lane's bonds q of its row and their neighbours j.
template <int LANES, typename F> __device__ __forceinline__ void for_row(const RowPoint &r, const int32_t *col, F &&bond) {
  int64_t q = r.begin + r.lane;
  int32_t j = q < r.end ? __ldg(col + q) : 0;
#pragma unroll 2
  for (; q < r.end; q += LANES) {
    const int32_t next = q + LANES < r.end ? __ldg(col + q + LANES) : 0;
    bond(q, (int64_t)j);
    j = next;
  }
}

// Where the bond sums read the points: the caller's arrays, or 32-byte records packed into memory of the caller's
// first (the entry points with records), one load per vector.
struct PointsPlain {
  const double *pos, *vol;
  __device__ __forceinline__ double4 xv(int64_t j) const {
    return make_double4(__ldg(pos + 3 * j), __ldg(pos + 3 * j + 1), __ldg(pos + 3 * j + 2), __ldg(vol + j));
  }
};
// The displacement u (deformation) or the current position x + u (damage) of a point.
template <bool CURRENT> struct VectorsPlain {
  const double *pos, *disp;
  __device__ __forceinline__ double4 at(int64_t j) const {
    double v[3];
#pragma unroll
    for (int c = 0; c < 3; ++c)
      v[c] = CURRENT ? __dadd_rn(__ldg(pos + 3 * j + c), __ldg(disp + 3 * j + c)) : __ldg(disp + 3 * j + c);
    return make_double4(v[0], v[1], v[2], 0.0);
  }
};
// The records pay where rows are long and points are many. Calls at horizon 4.015 h, plain | packed: damage 36,000
// points 83 | 66 us, 108,000 187 | 156, 250,000 405 | 328; deformation 250,000 261 | 273, 1M 1056 | 1042; shape
// tensors 250,000 204 | 205, 1M 718 | 665; with the 250,000 points in no order, damage 2 times as fast, the other two
// 1.9 times. (Not in the force sum: its nine words of M a bond outweigh the four of the point.)
struct Packed {
  const double4 *rec;
  __device__ __forceinline__ double4 xv(int64_t j) const { return ldg256(rec + j); }
  __device__ __forceinline__ double4 at(int64_t j) const { return ldg256(rec + j); }
};

template <bool CURRENT>
__global__ void k_pack_points(const double *pos, const double *vol, const double *disp, int64_t n, double4 *xv,
                              double4 *vec) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n)
    return;
  st256(xv + i, PointsPlain{pos, vol}.xv(i));
  if (vec)
    st256(vec + i, VectorsPlain<CURRENT>{pos, disp}.at(i));
}

// PdCorrespondenceSkeleton::initialize (:149-170)
template <int LANES, typename Points>
__device__ __forceinline__ void shape_inverse_row(Points points, int64_t t, int64_t n, const int64_t *row_ptr, const int32_t *col,
                                                   double *kinv, unsigned *status) {
  const RowPoint r = row_point<LANES>(n, row_ptr, t);
  const int64_t i = r.i;
  const double4 x = points.xv(i);
  double k00 = 0, k01 = 0, k02 = 0, k11 = 0, k12 = 0, k22 = 0;
  for_row<LANES>(r, col, [&](int64_t, int64_t j) {
    const double4 p = points.xv(j);
    const double e0 = p.x - x.x, e1 = p.y - x.y, e2 = p.z - x.z, v = p.w, w0 = v * e0, w1 = v * e1;
    k00 += w0 * e0, k01 += w0 * e1, k02 += w0 * e2;
    k11 += w1 * e1, k12 += w1 * e2, k22 += v * e2 * e2;
  });
  k00 = row_sum<LANES>(k00), k01 = row_sum<LANES>(k01), k02 = row_sum<LANES>(k02);
  k11 = row_sum<LANES>(k11), k12 = row_sum<LANES>(k12), k22 = row_sum<LANES>(k22);
  if (!r.valid || r.lane != 0)
    return;
  const double K[9] = {k00, k01, k02, k01, k11, k12, k02, k12, k22};
  double Ki[9];
  if (!m_inv(K, Ki)) {
    atomicOr(status, STATUS_SINGULAR_K);
    for (int c = 0; c < 9; ++c)
      Ki[c] = 0.0;
  }
  for (int c = 0; c < 9; ++c)
    kinv[9 * i + c] = Ki[c];
}
template <bool LARGE, typename Points>
__global__ void __launch_bounds__(kRowThreads) k_csr_shape_inverse(Points points, int64_t n, const int64_t *row_ptr,
                                                                   const int32_t *col, double *kinv,
                                                                   unsigned *status) {
  row_passes<LARGE>(n, row_ptr, [&](auto lanes, int64_t t) {
    shape_inverse_row<decltype(lanes)::value>(points, t, n, row_ptr, col, kinv, status);
  });
}

// computeDeformationGradients (:172-197), in displacement-gradient form
// F = I + [sum_j V_j (u_j - u_i) (x) xi] K^-1.
template <int LANES, typename Points, typename Vectors>
__device__ __forceinline__ void deformation_row(Points points, Vectors disp, int64_t t, int64_t n, const int64_t *row_ptr,
                                                 const int32_t *col, const double *kinv, double *F) {
  const RowPoint r = row_point<LANES>(n, row_ptr, t);
  const int64_t i = r.i;
  const double4 x = points.xv(i), u = disp.at(i);
  double G[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  for_row<LANES>(r, col, [&](int64_t, int64_t j) {
    const double4 p = points.xv(j), uj = disp.at(j);
    const double e[3] = {p.x - x.x, p.y - x.y, p.z - x.z};
    const double d[3] = {p.w * (uj.x - u.x), p.w * (uj.y - u.y), p.w * (uj.z - u.z)};
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int b = 0; b < 3; ++b)
        G[3 * a + b] += d[a] * e[b];
  });
#pragma unroll
  for (int c = 0; c < 9; ++c)
    G[c] = row_sum<LANES>(G[c]);
  if (!r.valid)
    return;
  double K[9];
#pragma unroll
  for (int c = 0; c < 9; ++c)
    K[c] = kinv[9 * i + c];
#pragma unroll
  for (int a = 0; a < 3; ++a)  // the row's lanes write the rows of F in turn
    if (a % LANES == r.lane)
#pragma unroll
      for (int b = 0; b < 3; ++b)
        F[9 * i + 3 * a + b] =
            (a == b ? 1.0 : 0.0) + (G[3 * a] * K[b] + G[3 * a + 1] * K[3 + b] + G[3 * a + 2] * K[6 + b]);
}
template <bool LARGE, typename Points, typename Vectors>
__global__ void __launch_bounds__(kRowThreads, 4) k_csr_deformation(Points points, Vectors disp, int64_t n,
                                                                    const int64_t *row_ptr, const int32_t *col,
                                                                    const double *kinv, double *F) {
  row_passes<LARGE>(n, row_ptr, [&](auto lanes, int64_t t) {
    deformation_row<decltype(lanes)::value>(points, disp, t, n, row_ptr, col, kinv, F);
  });
}

// The force map M = J sigma F^-T K^-1 of every point as the bond sum gathers it: entries 0..7 as four
// arrays of pairs, then entry 8 (9 n doubles in all).
__global__ void k_csr_force_map(const double *sigma, const double *F, const double *kinv,
                                int64_t n, double *M, unsigned *status) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n)
    return;
  double s[9], f[9], k[9], m[9];
  for (int c = 0; c < 9; ++c)
    s[c] = sigma[9 * i + c], f[c] = F[9 * i + c], k[c] = kinv[9 * i + c];
  if (!force_map(s, f, k, m)) {
    atomicOr(status, STATUS_SINGULAR_F);
    for (int c = 0; c < 9; ++c)
      m[c] = 0.0;
  }
  double2 *pairs = reinterpret_cast<double2 *>(M);
#pragma unroll
  for (int c = 0; c < 4; ++c)
    pairs[c * n + i] = make_double2(m[2 * c], m[2 * c + 1]);
  M[8 * n + i] = m[8];
}

// computeForceDensity (:199-230): f_i = sum (1 - clamp(d)) (M_i + M_j) xi V_j
template <int LANES>
__device__ __forceinline__ void force_row(PointsPlain points, int64_t t, int64_t n, const int64_t *row_ptr, const int32_t *col,
                                           const double *M, const double *bond_damage, double *force) {
  const double2 *pairs = reinterpret_cast<const double2 *>(M);
  const RowPoint r = row_point<LANES>(n, row_ptr, t);
  const int64_t i = r.i;
  const double4 x = points.xv(i);
  const double2 ai = __ldg(pairs + i), bi = __ldg(pairs + n + i), ci = __ldg(pairs + 2 * n + i),
                di = __ldg(pairs + 3 * n + i);
  const double m8i = __ldg(M + 8 * n + i);
  double f0 = 0, f1 = 0, f2 = 0;
  for_row<LANES>(r, col, [&](int64_t q, int64_t j) {
    const double4 p = points.xv(j);
    const double e0 = p.x - x.x, e1 = p.y - x.y, e2 = p.z - x.z;
    double dmg = bond_damage ? __ldg(bond_damage + q) : 0.0;
    dmg = dmg < 0.0 ? 0.0 : (dmg > 1.0 ? 1.0 : dmg);
    const double w = (1.0 - dmg) * p.w;
    const double2 a = __ldg(pairs + j), b = __ldg(pairs + n + j), c = __ldg(pairs + 2 * n + j),
                  d = __ldg(pairs + 3 * n + j);
    const double m8 = __ldg(M + 8 * n + j);
    f0 += w * ((ai.x + a.x) * e0 + (ai.y + a.y) * e1 + (bi.x + b.x) * e2);
    f1 += w * ((bi.y + b.y) * e0 + (ci.x + c.x) * e1 + (ci.y + c.y) * e2);
    f2 += w * ((di.x + d.x) * e0 + (di.y + d.y) * e1 + (m8i + m8) * e2);
  });
  f0 = row_sum<LANES>(f0), f1 = row_sum<LANES>(f1), f2 = row_sum<LANES>(f2);
  if (r.valid && r.lane == 0)
    force[3 * i] = f0, force[3 * i + 1] = f1, force[3 * i + 2] = f2;
}
template <bool LARGE>
__global__ void __launch_bounds__(kRowThreads, 3) k_csr_force(PointsPlain points, int64_t n, const int64_t *row_ptr,
                                                              const int32_t *col, const double *M,
                                                              const double *bond_damage, double *force) {
  row_passes<LARGE>(n, row_ptr, [&](auto lanes, int64_t t) {
    force_row<decltype(lanes)::value>(points, t, n, row_ptr, col, M, bond_damage, force);
  });
}

// ------------------------------------------------------------------ pointwise kernels
// The point-major tensors (nine doubles a point) of a block's 128 points are one run of memory: it is
// copied to shared memory 16 bytes at a time, each thread reads its nine words there (72 bytes apart: no bank
// conflict), and results go back the same way. Read and written by their threads directly, every load
// touched 18 lines and every store sent eight bytes of each sector on its own. Four blocks per SM (128
// registers; their tiles take 180 and 216 KB). Calls at 500,000 points on a B200, before | now:
// material_update on a plastic load path 333 | 213 us (271 with the four blocks alone), corotational_update 172 |
// 103 us; they move 464 and 324 MB, 72 and 50 us at the measured copy rate. What is left in the first is the
// return map's serial chain, in both about 25 us of status word, launch and synchronisation.
constexpr int kPointThreads = 128;
constexpr int kTensorTile = 9 * kPointThreads;  // doubles
using TensorTile = double[kTensorTile];

__device__ __forceinline__ bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// The block's tensors (9 count doubles from point `first` on) into a tile: asynchronous copies, complete at
// tiles_ready(). In a block that is not full each thread copies its own (and tile_out the same): a call on a few points is
// shorter so, corotational_update on one point 63 to 55 us, on two 57 to 54.
__device__ __forceinline__ void tile_in(const double *src, TensorTile &tile, int64_t first, int count) {
  const double *from = src + 9 * first;
  if (count < kPointThreads) {
    if ((int)threadIdx.x < count)
      for (int c = 0; c < 9; ++c)
        tile[9 * threadIdx.x + c] = from[9 * threadIdx.x + c];
  } else if (aligned16(from)) {
    for (int k = 2 * threadIdx.x; k < kTensorTile; k += 2 * kPointThreads)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(umma::smem_u32(tile + k)), "l"(from + k) : "memory");
  } else {
    for (int k = threadIdx.x; k < kTensorTile; k += kPointThreads)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(umma::smem_u32(tile + k)), "l"(from + k) : "memory");
  }
}
__device__ __forceinline__ void tiles_ready() {
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
}
// A tile back to the block's tensors; after a barrier that follows the threads' writes to it.
__device__ __forceinline__ void tile_out(double *dst, const TensorTile &tile, int64_t first, int count) {
  double *to = dst + 9 * first;
  if (count < kPointThreads) {
    if ((int)threadIdx.x < count)
      for (int c = 0; c < 9; ++c)
        to[9 * threadIdx.x + c] = tile[9 * threadIdx.x + c];
  } else if (aligned16(to)) {
    for (int k = 2 * threadIdx.x; k < kTensorTile; k += 2 * kPointThreads)
      *reinterpret_cast<double2 *>(to + k) = *reinterpret_cast<const double2 *>(tile + k);
  } else {
    for (int k = threadIdx.x; k < kTensorTile; k += kPointThreads)
      to[k] = tile[k];
  }
}
__device__ __forceinline__ void get9(const TensorTile &tile, double (&v)[9]) {
#pragma unroll
  for (int c = 0; c < 9; ++c)
    v[c] = tile[9 * threadIdx.x + c];
}
__device__ __forceinline__ void put9(TensorTile &tile, const double (&v)[9]) {
#pragma unroll
  for (int c = 0; c < 9; ++c)
    tile[9 * threadIdx.x + c] = v[c];
}

constexpr int kCorotationalTiles = 5;
__global__ void __launch_bounds__(kPointThreads, 4)
    k_corotational(int64_t n, const double *fN, const double *fNP1, const double *vN, const double *rN, double dt,
                   double *dbar, double *spin, double *rNew, double *vNew, double *strain, unsigned *status) {
  extern __shared__ __align__(16) double s_points[];
  TensorTile *tile = reinterpret_cast<TensorTile *>(s_points);
  const int64_t first = (int64_t)blockIdx.x * kPointThreads;
  const int count = (int)min((int64_t)kPointThreads, n - first);
  tile_in(fN, tile[0], first, count), tile_in(fNP1, tile[1], first, count);
  tile_in(vN, tile[2], first, count), tile_in(rN, tile[3], first, count);
  tiles_ready();
  if ((int)threadIdx.x < count) {
    double a[9], b[9], v[9], r[9];
    get9(tile[0], a), get9(tile[1], b), get9(tile[2], v), get9(tile[3], r);
    Corotational co;
    if (!corotational_update(a, b, v, r, dt, co))
      atomicOr(status, STATUS_SINGULAR_KINEMATICS);
    double e6[6], e[9];
    green_lagrange6(b, e6);
    voigt_to_full(e6, e);
    put9(tile[0], co.dbar), put9(tile[1], co.spin), put9(tile[2], co.v), put9(tile[3], co.r), put9(tile[4], e);
  }
  __syncthreads();
  tile_out(dbar, tile[0], first, count), tile_out(spin, tile[1], first, count);
  tile_out(vNew, tile[2], first, count), tile_out(rNew, tile[3], first, count);
  tile_out(strain, tile[4], first, count);
}

// VumatPdCorrespondenceMaterial::update for one point (:155-170,195-210).
constexpr int kMaterialTiles = 6;
__global__ void __launch_bounds__(kPointThreads, 4)
    k_material_update(int64_t n, JcParams jc, int nstatev, double dt, const double *Fnew, double *Fold,
                      double *stretch, double *rotation, double *strain, double *sig, double *state, double *temp,
                      double *eI, double *eP, double *spatial, unsigned *status) {
  extern __shared__ __align__(16) double s_points[];
  TensorTile *tile = reinterpret_cast<TensorTile *>(s_points);  // F, F_n, V, R, stress, strain
  const int64_t first = (int64_t)blockIdx.x * kPointThreads, i = first + threadIdx.x;
  const int count = (int)min((int64_t)kPointThreads, n - first);
  tile_in(Fnew, tile[0], first, count), tile_in(Fold, tile[1], first, count);
  tile_in(stretch, tile[2], first, count), tile_in(rotation, tile[3], first, count);
  tile_in(sig, tile[4], first, count);
  JcPoint pt;
  if ((int)threadIdx.x < count) {
    for (int c = 0; c < 6; ++c)
      pt.state[c] = state[(size_t)nstatev * i + c];
    pt.eInternal = eI[i];
    pt.eInelastic = eP[i];
  }
  tiles_ready();
  if ((int)threadIdx.x < count) {
    double d[9];
    bool updated;
    {
      double F[9], Fn[9], Vn[9], Rn[9];
      get9(tile[0], F), get9(tile[1], Fn), get9(tile[2], Vn), get9(tile[3], Rn);
      Corotational co;
      updated = corotational_update(Fn, F, Vn, Rn, dt, co);
      if (updated) {  // V and R go to their tiles now, out of the registers
        put9(tile[2], co.v), put9(tile[3], co.r);
#pragma unroll
        for (int c = 0; c < 9; ++c)
          d[c] = co.dbar[c];
      } else {  // the point keeps every field
        atomicOr(status, STATUS_SINGULAR_KINEMATICS);
        put9(tile[0], Fn);
        for (int c = 0; c < 9; ++c)
          tile[1][9 * threadIdx.x + c] = spatial[9 * i + c], tile[5][9 * threadIdx.x + c] = strain[9 * i + c];
      }
    }
    if (updated) {
      double s9[9];
      get9(tile[4], s9);
      full_to_voigt(s9, pt.stress);
      const double inc[6] = {d[0] * dt, d[4] * dt, d[8] * dt, 0.5 * (d[5] + d[7]) * dt,
                             0.5 * (d[2] + d[6]) * dt, 0.5 * (d[1] + d[3]) * dt};
      jc_update(jc, dt, inc, pt);
      double F[9], R[9], full[9], sp[9], e6[6], e[9];
      get9(tile[3], R);
      voigt_to_full(pt.stress, full);
      rotate_to_spatial(full, R, sp);
      put9(tile[4], full), put9(tile[1], sp);
      get9(tile[0], F);
      green_lagrange6(F, e6);
      voigt_to_full(e6, e);
      put9(tile[5], e);
      for (int c = 0; c < 6; ++c)
        state[(size_t)nstatev * i + c] = pt.state[c];
      temp[i] = pt.state[2];
      eI[i] = pt.eInternal;
      eP[i] = pt.eInelastic;
    }
  }
  __syncthreads();
  tile_out(Fold, tile[0], first, count), tile_out(stretch, tile[2], first, count);
  tile_out(rotation, tile[3], first, count), tile_out(strain, tile[5], first, count);
  tile_out(sig, tile[4], first, count), tile_out(spatial, tile[1], first, count);
}

// The VUMAT's return map alone for one point (JohnsonCook.f90:74-136): the elastic trial from
// the old stress and state, then the bisection, certified (jc_return_map) or literal
// (jc_bisection). A point on its initialising call (state[0] == 0) reports 0 iterations.
template <bool CERTIFIED>
__global__ void __launch_bounds__(kPointThreads, 8) k_jc_return_map(int64_t n, JcParams jc, double dt, const double *inc, const double *sig,
                                const double *state, int nstatev, double *epInc, double *yield, int32_t *iters) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n)
    return;
  JcPoint pt;
  double d[6];
  for (int c = 0; c < 6; ++c)
    d[c] = inc[6 * i + c], pt.stress[c] = sig[6 * i + c], pt.state[c] = state[(size_t)nstatev * i + c];
  pt.eInternal = pt.eInelastic = 0.0;
  JcTrial t;
  double e = 0.0, y = 0.0;
  int it = 0;
  if (jc_trial(jc, d, pt, t))
    it = CERTIFIED ? jc_return_map(jc, dt, t, pt.state[4], e, y) : jc_bisection(jc, dt, t, pt.state[4], e, y);
  epInc[i] = e, yield[i] = y, iters[i] = it;
}

// PdSimpleDamage::update critical_stretch (:51-82) with the reference's rounding, and the
// damage index (:23-36). A bond whose squared lengths lie clear of both thresholds (by 1e-9 of them,
// against roundings of 1e-15) is decided from those; the others, and lengths whose squares may not be
// normal numbers, take the reference's square roots and division. In compression the formula's stretch carries a
// rounding of 1e-16 of the initial length, which may be any part of the current one: where the threshold leaves less
// than kLeastLeft of a bond, every bond shorter than twice that takes the formula.
struct StretchTest {
  double initiation, failure, tension2;  // thresholds on the stretch, and on (1 + it)^2
  double surely_broken2, surely_whole2;  // current over initial length squared, in compression: below, above
  int use_compression;
};
constexpr double kLeastLeft = 0.01;
static StretchTest stretch_test(double initiation, double failure) {
  StretchTest t{initiation, failure, (1.0 + initiation) * (1.0 + initiation), -1.0, 0.0,
                failure > 0.0 && std::isfinite(failure)};
  const double left = 1.0 - failure;
  if (left >= kLeastLeft)
    t.surely_broken2 = left * left * (1.0 - 1.0e-9), t.surely_whole2 = left * left * (1.0 + 1.0e-9);
  else if (left > 0.0)
    t.surely_whole2 = 4.0 * kLeastLeft * kLeastLeft;
  return t;
}
__device__ __forceinline__ bool stretch_breaks(const StretchTest &t, const double (&e)[3], const double (&y)[3]) {
  const double xx =
      __dadd_rn(__dadd_rn(__dmul_rn(e[0], e[0]), __dmul_rn(e[1], e[1])), __dmul_rn(e[2], e[2]));
  const double yy =
      __dadd_rn(__dadd_rn(__dmul_rn(y[0], y[0]), __dmul_rn(y[1], y[1])), __dmul_rn(y[2], y[2]));
  if (xx > 1.0e-200 && xx < 1.0e200 && yy > 1.0e-200 && yy < 1.0e200) {
    const double tt = t.tension2 * xx;
    if (yy > tt * (1.0 + 1.0e-9))
      return true;
    if (yy < tt * (1.0 - 1.0e-9)) {
      if (!t.use_compression)
        return false;
      if (yy < t.surely_broken2 * xx)
        return true;
      if (yy > t.surely_whole2 * xx)
        return false;
    }
  }
  const double initial = __dsqrt_rn(xx);
  const double stretch = __ddiv_rn(__dsub_rn(__dsqrt_rn(yy), initial), initial);
  return stretch > t.initiation || (t.use_compression && stretch < -t.failure);
}

template <int LANES, typename Points, typename Vectors>
__device__ __forceinline__ void damage_row(Points points, Vectors current, int64_t t, int64_t n, const int64_t *row_ptr,
                                            const int32_t *col, const StretchTest &test, double *bond_damage,
                                            double *damage_index) {
  const RowPoint r = row_point<LANES>(n, row_ptr, t);
  const int64_t i = r.i;
  const double4 x = points.xv(i), yi = current.at(i);
  double damaged = 0.0, total = 0.0;
  for_row<LANES>(r, col, [&](int64_t q, int64_t j) {
    const double4 p = points.xv(j), yj = current.at(j);
    const double e[3] = {__dsub_rn(p.x, x.x), __dsub_rn(p.y, x.y), __dsub_rn(p.z, x.z)};
    const double y[3] = {__dsub_rn(yj.x, yi.x), __dsub_rn(yj.y, yi.y), __dsub_rn(yj.z, yi.z)};
    double d = bond_damage[q];
    if (stretch_breaks(test, e, y) && d != 1.0)
      bond_damage[q] = d = 1.0;
    damaged += d * p.w;
    total += p.w;
  });
  damaged = row_sum<LANES>(damaged), total = row_sum<LANES>(total);
  if (damage_index && r.valid && r.lane == 0)
    damage_index[i] = total > 0.0 ? damaged / total : 0.0;
}
template <bool LARGE, typename Points, typename Vectors>
__global__ void __launch_bounds__(kRowThreads, 4) k_csr_damage(Points points, Vectors current, int64_t n,
                                                               const int64_t *row_ptr, const int32_t *col,
                                                               StretchTest test, double *bond_damage,
                                                               double *damage_index) {
  row_passes<LARGE>(n, row_ptr, [&](auto lanes, int64_t t) {
    damage_row<decltype(lanes)::value>(points, current, t, n, row_ptr, col, test, bond_damage, damage_index);
  });
}

// Johnson-Cook on one column-major block (the plugin ABI).
__global__ void k_vumat_block(int nb, JcParams jc, double dt, int nstatev, const double *strainInc,
                              const double *stressOld, const double *stateOld,
                              const double *enerInternOld, const double *enerInelasOld,
                              double *stressNew, double *stateNew, double *tempNew,
                              double *enerInternNew, double *enerInelasNew) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nb)
    return;
  JcPoint pt;
  double inc[6];
  for (int c = 0; c < 6; ++c) {
    pt.stress[c] = stressOld[k + nb * c];
    inc[c] = strainInc[k + nb * c];
    pt.state[c] = stateOld[k + nb * c];
  }
  pt.eInternal = enerInternOld[k];
  pt.eInelastic = enerInelasOld[k];
  jc_update(jc, dt, inc, pt);
  for (int c = 0; c < 6; ++c) {
    stressNew[k + nb * c] = pt.stress[c];
    stateNew[k + nb * c] = pt.state[c];
  }
  for (int c = 6; c < nstatev; ++c)
    stateNew[k + nb * c] = stateOld[k + nb * c];
  tempNew[k] = pt.state[2];
  enerInternNew[k] = pt.eInternal;
  enerInelasNew[k] = pt.eInelastic;
}

static int check_status(unsigned *dstatus, cudaStream_t s) {
  unsigned st = 0;
  VPD_CUDA(cudaMemcpyAsync(&st, dstatus, sizeof st, cudaMemcpyDeviceToHost, s));
  VPD_CUDA(cudaStreamSynchronize(s));
  if (st & STATUS_SINGULAR_K)
    return set_error(VPD_ERR_SINGULAR, "Singular tensor in PD shape tensor.");
  if (st & STATUS_SINGULAR_F)
    return set_error(VPD_ERR_SINGULAR, "Invalid deformation gradient determinant.");
  if (st & STATUS_SINGULAR_KINEMATICS)
    return set_error(VPD_ERR_SINGULAR, "Corotational update encountered a singular tensor.");
  return VPD_OK;
}

// A device status word owned by the calling thread.
static unsigned *thread_status() {
  thread_local unsigned *word = nullptr;
  if (!word && cudaMalloc(&word, sizeof(unsigned)) != cudaSuccess)
    word = nullptr;
  return word;
}

static unsigned blocks(int64_t n) { return (unsigned)std::max<int64_t>(1, (n + 127) / 128); }

int launch_csr_force(const double *positions, const double *volumes, int64_t n, const int64_t *row_ptr,
                     const int32_t *col, const double *kinv, const double *defgrad, const double *cauchy_stress,
                     const double *bond_damage, double *force, double *M, unsigned *status, cudaStream_t s) {
  k_csr_force_map<<<blocks(n), 128, 0, s>>>(cauchy_stress, defgrad, kinv, n, M, status);
  launch_rows(n, kLargeBody, [&](auto large, unsigned blocks) {
    k_csr_force<decltype(large)::value><<<blocks, kRowThreads, 0, s>>>(PointsPlain{positions, volumes}, n,
        row_ptr, col, M, bond_damage, force);
  });
  VPD_CUDA(cudaGetLastError());
  return VPD_OK;
}

// The bond sums of the entry points, with or without room for packed records.
static int check_records(const double *records, const char *entry) {
  if (!records || (reinterpret_cast<uintptr_t>(records) & 31))
    return set_error(VPD_ERR_INVALID, std::string(entry) + ": needs records on a 32-byte boundary");
  return VPD_OK;
}

static int shape_tensor_inverse(const double *positions, const double *volumes, int64_t n, const int64_t *row_ptr,
                                const int32_t *col, double *kinv, double4 *rec, cudaStream_t s) {
  unsigned *st = thread_status();
  if (!st)
    return set_error(VPD_ERR_CUDA, "status word allocation failed");
  if (n <= 0)
    return VPD_OK;
  VPD_CUDA(cudaMemsetAsync(st, 0, sizeof(unsigned), s));
  if (rec) {
    k_pack_points<false><<<blocks(n), 128, 0, s>>>(positions, volumes, nullptr, n, rec, nullptr);
    launch_rows(n, kLargePackedShapes, [&](auto large, unsigned blocks) {
      k_csr_shape_inverse<decltype(large)::value><<<blocks, kRowThreads, 0, s>>>(Packed{rec}, n, row_ptr,
          col, kinv, st);
    });
  } else {
    launch_rows(n, kLargeBody, [&](auto large, unsigned blocks) {
      k_csr_shape_inverse<decltype(large)::value><<<blocks, kRowThreads, 0, s>>>(PointsPlain{positions,
          volumes}, n, row_ptr, col, kinv, st);
    });
  }
  VPD_CUDA(cudaGetLastError());
  return check_status(st, s);
}

static int deformation_gradients(const double *positions, const double *displacement, const double *volumes, int64_t n,
                                 const int64_t *row_ptr, const int32_t *col, const double *kinv, double *defgrad,
                                 double4 *rec, cudaStream_t s) {
  if (n <= 0)
    return VPD_OK;
  if (rec) {
    k_pack_points<false><<<blocks(n), 128, 0, s>>>(positions, volumes, displacement, n, rec, rec + n);
    launch_rows(n, kLargePackedBody, [&](auto large, unsigned blocks) {
      k_csr_deformation<decltype(large)::value><<<blocks, kRowThreads, 0, s>>>(Packed{rec}, Packed{rec + n},
          n, row_ptr, col, kinv, defgrad);
    });
  } else {
    launch_rows(n, kLargeBody, [&](auto large, unsigned blocks) {
      k_csr_deformation<decltype(large)::value><<<blocks, kRowThreads, 0, s>>>(PointsPlain{positions,
          volumes}, VectorsPlain<false>{positions, displacement}, n, row_ptr, col, kinv, defgrad);
    });
  }
  VPD_CUDA(cudaGetLastError());
  return VPD_OK;
}

static int damage_update(const double *positions, const double *displacement, const double *volumes, int64_t n,
                         const int64_t *row_ptr, const int32_t *col, double initiation, double failure,
                         double *bond_damage, double *damage_index, double4 *rec, cudaStream_t s) {
  if (!(initiation > 0.0))
    return set_error(VPD_ERR_INVALID, "critical_stretch requires initiation > 0.");
  if (n <= 0)
    return VPD_OK;
  const StretchTest test = stretch_test(initiation, failure);
  if (rec) {
    k_pack_points<true><<<blocks(n), 128, 0, s>>>(positions, volumes, displacement, n, rec, rec + n);
    launch_rows(n, kLargePackedBody, [&](auto large, unsigned blocks) {
      k_csr_damage<decltype(large)::value><<<blocks, kRowThreads, 0, s>>>(Packed{rec}, Packed{rec + n}, n,
          row_ptr, col, test, bond_damage, damage_index);
    });
  } else {
    launch_rows(n, kLargeBody, [&](auto large, unsigned blocks) {
      k_csr_damage<decltype(large)::value><<<blocks, kRowThreads, 0, s>>>(PointsPlain{positions, volumes},
          VectorsPlain<true>{positions, displacement}, n, row_ptr, col, test, bond_damage, damage_index);
    });
  }
  VPD_CUDA(cudaGetLastError());
  return VPD_OK;
}

}  // namespace vpd

using namespace vpd;

extern "C" {

int vpd_build_neighbor_list(const double *positions, int64_t n, double horizon, int64_t *row_ptr,
                            int32_t *col, int64_t *total, void *stream) {
  if (!positions || !row_ptr || !total || n <= 0)
    return set_error(VPD_ERR_INVALID, "vpd_build_neighbor_list: invalid argument");
  cudaStream_t s = (cudaStream_t)stream;
  Workspace ws(s);
  double4 *xv = nullptr;
  int rc = ws.alloc(&xv, n);
  if (rc)
    return rc;
  k_pack_positions<<<blocks(n), 128, 0, s>>>(positions, n, xv);
  NeighborScratch scr;
  NeighborGrid grid;
  rc = neighbor_scratch_alloc(scr, n, s);
  if (rc == VPD_OK)
    rc = neighbor_count(xv, n, horizon, row_ptr, grid, scr, s);
  if (rc == VPD_OK) {
    cudaError_t e = cudaMemcpyAsync(total, row_ptr + n, sizeof(int64_t), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess)
      e = cudaStreamSynchronize(s);
    if (e != cudaSuccess)
      rc = cuda_error(e, "neighbour total");
  }
  if (rc == VPD_OK && col)
    rc = neighbor_fill(xv, n, row_ptr, col, grid, scr, s);
  neighbor_scratch_free(scr);
  if (ws.bytes >= kWorkspaceSmall / 2) {  // (the search's own scratch is about as large as the packed positions)
    ws.release();
    const cudaError_t e = cudaStreamSynchronize(s);
    if (rc == VPD_OK && e != cudaSuccess)
      rc = cuda_error(e, "neighbour list");
  }
  return rc;
}

int vpd_shape_tensor_inverse(const double *positions, const double *volumes, int64_t n,
                             const int64_t *row_ptr, const int32_t *col, double *kinv, void *stream) {
  return shape_tensor_inverse(positions, volumes, n, row_ptr, col, kinv, nullptr, (cudaStream_t)stream);
}
int vpd_shape_tensor_inverse_packed(const double *positions, const double *volumes, int64_t n, const int64_t *row_ptr,
                                    const int32_t *col, double *kinv, double *records, void *stream) {
  const int rc = check_records(records, "vpd_shape_tensor_inverse_packed");
  return rc ? rc
            : shape_tensor_inverse(positions, volumes, n, row_ptr, col, kinv, reinterpret_cast<double4 *>(records),
                                   (cudaStream_t)stream);
}

int vpd_deformation_gradients(const double *positions, const double *displacement, const double *volumes,
                              int64_t n, const int64_t *row_ptr, const int32_t *col, const double *kinv,
                              double *defgrad, void *stream) {
  return deformation_gradients(positions, displacement, volumes, n, row_ptr, col, kinv, defgrad, nullptr,
                               (cudaStream_t)stream);
}
int vpd_deformation_gradients_packed(const double *positions, const double *displacement, const double *volumes,
                                     int64_t n, const int64_t *row_ptr, const int32_t *col, const double *kinv,
                                     double *defgrad, double *records, void *stream) {
  const int rc = check_records(records, "vpd_deformation_gradients_packed");
  return rc ? rc
            : deformation_gradients(positions, displacement, volumes, n, row_ptr, col, kinv, defgrad,
                                    reinterpret_cast<double4 *>(records), (cudaStream_t)stream);
}

int vpd_force_density(const double *positions, const double *volumes, int64_t n, const int64_t *row_ptr,
                      const int32_t *col, const double *kinv, const double *defgrad,
                      const double *cauchy_stress, const double *bond_damage, double *force,
                      void *stream) {
  cudaStream_t s = (cudaStream_t)stream;
  unsigned *st = thread_status();
  if (!st)
    return set_error(VPD_ERR_CUDA, "status word allocation failed");
  if (n <= 0)
    return VPD_OK;
  Workspace ws(s);
  double *M = nullptr;
  int rc = ws.alloc(&M, 9 * n);
  if (rc)
    return rc;
  VPD_CUDA(cudaMemsetAsync(st, 0, sizeof(unsigned), s));
  if ((rc = launch_csr_force(positions, volumes, n, row_ptr, col, kinv, defgrad, cauchy_stress, bond_damage, force, M,
                             st, s)))
    return rc;
  ws.finish();
  return check_status(st, s);
}

int vpd_corotational_update(int64_t n, const double *defgrad_old, const double *defgrad_new,
                            const double *stretch_old, const double *rotation_old, double dt,
                            double *rate_of_deformation, double *relative_spin, double *rotation_new,
                            double *stretch_new, double *strain_new, void *stream) {
  if (!(dt > 0.0))
    return set_error(VPD_ERR_INVALID, "Corotational update requires dt > 0.");
  cudaStream_t s = (cudaStream_t)stream;
  unsigned *st = thread_status();
  if (!st)
    return set_error(VPD_ERR_CUDA, "status word allocation failed");
  VPD_CUDA(cudaMemsetAsync(st, 0, sizeof(unsigned), s));
  if (n <= 0)
    return check_status(st, s);
  VPD_CUDA(cudaFuncSetAttribute(k_corotational, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)(kCorotationalTiles * sizeof(TensorTile))));
  k_corotational<<<blocks(n), kPointThreads, kCorotationalTiles * sizeof(TensorTile), s>>>(n, defgrad_old, defgrad_new, stretch_old, rotation_old, dt,
                                           rate_of_deformation, relative_spin, rotation_new, stretch_new,
                                           strain_new, st);
  VPD_CUDA(cudaGetLastError());
  return check_status(st, s);
}

int vpd_material_update(int64_t n, const double *props, int32_t nstatev, double dt, const double *defgrad_new,
                        double *defgrad_old, double *stretch, double *rotation, double *strain,
                        double *stress_corotational, double *state, double *temperature,
                        double *energy_internal, double *energy_inelastic, double *stress_spatial,
                        void *stream) {
  if (!props || nstatev < 6 || !(dt > 0.0))
    return set_error(VPD_ERR_INVALID, "VUMAT-PD material update requires props, nstatev >= 6 and dt > 0.");
  cudaStream_t s = (cudaStream_t)stream;
  unsigned *st = thread_status();
  if (!st)
    return set_error(VPD_ERR_CUDA, "status word allocation failed");
  VPD_CUDA(cudaMemsetAsync(st, 0, sizeof(unsigned), s));
  if (n <= 0)
    return check_status(st, s);
  VPD_CUDA(cudaFuncSetAttribute(k_material_update, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)(kMaterialTiles * sizeof(TensorTile))));
  k_material_update<<<blocks(n), kPointThreads, kMaterialTiles * sizeof(TensorTile), s>>>(n, make_jc_params(props), nstatev, dt, defgrad_new, defgrad_old,
                                              stretch, rotation, strain, stress_corotational, state,
                                              temperature, energy_internal, energy_inelastic, stress_spatial, st);
  VPD_CUDA(cudaGetLastError());
  return check_status(st, s);
}

int vpd_jc_return_map(int64_t n, const double *props, double dt, const double *strain_inc, const double *stress,
                      const double *state, int32_t nstatev, int32_t method, double *ep_inc, double *yield,
                      int32_t *iterations, void *stream) {
  if (!props || nstatev < 6 || !(dt > 0.0) || n < 0 || (method != 0 && method != 1))
    return set_error(VPD_ERR_INVALID, "JC return map requires props, nstatev >= 6, dt > 0, n >= 0 and method 0 or 1.");
  if (n == 0)
    return VPD_OK;
  cudaStream_t s = (cudaStream_t)stream;
  const JcParams jc = make_jc_params(props);
  if (method == 0)
    k_jc_return_map<true><<<blocks(n), 128, 0, s>>>(n, jc, dt, strain_inc, stress, state, nstatev, ep_inc, yield,
                                                   iterations);
  else
    k_jc_return_map<false><<<blocks(n), 128, 0, s>>>(n, jc, dt, strain_inc, stress, state, nstatev, ep_inc, yield,
                                                    iterations);
  VPD_CUDA(cudaGetLastError());
  return VPD_OK;
}

int vpd_damage_update(const double *positions, const double *displacement, const double *volumes, int64_t n,
                      const int64_t *row_ptr, const int32_t *col, double initiation, double failure,
                      double *bond_damage, double *damage_index, void *stream) {
  return damage_update(positions, displacement, volumes, n, row_ptr, col, initiation, failure, bond_damage,
                       damage_index, nullptr, (cudaStream_t)stream);
}
int vpd_damage_update_packed(const double *positions, const double *displacement, const double *volumes, int64_t n,
                             const int64_t *row_ptr, const int32_t *col, double initiation, double failure,
                             double *bond_damage, double *damage_index, double *records, void *stream) {
  const int rc = check_records(records, "vpd_damage_update_packed");
  return rc ? rc
            : damage_update(positions, displacement, volumes, n, row_ptr, col, initiation, failure, bond_damage,
                            damage_index, reinterpret_cast<double4 *>(records), (cudaStream_t)stream);
}

void vumat_adapter_call(int *nblock, int *ndir, int *nshr, int *nstatev, int *nfieldv, int *nprops,
                        int *lanneal, double *stepTime, double *totalTime, double *dt, char *cmname,
                        double *coordMp, double *charLength, double *props, double *density,
                        double *strainInc, double *relSpinInc, double *tempOld, double *stretchOld,
                        double *defgradOld, double *fieldOld, double *stressOld, double *stateOld,
                        double *enerInternOld, double *enerInelasOld, double *tempNew, double *stretchNew,
                        double *defgradNew, double *fieldNew, double *stressNew, double *stateNew,
                        double *enerInternNew, double *enerInelasNew) {
  (void)lanneal, (void)stepTime, (void)totalTime, (void)cmname, (void)coordMp, (void)charLength;
  (void)density, (void)relSpinInc, (void)tempOld;
  // The Fortran routine stops the process on these (JohnsonCook.f90:52-53); so does this entry.
  if (*ndir != 3 || *nshr != 3) {
    fprintf(stderr, "JohnsonCook VUMAT requires ndir=3,nshr=3\n");
    exit(1);
  }
  if (*nprops < 14 || *nstatev < 6) {
    fprintf(stderr, "JohnsonCook VUMAT requires 14 props and 6 states\n");
    exit(1);
  }
  const int nb = *nblock, nsv = *nstatev;
  // copy-through outputs (JohnsonCook.f90:84-90)
  std::memcpy(stretchNew, stretchOld, sizeof(double) * 6 * nb);
  std::memcpy(defgradNew, defgradOld, sizeof(double) * 9 * nb);
  if (*nfieldv > 0)
    std::memcpy(fieldNew, fieldOld, sizeof(double) * (size_t)(*nfieldv) * nb);
  // per-thread device block (the reference keeps one adapter per OpenMP thread)
  struct Block {
    cudaStream_t s = nullptr;
    double *buf = nullptr;
    size_t cap = 0;
  };
  thread_local Block blk;
  const size_t per = (size_t)(6 + 6 + nsv + 1 + 1 + 6 + nsv + 1 + 1 + 1);
  const size_t need = per * (size_t)nb;
  auto fail = [](cudaError_t e) {
    fprintf(stderr, "vumat_adapter_call: CUDA error %s\n", cudaGetErrorString(e));
    exit(1);
  };
  cudaError_t e = cudaSuccess;
  if (!blk.s && (e = cudaStreamCreateWithFlags(&blk.s, cudaStreamNonBlocking)) != cudaSuccess)
    fail(e);
  if (blk.cap < need) {
    cudaFree(blk.buf);
    if ((e = cudaMalloc(&blk.buf, need * sizeof(double))) != cudaSuccess)
      fail(e);
    blk.cap = need;
  }
  double *d_inc = blk.buf, *d_sold = d_inc + 6 * nb, *d_stold = d_sold + 6 * nb;
  double *d_eio = d_stold + (size_t)nsv * nb, *d_epo = d_eio + nb, *d_snew = d_epo + nb;
  double *d_stnew = d_snew + 6 * nb, *d_tnew = d_stnew + (size_t)nsv * nb, *d_ein = d_tnew + nb;
  double *d_epn = d_ein + nb;
  cudaStream_t s = blk.s;
  cudaMemcpyAsync(d_inc, strainInc, sizeof(double) * 6 * nb, cudaMemcpyHostToDevice, s);
  cudaMemcpyAsync(d_sold, stressOld, sizeof(double) * 6 * nb, cudaMemcpyHostToDevice, s);
  cudaMemcpyAsync(d_stold, stateOld, sizeof(double) * nsv * nb, cudaMemcpyHostToDevice, s);
  cudaMemcpyAsync(d_eio, enerInternOld, sizeof(double) * nb, cudaMemcpyHostToDevice, s);
  cudaMemcpyAsync(d_epo, enerInelasOld, sizeof(double) * nb, cudaMemcpyHostToDevice, s);
  k_vumat_block<<<(unsigned)((nb + 127) / 128), 128, 0, s>>>(nb, make_jc_params(props), *dt, nsv, d_inc, d_sold,
                                                              d_stold, d_eio, d_epo, d_snew, d_stnew, d_tnew,
                                                              d_ein, d_epn);
  cudaMemcpyAsync(stressNew, d_snew, sizeof(double) * 6 * nb, cudaMemcpyDeviceToHost, s);
  cudaMemcpyAsync(stateNew, d_stnew, sizeof(double) * nsv * nb, cudaMemcpyDeviceToHost, s);
  cudaMemcpyAsync(tempNew, d_tnew, sizeof(double) * nb, cudaMemcpyDeviceToHost, s);
  cudaMemcpyAsync(enerInternNew, d_ein, sizeof(double) * nb, cudaMemcpyDeviceToHost, s);
  cudaMemcpyAsync(enerInelasNew, d_epn, sizeof(double) * nb, cudaMemcpyDeviceToHost, s);
  if ((e = cudaStreamSynchronize(s)) != cudaSuccess || (e = cudaGetLastError()) != cudaSuccess)
    fail(e);
}

}  // extern "C"
