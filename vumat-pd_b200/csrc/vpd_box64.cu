// FP64 bond kernels for lattices too small to fill the GPU with the tiles of vpd_tiled64.cu: boxes of
// lattice points staged in shared memory with their neighbourhood, one thread per point and tensor
// row.
//
// A small lattice is bound by latency, not by a pipe or by memory: with two or three points per
// thread in 256- or 384-thread blocks, the 4,000 points of a 40x10x10 bar occupy 4 to 8 of the 148
// SMs, and each thread walks its points' bonds group by group with a memory round trip per
// group. Here a block takes a box of at most 32 points (64 or 128 where that needs fewer waves),
// copies every record that its bonds reach with cp.async, all copies in flight at once, and then
// walks the stencil's slots in shared memory, where a read takes tens of cycles instead of
// hundreds. Warp r of each three sums row r of the deformation sum (or component r of the force),
// so the lattice spreads over six to nine times as many warps; a row repeats the differences of
// the reference positions, a third more FP64 work per bond, which an idle pipe takes for free.
//
// The staged arrays are split into 16- and 8-byte elements, and a row's stride along z is the box's
// extent along z modulo 8, so that the consecutive points of a warp fall into different banks. Their
// length is a template parameter (at least the region's), so that one address serves every array.
//
// Measured on a B200, per increment with the material and integration kernels (28 us), against two points per
// thread in 256-thread blocks: 40x10x10 bar at horizon 3.015 h 92 to 43 us, the archived 101x21x5 lattice at 3 h
// 113 to 57 us. Both kernels are
// still bound by latency: about 3 us to stage the region and 4 us for the 122 slots at one warp
// per scheduler.
//
// Every accumulator takes its point's bonds in slot order with the operations of the per-slot
// kernels (bond_deform64's and k_force_stencil's, roundings spelled out), so the results are
// bit-identical to theirs and to the tiled kernels'.
#include "vpd_bond.cuh"
#include "vpd_umma.cuh"  // smem_u32

#include <type_traits>

namespace vpd {

using umma::smem_u32;

template <int BYTES> __device__ __forceinline__ void copy_async(void *dst, const void *src, bool in) {
  const uint32_t bytes = in ? BYTES : 0;  // 0: zero fill, nothing is read
  if (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes) : "memory");
}

constexpr int kBatch = 4;  // slots read together (a divisor of 32)

// The calling thread's place in its block's box, and the box's place in the lattice.
struct BoxPoint {
  int64_t i;   // point index (0 where !valid)
  bool valid;
  int local;   // the point's index in the staged region
};

// Common start of both kernels: copies the box's region with STAGE(local index, point index, inside),
// fills the slots' offsets within the region and the words' slot counts, and places the thread.
template <typename Stage>
__device__ __forceinline__ BoxPoint box_begin(const StepParams &p, int32_t *s_off, int32_t *s_cnt, Stage stage) {
  const BoxTiles &b = p.box;
  const int ny = p.lat_ny, nz = p.lat_nz;
  const int tile = blockIdx.x, bz = tile % b.tiles_z, by = (tile / b.tiles_z) % b.tiles_y, bx = tile / (b.tiles_z * b.tiles_y);
  const int x0 = bx * b.tx - p.st.rx, y0 = by * b.ty - p.st.ry, z0 = bz * b.tz - p.st.rz;
  for (int e = threadIdx.x; e < b.ex * b.ey * b.ez; e += blockDim.x) {
    const int c = e % b.ez, r = e / b.ez, y = r % b.ey, x = r / b.ey;
    const int gx = x0 + x, gy = y0 + y, gz = z0 + c;
    const bool in = gx >= 0 && gx < p.lat_nx && gy >= 0 && gy < ny && gz >= 0 && gz < nz;
    stage((x * b.ey + y) * b.sz + c, in ? ((int64_t)gx * ny + gy) * nz + gz : 0, in);
  }
  for (int w = threadIdx.x; w < p.st.nw; w += blockDim.x)
    s_cnt[w] = 0;
  for (int k = threadIdx.x; k < 32 * p.st.nw; k += blockDim.x)
    s_off[k] = 0;  // padding slots: never a bond
  __syncthreads();
  for (int g = threadIdx.x; g < p.st.ngroups; g += blockDim.x) {
    const int4 gr = __ldg(p.st.groups + g);  // dx, dz, lowest dy, (slots << 16) | first slot
    const int cnt = gr.w >> 16, pos = gr.w & 0xffff;
    for (int k = 0; k < cnt; ++k)
      s_off[pos + k] = (gr.x * b.ey + gr.z + k) * b.sz + gr.y;
    atomicMax(s_cnt + (pos >> 5), (pos & 31) + cnt);
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  const int q = (threadIdx.x / 96) * 32 + (threadIdx.x & 31);  // point of the box
  const int lz = q % b.tz, ly = (q / b.tz) % b.ty, lx = q / (b.tz * b.ty);
  const int x = bx * b.tx + lx, y = by * b.ty + ly, z = bz * b.tz + lz;
  BoxPoint pt;
  pt.valid = lx < b.tx && x < p.lat_nx && y < ny && z < nz;
  pt.i = pt.valid ? ((int64_t)x * ny + y) * nz + z : 0;
  pt.local = (min(lx, b.tx - 1) + p.st.rx) * b.ey * b.sz + (ly + p.st.ry) * b.sz + lz + p.st.rz;
  return pt;
}

// Row r of F = I + [sum_j V_j (u_j - u_i) (x) xi] K^-1 over all bonds. With damage, the
// critical-stretch tests of the intact forward bonds follow (k_deformation_stencil's), the mask
// words dealt out to the three warps of a point.
template <bool DAMAGE, int M> __global__ void __launch_bounds__(384) k_deformation_box(const __grid_constant__ StepParams p) {
  extern __shared__ __align__(16) unsigned char s_box[];
  __shared__ __align__(16) int32_t s_off[32 * kMaxStencilWords], s_cnt[kMaxStencilWords];
  const int64_t n = p.n;
  double2 *sxy = reinterpret_cast<double2 *>(s_box), *szv = sxy + M;  // (x, y), (z, V)
  double *su = reinterpret_cast<double *>(szv + M);                   // ux | uy | uz
  const double4 *U = (*p.step & 1) ? p.u1 : p.u0;
  const BoxPoint pt = box_begin(p, s_off, s_cnt, [&](int l, int64_t j, bool in) {
    const double *x = reinterpret_cast<const double *>(p.xv + j), *u = reinterpret_cast<const double *>(U + j);
    copy_async<16>(sxy + l, x, in), copy_async<16>(szv + l, x + 2, in);
    copy_async<8>(su + l, u, in), copy_async<8>(su + M + l, u + 1, in), copy_async<8>(su + 2 * M + l, u + 2, in);
  });
  const int r = (threadIdx.x >> 5) % 3, c = pt.local;
  const double2 *xy = sxy + c;  // (z, V) M records on
  const double *ur = su + r * M + c;
  const double x0 = xy[0].x, x1 = xy[0].y, x2 = xy[M].x, ui = ur[0];
  double g0 = 0.0, g1 = 0.0, g2 = 0.0;
  uint32_t mw = pt.valid ? __ldg(p.st.mask + pt.i) : 0u;
  for (int w = 0; w < p.st.nw; ++w) {
    const uint32_t mk = mw;
    if (w + 1 < p.st.nw)
      mw = pt.valid ? __ldg(p.st.mask + (int64_t)(w + 1) * n + pt.i) : 0u;
    const int cnt = s_cnt[w];
    for (int b0 = 0; b0 < cnt; b0 += kBatch) {  // (slots past cnt are padding: zero terms)
      int d[kBatch];
      double2 a[kBatch], z[kBatch];
      double u[kBatch];
#pragma unroll
      for (int b = 0; b < kBatch; ++b)
        d[b] = s_off[32 * w + b0 + b];
#pragma unroll
      for (int b = 0; b < kBatch; ++b)
        a[b] = xy[d[b]], z[b] = xy[M + d[b]], u[b] = ur[d[b]];
#pragma unroll
      for (int b = 0; b < kBatch; ++b) {
        const double v = ((mk >> (b0 + b)) & 1u) ? z[b].y : 0.0;
        const double wd = __dmul_rn(v, u[b] - ui);
        g0 = __fma_rn(wd, a[b].x - x0, g0);
        g1 = __fma_rn(wd, a[b].y - x1, g1);
        g2 = __fma_rn(wd, z[b].x - x2, g2);
      }
    }
  }
  if (pt.valid) {
    double K[9];
#pragma unroll
    for (int k = 0; k < 9; ++k)
      K[k] = p.kinv[k * n + pt.i];
#pragma unroll
    for (int k = 0; k < 3; ++k)
      p.F[(3 * r + k) * n + pt.i] = __dadd_rn(r == k ? 1.0 : 0.0, dot3_rn(g0, g1, g2, K[k], K[3 + k], K[6 + k]));
  }
  if (!DAMAGE)
    return;
  const double lo = 1.0 - 1.0e-9, hi = 1.0 + 1.0e-9;
  const double *u = su + c;
  for (int w = r; w < p.st.nw; w += 3) {
    uint32_t live = pt.valid ? __ldg(p.st.mask + (int64_t)w * n + pt.i) & __ldg(p.st.forward + w) : 0u;
    if (live)
      live &= ~p.st.broken[(int64_t)w * n + pt.i];
    uint32_t fresh = 0u;
    for (uint32_t f = live; f; f &= f - 1) {
      const int b = __ffs(f) - 1, d = s_off[32 * w + b];
      const double e0 = xy[d].x - x0, e1 = xy[d].y - x1, e2 = xy[M + d].x - x2;
      const double y0 = e0 + (u[d] - u[0]), y1 = e1 + (u[M + d] - u[M]), y2 = e2 + (u[2 * M + d] - u[2 * M]);
      const double yy = y0 * y0 + y1 * y1 + y2 * y2;
      const double xx = e0 * e0 + e1 * e1 + e2 * e2;
      const double t = p.tension2 * xx;
      bool broke = false, near = false;
      if (yy > t * hi)
        broke = true;
      else if (yy >= t * lo)
        near = true;
      else if (p.use_compression) {
        const double k = p.compression2 * xx;
        if (yy < k * lo)
          broke = true;
        else if (yy <= k * hi)
          near = true;
      }
      if (near)
        broke = exact_break(p.xv, U, pt.i, pt.i + p.st.delta[32 * w + b], p.dmg_initiation, p.dmg_failure,
                            p.use_compression);
      if (broke)
        fresh |= 1u << b;
    }
    if (fresh) {
      atomicOr(p.st.broken + (int64_t)w * n + pt.i, fresh);
      for (uint32_t f = fresh; f; f &= f - 1) {
        const int sl = 32 * w + __ffs(f) - 1, rv = p.st.reverse[sl];
        atomicOr(p.st.broken + (int64_t)(rv >> 5) * n + (pt.i + p.st.delta[sl]), 1u << (rv & 31));
      }
    }
  }
}

// Component r of f_i = sum_j V_j M_j xi over intact bonds + M_i s_i, s_i = vxi_i - sum_{broken j}
// V_j xi: a bond reads row r of j's force map and its position.
template <int M> __global__ void __launch_bounds__(384) k_force_box(const __grid_constant__ StepParams p) {
  extern __shared__ __align__(16) unsigned char s_box[];
  __shared__ __align__(16) int32_t s_off[32 * kMaxStencilWords], s_cnt[kMaxStencilWords];
  const int64_t n = p.n;
  double2 *sxy = reinterpret_cast<double2 *>(s_box), *sm01 = sxy + M;       // (x, y); rows' (VM_r0, VM_r1)
  double *szz = reinterpret_cast<double *>(sm01 + 3 * M), *sm2 = szz + M;  // z; rows' VM_r2
  const BoxPoint pt = box_begin(p, s_off, s_cnt, [&](int l, int64_t j, bool in) {
    const double *x = reinterpret_cast<const double *>(p.xv + j);
    copy_async<16>(sxy + l, x, in), copy_async<8>(szz + l, x + 2, in);
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const double *f = reinterpret_cast<const double *>(p.fmap + q * n + j);
      copy_async<16>(sm01 + q * M + l, f, in), copy_async<8>(sm2 + q * M + l, f + 2, in);
    }
  });
  const int r = (threadIdx.x >> 5) % 3, c = pt.local;
  const double2 *xy = sxy + c, *m01 = sm01 + r * M + c;
  const double *zz = szz + c, *m2 = sm2 + r * M + c;
  const double x0 = xy->x, x1 = xy->y, x2 = *zz;
  double f = 0.0, c0 = 0.0, c1 = 0.0, c2 = 0.0;
  uint32_t mw = pt.valid ? __ldg(p.st.mask + pt.i) : 0u;
  for (int w = 0; w < p.st.nw; ++w) {
    uint32_t mk = mw;
    if (w + 1 < p.st.nw)
      mw = pt.valid ? __ldg(p.st.mask + (int64_t)(w + 1) * n + pt.i) : 0u;
    if (p.damage && mk) {
      const uint32_t bk = mk & __ldg(p.st.broken + (int64_t)w * n + pt.i);
      for (uint32_t q = bk; q; q &= q - 1) {  // broken bonds leave s_i
        const double4 xj = p.xv[pt.i + p.st.delta[32 * w + __ffs(q) - 1]];
        c0 += xj.w * (xj.x - x0), c1 += xj.w * (xj.y - x1), c2 += xj.w * (xj.z - x2);
      }
      mk &= ~bk;
    }
    const int cnt = s_cnt[w];
    for (int b0 = 0; b0 < cnt; b0 += kBatch) {  // (slots past cnt are padding: zero terms)
      int d[kBatch];
      double2 a[kBatch], k[kBatch];
      double z[kBatch], k2[kBatch];
#pragma unroll
      for (int b = 0; b < kBatch; ++b)
        d[b] = s_off[32 * w + b0 + b];
#pragma unroll
      for (int b = 0; b < kBatch; ++b)
        a[b] = xy[d[b]], k[b] = m01[d[b]], z[b] = zz[d[b]], k2[b] = m2[d[b]];
#pragma unroll
      for (int b = 0; b < kBatch; ++b) {
        const bool bond = (mk >> (b0 + b)) & 1u;
        const double e0 = bond ? a[b].x - x0 : 0.0, e1 = bond ? a[b].y - x1 : 0.0, e2 = bond ? z[b] - x2 : 0.0;
        f = __dadd_rn(f, dot3_rn(k[b].x, k[b].y, k2[b], e0, e1, e2));
      }
    }
  }
  if (!pt.valid)
    return;
  const double4 s = p.vxi[pt.i];
  const double s0 = s.x - c0, s1 = s.y - c1, s2 = s.z - c2;
  f = __dadd_rn(f, __dmul_rn(dot3_rn(m01->x, m01->y, *m2, s0, s1, s2), 1.0 / p.xv[pt.i].w));
  double *out = reinterpret_cast<double *>(p.force + pt.i);
  if (r < 2)
    out[r] = f;
  else
    *reinterpret_cast<double2 *>(out + 2) = make_double2(f, 0.0);
}

constexpr size_t kDeformRecord = 2 * sizeof(double2) + 3 * sizeof(double);
constexpr size_t kForceRecord = 4 * sizeof(double2) + 4 * sizeof(double);
constexpr size_t kBoxStatic = 33 * kMaxStencilWords * sizeof(int32_t);
constexpr size_t kBoxMaxBytes = 227 * 1024 - kBoxStatic;

// kernel(std::integral_constant<int, M>) with the smallest staged length M that holds `records`
template <typename F> static int with_records(int records, F &&kernel) {
  if (records <= 768)
    return kernel(std::integral_constant<int, 768>{});
  if (records <= 1152)
    return kernel(std::integral_constant<int, 1152>{});
  if (records <= 1536)
    return kernel(std::integral_constant<int, 1536>{});
  return kernel(std::integral_constant<int, 2304>{});
}
constexpr int kBoxMaxRecords = 2304;

// The boxes of a lattice: the extents whose tiles need the fewest waves of 148 blocks, then the
// smallest staged regions, of at most 32 points (one block per SM up to 4,736 points), 64 or 128
// (more points per staged region where several blocks would queue per SM anyway). Boxes that need a second wave are
// not taken (unless asked for, p.tiled 7): a long reach leaves room for a few points beside it in a region, and each
// box stages it again. Per increment in microseconds, boxes | tiles: one wave, 10,605 points at 4.5 h, 118 | 112; two,
// 9,000 points at 5 h, 175 | 99; twelve, 4,913 points at 5 h, 877 | 148.
int setup_box64(StepParams &p) {
  p.box = BoxTiles{};
  const int points = p.n <= 148 * 32 ? 32 : (p.n <= 148 * 48 ? 64 : 128);
  double best = 0.0;
  for (int tx = 1; tx <= points; ++tx)
    for (int ty = 1; tx * ty <= points; ++ty)
      for (int tz = 1; tx * ty * tz <= points; ++tz) {
        BoxTiles b;
        b.tx = tx, b.ty = ty, b.tz = tz, b.threads = 3 * points;
        b.ex = tx + 2 * p.st.rx, b.ey = ty + 2 * p.st.ry, b.ez = tz + 2 * p.st.rz;
        b.sz = b.ez + ((tz - b.ez) % 8 + 8) % 8;
        b.records = b.ex * b.ey * b.sz;
        if (b.records > kBoxMaxRecords)
          continue;
        b.tiles_y = (p.lat_ny + ty - 1) / ty, b.tiles_z = (p.lat_nz + tz - 1) / tz;
        b.tiles = (int64_t)((p.lat_nx + tx - 1) / tx) * b.tiles_y * b.tiles_z;
        const double waves = (double)((b.tiles + 147) / 148), cost = waves * (4096.0 + (double)b.records);
        if (!p.box.threads || cost < best)
          best = cost, p.box = b;
      }
  if (p.box.tiles > 148 && p.tiled != 7)
    p.box = BoxTiles{};
  if (!p.box.threads)
    return VPD_OK;
  return with_records(p.box.records, [&](auto m) {
    constexpr int M = decltype(m)::value;
    static_assert(M * kForceRecord <= kBoxMaxBytes, "the staged region exceeds shared memory");
    const cudaFuncAttribute attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    VPD_CUDA(cudaFuncSetAttribute(k_deformation_box<true, M>, attr, (int)(M * kDeformRecord)));
    VPD_CUDA(cudaFuncSetAttribute(k_deformation_box<false, M>, attr, (int)(M * kDeformRecord)));
    VPD_CUDA(cudaFuncSetAttribute(k_force_box<M>, attr, (int)(M * kForceRecord)));
    return (int)VPD_OK;
  });
}

int launch_deformation_box64(const StepParams &p, cudaStream_t s) {
  return with_records(p.box.records, [&](auto m) {
    constexpr int M = decltype(m)::value;
    const unsigned grid = (unsigned)p.box.tiles;
    if (p.damage)
      k_deformation_box<true, M><<<grid, p.box.threads, M * kDeformRecord, s>>>(p);
    else
      k_deformation_box<false, M><<<grid, p.box.threads, M * kDeformRecord, s>>>(p);
    VPD_CUDA(cudaGetLastError());
    return (int)VPD_OK;
  });
}
int launch_force_box64(const StepParams &p, cudaStream_t s) {
  return with_records(p.box.records, [&](auto m) {
    constexpr int M = decltype(m)::value;
    k_force_box<M><<<(unsigned)p.box.tiles, p.box.threads, M * kForceRecord, s>>>(p);
    VPD_CUDA(cudaGetLastError());
    return (int)VPD_OK;
  });
}

}  // namespace vpd
