// The surrogate network's forward pass and gradients on the tensor cores.
//
// Network: 10 -> 128 -> 128 -> 128 -> 7 with SiLU activations, BF16 weights and activations,
// FP32 accumulation. Inputs and outputs are padded to 16 columns (zero weights outside).
// A tile is 128 batch rows; its rows are TMEM lanes. The MMAs are tcgen05.mma kind::f16 (BF16 x BF16 ->
// FP32 in TMEM), issued by one thread, completion signalled through an mbarrier (tcgen05.commit);
// every wait is bounded and reports a timeout in *err.
#include "vpd_mlp_tile.cuh"
#include "vpd_surrogate.cuh"

#include <algorithm>
#include <vector>

namespace vpd {

// W1 (128x16) | W2 (128x128) | W3 | W4 (16x128), as staged by both kernels
constexpr int kWeightBytes = 4096 + 32768 + 32768 + 4096;
struct StagedWeights {
  unsigned char *w1, *w2, *w3, *w4;
};
// Every thread calls it; complete at stage_wait() and, for tiled weights, the first phase of wbar (initialised by
// thread 0).
__device__ __forceinline__ StagedWeights stage_weights(unsigned char *s, const MlpWeights &w, uint64_t *wbar) {
  const StagedWeights sw{s, s + 4096, s + 4096 + 32768, s + 4096 + 65536};
  if (w.tiled) {
    if (threadIdx.x == 0)
      umma::bulk_load(s, w.w1, kWeightBytes, wbar);
    return sw;
  }
  stage_rowmajor(sw.w1, w.w1, kMlpHidden, kMlpIn);
  stage_rowmajor(sw.w2, w.w2, kMlpHidden, kMlpHidden);
  stage_rowmajor(sw.w3, w.w3, kMlpHidden, kMlpHidden);
  stage_rowmajor(sw.w4, w.w4, kMlpOut, kMlpHidden);
  return sw;
}

// ------------------------------------------------------------------ forward
// Persistent blocks, one per SM: the weights are staged once, and four groups of 128 threads run a tile each
// (thread t of a group = TMEM lane t), with their own operand tile, 128 TMEM columns, mbarrier and
// named barrier. A tile's four products and epilogues are a serial chain; the four groups of a block
// overlap theirs. The hidden layers are formed as Y^T = W Y_prev^T, features along the lanes, so that a thread
// has one bias a layer, in a register: with batch rows along the lanes a thread read all 128 from shared memory. The
// activations are stored [feature][batch row], for the next product to read through MN-major descriptors; the output
// layer reads them as its first operand, so its batch rows are lanes again.
// What bounds it is the epilogue: 384 tanh per row at 16 per SM and clock, 83 us for 1M rows,
// against 43 us of tensor work and 20 us of memory traffic. Measured on a B200: 137 us for 1M rows (152 with
// the batch rows along the lanes; 490 with a block per tile that staged the 72 KB of weights each time), 60 %
// of it the tanh unit's own time; without its tanh the kernel takes 106 us, without its tensor work 130. Two warps a
// TMEM quarter (142 us) and two half tiles a group in turn (148) have shorter waits but more of them.
constexpr int kGroups = 4;
constexpr size_t kFwdSmem = kWeightBytes + kGroups * 32768 + (kGroups + 1) * 16 + 4 * kBiasFloats;

// Four consecutive floats; the callers' arrays may start at any multiple of 4 bytes (vec: at one of 16).
__device__ __forceinline__ float4 load4(const float *p, bool vec) {
  return vec ? __ldg(reinterpret_cast<const float4 *>(p)) : make_float4(__ldg(p), __ldg(p + 1), __ldg(p + 2), __ldg(p + 3));
}
__device__ __forceinline__ void store4(float *p, float4 v, bool vec) {
  if (vec)
    *reinterpret_cast<float4 *>(p) = v;
  else
    p[0] = v.x, p[1] = v.y, p[2] = v.z, p[3] = v.w;
}
__device__ __forceinline__ bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// Barrier and vote of one group's 128 threads.
__device__ __forceinline__ void group_sync(int g) { asm volatile("bar.sync %0, 128;" ::"r"(g + 1) : "memory"); }
__device__ __forceinline__ bool group_all(int g, bool v) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "bar.red.and.pred q, %2, 128, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}\n"
      : "=r"(r)
      : "r"((uint32_t)v), "r"(g + 1)
      : "memory");
  return r != 0;
}

__global__ void __launch_bounds__(128 * kGroups, 1) k_mlp_forward(MlpWeights w, const float *x, int64_t B, float *out,
                                                                  unsigned *err) {
  extern __shared__ __align__(1024) unsigned char smem[];
  unsigned char *sAll = smem + kWeightBytes;
  uint64_t *mbars = reinterpret_cast<uint64_t *>(sAll + kGroups * 32768);
  uint64_t *wbar = mbars + 2 * kGroups;
  float *sBias = reinterpret_cast<float *>(sAll + kGroups * 32768 + (kGroups + 1) * 16);
  __shared__ uint32_t s_tmem;
  const int g = threadIdx.x >> 7, t = threadIdx.x & 127;
  if (threadIdx.x < 32)
    umma::tmem_alloc(&s_tmem, 128 * kGroups);
  if (t == 0)
    umma::mbar_init(mbars + 2 * g, 1);
  if (threadIdx.x == 0)
    umma::mbar_init(wbar, 1);
  const StagedWeights sw = stage_weights(smem, w, wbar);
  stage_biases(sBias, w);
  stage_wait();
  umma::fence_proxy_async();
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  unsigned char *sA = sAll + g * 32768;  // the batch rows' 16 features (in its first 4 KB), then the activations
  uint64_t *mbar = mbars + 2 * g;
  const uint32_t tmem = s_tmem + 128u * g;
  const uint32_t trow = tmem + ((uint32_t)(t & ~31) << 16);  // this warp's TMEM lanes
  uint32_t phase = 0;
  bool ok = !w.tiled || group_all(g, umma::mbar_wait(wbar, 0u, kWaitLimit));
  const float b1 = sBias[t], b2 = sBias[kMlpHidden + t], b3 = sBias[2 * kMlpHidden + t];
  // D = A B^T by the group's first thread, awaited by the group. A wait that runs out leaves ok false; the group
  // votes on it once a tile.
  auto product = [&](const umma::Operand &a, const umma::Operand &b, int K, int N) {
    umma::fence_proxy_async();
    umma::fence_before_sync();
    group_sync(g);
    if (t == 0) {
      umma::fence_after_sync();
      umma::gemm_issue(tmem, a, b, K, N);
      umma::commit(mbar);
    }
    ok = umma::mbar_wait(mbar, phase, kWaitLimit) && ok;
    phase ^= 1u;
    umma::fence_after_sync();
  };
  const int64_t tiles = (B + 127) / 128;
  const bool vecx = aligned16(x), veco = aligned16(out);
  float4 next[4];
  auto load = [&](int64_t tile) {
    const int64_t row = tile * 128 + t;
#pragma unroll
    for (int c = 0; c < 4; ++c)
      next[c] = row < B ? load4(x + row * kMlpIn + 4 * c, vecx) : make_float4(0.f, 0.f, 0.f, 0.f);
  };
  // group g of block b takes tiles b + (g + kGroups k) gridDim: few tiles spread over the blocks first
  const int64_t stride = (int64_t)kGroups * gridDim.x;
  int64_t tile = blockIdx.x + (int64_t)g * gridDim.x;
  if (tile < tiles)
    load(tile);
  for (; tile < tiles && ok; tile += stride) {
    __align__(16) __nv_bfloat16 xb[16];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      xb[4 * c] = __float2bfloat16(next[c].x), xb[4 * c + 1] = __float2bfloat16(next[c].y);
      xb[4 * c + 2] = __float2bfloat16(next[c].z), xb[4 * c + 3] = __float2bfloat16(next[c].w);
    }
    *reinterpret_cast<uint4 *>(sA + kmajor_offset(t, 0, kMlpIn)) = *reinterpret_cast<const uint4 *>(xb);
    *reinterpret_cast<uint4 *>(sA + kmajor_offset(t, 8, kMlpIn)) = *reinterpret_cast<const uint4 *>(xb + 8);
    if (tile + stride < tiles)
      load(tile + stride);
    const umma::Operand y = umma::mn_major(sA, 128);
    product(umma::k_major(sw.w1, kMlpIn), umma::k_major(sA, kMlpIn), kMlpIn, 128);
    feature_epilogue(trow, b1, sA, t);
    product(umma::k_major(sw.w2, kMlpHidden), y, kMlpHidden, 128);
    feature_epilogue(trow, b2, sA, t);
    product(umma::k_major(sw.w3, kMlpHidden), y, kMlpHidden, 128);
    feature_epilogue(trow, b3, sA, t);
    product(y, umma::k_major(sw.w4, kMlpHidden), kMlpHidden, kMlpOut);
    ok = group_all(g, ok);
    const int64_t row = tile * 128 + t;
    float v[16];
    if (ok)
      umma::tmem_ld16(trow, v);
    if (row < B) {
#pragma unroll
      for (int c = 0; c < kMlpOut; c += 4) {
        const float4 bb = *reinterpret_cast<const float4 *>(sBias + 3 * kMlpHidden + c);
        store4(out + row * kMlpOut + c,
               ok ? make_float4(v[c] + bb.x, v[c + 1] + bb.y, v[c + 2] + bb.z, v[c + 3] + bb.w)
                  : make_float4(0.f, 0.f, 0.f, 0.f),
               veco);
      }
    }
  }
  if (!ok && t == 0)
    atomicOr(err, 1u);
  umma::fence_before_sync();
  __syncthreads();
  if (threadIdx.x < 32)
    umma::tmem_dealloc(s_tmem, 128 * kGroups);
}

// ------------------------------------------------------------------ gradients
// Forward and backward of one 128-row tile per block, everything between in shared memory and TMEM (the two
// passes as kernels of their own wrote and read 2.3 KB a row of pre-activations and activations, a third kernel
// transposed the weights, and 128 threads ran every epilogue of the tile alone). 512 threads: warp w holds the TMEM
// lanes (rows) of its quarter w % 4 and the 32 columns of its group w / 4.
//   forward   Z1 = X W1^T, Y1 = silu(Z1 + b1) ... Y3; Z2 and Z3 stay in TMEM, Z1 (one K = 16 product) is formed again
//   backward  dZ = dY * silu'(Z); dW = dZ^T Y_prev and dY_prev = dZ W. The products that need an operand the other
//             way round read the forward pass's own tiles through MN-major descriptors.
// The tile's weight and bias gradients go to the block's slice of `partials`; the slices are summed in block
// order, so the gradient does not depend on the order the blocks run in. Batch 8192 on a B200: 21 us (20 with
// tiled weights) and 3.3 us for the sum (46 + 60 + 6 us in the separate kernels). Eight dependent stages at one
// block on 64 SMs, so latency: about 4 us to start and stage, 0.2 to 0.5 us a product, 0.7 us a forward epilogue, 1.6
// to 3 us a backward one with its stores (5.5 us before they turned through shared memory).
constexpr int kGradThreads = 512;
// weights | Y0 (128x16) | Y1 | Y2 | Y3 | dZ (128x128) | dZ4 (128x16) | mbarrier | biases
constexpr size_t kGradSmem = kWeightBytes + 4096 + 4 * 32768 + 4096 + 64 + 4 * kBiasFloats;

// Column sums of a 16-column slab over the 32 lanes of a warp, by halving: each step a lane
// keeps half of its columns and adds the partner's copy of them (16 shuffles in all). Lane l
// returns the sum of column col = 8 b4 + 4 b3 + 2 b2 + b1 (b_k: bit k of l); lanes l and l ^ 1
// hold the same column.
__device__ __forceinline__ float warp_column_sums16(const float (&v)[16], int lane, int &col) {
  const bool h4 = lane & 16, h3 = lane & 8, h2 = lane & 4, h1 = lane & 2;
  float a[8], b[4], d[2];
#pragma unroll
  for (int c = 0; c < 8; ++c)
    a[c] = (h4 ? v[c + 8] : v[c]) + __shfl_xor_sync(0xffffffffu, h4 ? v[c] : v[c + 8], 16);
#pragma unroll
  for (int c = 0; c < 4; ++c)
    b[c] = (h3 ? a[c + 4] : a[c]) + __shfl_xor_sync(0xffffffffu, h3 ? a[c] : a[c + 4], 8);
#pragma unroll
  for (int c = 0; c < 2; ++c)
    d[c] = (h2 ? b[c + 2] : b[c]) + __shfl_xor_sync(0xffffffffu, h2 ? b[c] : b[c + 2], 4);
  float e = (h1 ? d[1] : d[0]) + __shfl_xor_sync(0xffffffffu, h1 ? d[0] : d[1], 2);
  e += __shfl_xor_sync(0xffffffffu, e, 1);
  col = (h4 ? 8 : 0) + (h3 ? 4 : 0) + (h2 ? 2 : 0) + (h1 ? 1 : 0);
  return e;
}

template <bool TRAIN>
__global__ void __launch_bounds__(kGradThreads, 1) k_mlp_gradient(MlpWeights w, MlpBatch batch, int64_t B, float *partials,
                                                                  unsigned *err) {
  extern __shared__ __align__(1024) unsigned char smem[];
  unsigned char *sY0 = smem + kWeightBytes, *sY1 = sY0 + 4096, *sY2 = sY1 + 32768, *sY3 = sY2 + 32768;
  unsigned char *sDZ = sY3 + 32768, *sDZ4 = sDZ + 32768;
  uint64_t *mbar = reinterpret_cast<uint64_t *>(sDZ4 + 4096);
  float *sBias = reinterpret_cast<float *>(sDZ4 + 4096 + 64);
  __shared__ uint32_t s_tmem;
  __shared__ float s_db[4][kMlpHidden];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, quarter = warp & 3, group = warp >> 2;
  const int t = quarter * 32 + lane;  // the thread's row (of the tile, and of dW)
  const int c0 = group * 32;          // ... and its first column
  const int64_t row0 = (int64_t)blockIdx.x * 128, row = row0 + t;
  const bool keep = row < B;
  const MlpGrads grad = mlp_grads(partials + (size_t)blockIdx.x * kMlpParams);
  if (warp == 0)
    umma::tmem_alloc(&s_tmem, 512);
  uint64_t *wbar = mbar + 2;
  if (threadIdx.x == 0)
    umma::mbar_init(mbar, 1), umma::mbar_init(wbar, 1);
  const StagedWeights sw = stage_weights(smem, w, wbar);
  stage_biases(sBias, w);
  // the batch row's place in the arrays it is read from
  auto source = [&](int64_t r) {
    return TRAIN ? (int64_t)((batch.mul * (uint64_t)(batch.first + r) + batch.add) % (uint64_t)batch.rows) : r;
  };
  {  // inputs: four threads a row
    const int rr = threadIdx.x >> 2, part = threadIdx.x & 3;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (row0 + rr < B)
      v = load4(batch.x + source(row0 + rr) * kMlpIn + 4 * part, aligned16(batch.x));
    __align__(8) __nv_bfloat16 xb[4] = {__float2bfloat16(v.x), __float2bfloat16(v.y), __float2bfloat16(v.z),
                                        __float2bfloat16(v.w)};
    *reinterpret_cast<uint2 *>(sY0 + kmajor_offset(rr, 4 * part, kMlpIn)) = *reinterpret_cast<const uint2 *>(xb);
  }
  // the output layer's rows, a row per thread of the first group: read now, used after the forward pass
  float4 last[4];
  if (group == 0) {
    const float *from = TRAIN ? batch.target + (keep ? source(row) : 0) * 16 : batch.gout + (keep ? row : 0) * kMlpOut;
    const bool vec = aligned16(from);
#pragma unroll
    for (int c = 0; c < 4; ++c)
      last[c] = load4(from + 4 * c, vec);
  }
  stage_wait();
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tmem = s_tmem, lanes = (uint32_t)(quarter * 32) << 16;
  // four accumulators of 128 columns
  const uint32_t T0 = tmem, T1 = tmem + 128, T2 = tmem + 256, T3 = tmem + 384;
  Sync sy{mbar, 0u, err, 1u, true};
  if (w.tiled) {
    sy.ok = __syncthreads_and(umma::mbar_wait(wbar, 0u, kWaitLimit)) != 0;
    if (!sy.ok && threadIdx.x == 0)
      atomicOr(err, 1u);
  }
  // The stage's products, issued by one thread once every thread's operands are in place, awaited by all.
  auto stage = [&](auto issue) {
    umma::fence_proxy_async();
    umma::fence_before_sync();
    __syncthreads();
    if (threadIdx.x == 0) {
      umma::fence_after_sync();
      issue();
      umma::commit(mbar);
    }
    sy.wait();
  };
  auto hidden = [&](uint32_t acc, const float *bias, unsigned char *Y) {
    float v[32];
    umma::tmem_ld32(acc + lanes + c0, v);
    hidden_columns(v, bias, Y, t, c0);
  };
  const int H = kMlpHidden;

  // ---- forward
  stage([&] { umma::gemm_issue(T0, umma::k_major(sY0, kMlpIn), umma::k_major(sw.w1, kMlpIn), kMlpIn, H); });
  if (sy.ok)
    hidden(T0, sBias, sY1);
  stage([&] { umma::gemm_issue(T1, umma::k_major(sY1, H), umma::k_major(sw.w2, H), H, H); });
  if (sy.ok)
    hidden(T1, sBias + H, sY2);
  stage([&] { umma::gemm_issue(T2, umma::k_major(sY2, H), umma::k_major(sw.w3, H), H, H); });
  if (sy.ok)
    hidden(T2, sBias + 2 * H, sY3);
  if (TRAIN)
    stage([&] { umma::gemm_issue(T3, umma::k_major(sY3, H), umma::k_major(sw.w4, H), H, kMlpOut); });

  // ---- output layer: dZ4 = gout, a row per thread of the first group
  if (group == 0) {
    float dz4[kMlpOut];
    if (TRAIN) {
      // weighted MSE over the 7 targets (row weight in target column 15, target 0 weighted 4)
      float o[16], l = 0.0f;
      if (sy.ok)
        umma::tmem_ld16(T3 + lanes, o);
      const float target[16] = {last[0].x, last[0].y, last[0].z, last[0].w, last[1].x, last[1].y, last[1].z, last[1].w,
                                last[2].x, last[2].y, last[2].z, last[2].w, last[3].x, last[3].y, last[3].z, last[3].w};
      const float wr = keep ? target[15] : 0.0f, norm = 1.0f / (float)(B * SURROGATE_TARGETS);
#pragma unroll
      for (int c = 0; c < kMlpOut; ++c) {
        const float cw = c == 0 ? 4.0f : 1.0f;
        const float d = keep && sy.ok && c < SURROGATE_TARGETS ? (o[c] + sBias[3 * H + c]) - target[c] : 0.0f;
        dz4[c] = 2.0f * wr * cw * d * norm;
        l += wr * cw * d * d * norm;
      }
#pragma unroll
      for (int k = 16; k > 0; k >>= 1)
        l += __shfl_xor_sync(0xffffffffu, l, k);
      if (lane == 0)
        atomicAdd(batch.loss, l);
    } else {
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        dz4[4 * c] = keep ? last[c].x : 0.0f, dz4[4 * c + 1] = keep ? last[c].y : 0.0f;
        dz4[4 * c + 2] = keep ? last[c].z : 0.0f, dz4[4 * c + 3] = keep ? last[c].w : 0.0f;
      }
    }
    __align__(16) __nv_bfloat16 zb[16];
#pragma unroll
    for (int c = 0; c < kMlpOut; ++c)
      zb[c] = __float2bfloat16(dz4[c]);
    *reinterpret_cast<uint4 *>(sDZ4 + kmajor_offset(t, 0, kMlpOut)) = *reinterpret_cast<const uint4 *>(zb);
    *reinterpret_cast<uint4 *>(sDZ4 + kmajor_offset(t, 8, kMlpOut)) = *reinterpret_cast<const uint4 *>(zb + 8);
    int col;
    const float sum = warp_column_sums16(dz4, lane, col);
    if (!(lane & 1))
      s_db[quarter][col] = sum;
  }
  // dW4^T [in][out] = Y3^T dZ4 ; dY3 = dZ4 W4
  stage([&] {
    umma::gemm_issue(T0, umma::mn_major(sY3, H), umma::mn_major(sDZ4, kMlpOut), 128, kMlpOut);
    umma::gemm_issue(T3, umma::k_major(sDZ4, kMlpOut), umma::mn_major(sw.w4, H), kMlpOut, H);
  });
  if (threadIdx.x < kMlpOut)
    grad.b4[threadIdx.x] =
        s_db[0][threadIdx.x] + s_db[1][threadIdx.x] + s_db[2][threadIdx.x] + s_db[3][threadIdx.x];
  if (group == 0 && sy.ok) {  // thread t holds dW4^T row t (input t): grad_w4[out][t]
    float v[16];
    umma::tmem_ld16(T0 + lanes, v);
#pragma unroll
    for (int c = 0; c < kMlpOut; ++c)
      grad.w4[(size_t)c * H + t] = v[c];
  }
  __syncthreads();  // s_db is written again below

  // ---- hidden layers 3, 2, 1
#pragma unroll 1  // one copy of the code: every instruction is fetched once per layer otherwise
  for (int layer = 3; layer >= 1; --layer) {
    if (!sy.ok)
      break;
    const uint32_t Z = layer == 3 ? T2 : (layer == 2 ? T1 : T0);
    const float *bias = sBias + (layer - 1) * H;
    // dZ = dY * SiLU'(Z): the thread's columns of its row
    {
      float v[32], z[32];
      umma::tmem_ld32(T3 + lanes + c0, v);
      umma::tmem_ld32(Z + lanes + c0, z);
      __align__(16) __nv_bfloat162 zb[16];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const float4 bb = *reinterpret_cast<const float4 *>(bias + c0 + 4 * q);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int c = 4 * q + 2 * e;
          float2 d = silu_grad2(make_float2(v[c], v[c + 1]), make_float2(z[c], z[c + 1]),
                                e ? make_float2(bb.z, bb.w) : make_float2(bb.x, bb.y));
          d = keep ? d : make_float2(0.0f, 0.0f);
          v[c] = d.x, v[c + 1] = d.y;
          zb[2 * q + e] = __floats2bfloat162_rn(d.x, d.y);
        }
      }
#pragma unroll
      for (int k = 0; k < 4; ++k)
        *reinterpret_cast<uint4 *>(sDZ + kmajor_offset(t, c0 + 8 * k, H)) = *reinterpret_cast<const uint4 *>(zb + 4 * k);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float slab[16];
#pragma unroll
        for (int c = 0; c < 16; ++c)
          slab[c] = v[16 * h + c];
        int col;
        const float sum = warp_column_sums16(slab, lane, col);
        if (!(lane & 1))
          s_db[quarter][c0 + 16 * h + col] = sum;
      }
    }
    // dW [out][in] = dZ^T Y_prev over Z's columns, dY_prev = dZ W over dY's
    stage([&] {
      if (layer > 1) {
        umma::gemm_issue(Z, umma::mn_major(sDZ, H), umma::mn_major(layer == 3 ? sY2 : sY1, H), 128, H);
        umma::gemm_issue(T3, umma::k_major(sDZ, H), umma::mn_major(layer == 3 ? sw.w3 : sw.w2, H), H, H);
      } else {
        umma::gemm_issue(Z, umma::mn_major(sDZ, H), umma::mn_major(sY0, kMlpIn), 128, kMlpIn);
      }
      if (layer == 2)  // Z1 again
        umma::gemm_issue(T0, umma::k_major(sY0, kMlpIn), umma::k_major(sw.w1, kMlpIn), kMlpIn, H);
    });
    float *gb = layer == 3 ? grad.b3 : (layer == 2 ? grad.b2 : grad.b1);
    if (threadIdx.x < H)
      gb[threadIdx.x] =
          s_db[0][threadIdx.x] + s_db[1][threadIdx.x] + s_db[2][threadIdx.x] + s_db[3][threadIdx.x];
    if (sy.ok) {
      if (layer > 1) {  // this thread's 32 columns of row t of dW [out][in]
        float v[32];
        umma::tmem_ld32(Z + lanes + c0, v);
        // through the warp's 2 KB of Y3 (not needed any more), 16 columns at a time: a store then covers 64 bytes of
        // eight rows instead of 16 bytes of 32 (the 16-byte chunks swizzled against bank conflicts)
        float4 *turn = reinterpret_cast<float4 *>(sY3) + warp * 128;
        float *dst = (layer == 3 ? grad.w3 : grad.w2) + (size_t)(quarter * 32) * H + c0;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
#pragma unroll
          for (int q = 0; q < 4; ++q)
            turn[lane * 4 + (q ^ ((lane >> 1) & 3))] =
                make_float4(v[16 * h + 4 * q], v[16 * h + 4 * q + 1], v[16 * h + 4 * q + 2], v[16 * h + 4 * q + 3]);
          __syncwarp();
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int rr = 8 * k + (lane >> 2), q = lane & 3;
            *reinterpret_cast<float4 *>(dst + (size_t)rr * H + 16 * h + 4 * q) = turn[rr * 4 + (q ^ ((rr >> 1) & 3))];
          }
          __syncwarp();
        }
      } else if (group == 0) {
        float v[16];
        umma::tmem_ld16(Z + lanes, v);
        float4 *dst = reinterpret_cast<float4 *>(grad.w1 + (size_t)t * kMlpIn);
#pragma unroll
        for (int q = 0; q < 4; ++q)
          dst[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
      }
    }
    __syncthreads();  // s_db is written again by the next layer
  }
  umma::fence_before_sync();
  __syncthreads();
  if (warp == 0)
    umma::tmem_dealloc(tmem, 512);
}

// s + the sum over blocks b (in order) of partials[b][i]
__device__ __forceinline__ float partial_sum(const float *partials, int nblocks, int i, float s = 0.0f) {
#pragma unroll 32
  for (int b = 0; b < nblocks; ++b)
    s += partials[(size_t)b * kMlpParams + i];
  return s;
}
// (first: the sum begins with these partials, else grad holds that of the blocks before them)
__global__ void k_sum_partials(const float *partials, int nblocks, float *grad, bool first) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < kMlpParams)
    grad[i] = partial_sum(partials, nblocks, i, first ? 0.0f : grad[i]);
}

// One Adam step on the summed gradient; the weights (the first kMlpWeights parameters) also to their BF16 copy, in
// tiled storage.
__global__ void k_adam(const float *partials, int nblocks, float *p, float *m, float *v, __nv_bfloat16 *pb, float lr,
                       float b1, float b2, float eps, float c1, float c2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= kMlpParams)
    return;
  const float g = partial_sum(partials, nblocks, i);
  const float mi = b1 * m[i] + (1.0f - b1) * g;
  const float vi = b2 * v[i] + (1.0f - b2) * g * g;
  m[i] = mi, v[i] = vi;
  const float pi = p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  p[i] = pi;
  if (i < kMlpWeights)
    pb[mlp_tile_index(i)] = __float2bfloat16(pi);
}

int mlp_forward(const MlpWeights &w, const float *x, int64_t B, float *out, unsigned *err, cudaStream_t s) {
  int dev = 0, sms = 0;
  VPD_CUDA(cudaGetDevice(&dev));
  VPD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  VPD_CUDA(cudaFuncSetAttribute(k_mlp_forward, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFwdSmem));
  const int64_t grid = std::min<int64_t>((B + 127) / 128, sms);
  k_mlp_forward<<<(unsigned)grid, 128 * kGroups, kFwdSmem, s>>>(w, x, B, out, err);
  VPD_CUDA(cudaGetLastError());
  return VPD_OK;
}

int64_t mlp_gradient_blocks(int64_t B) { return (B + 127) / 128; }

int mlp_gradient_partials(const MlpWeights &w, const MlpBatch &batch, int64_t B, float *partials, unsigned *err,
                          cudaStream_t s) {
  auto *kernel = batch.gout ? k_mlp_gradient<false> : k_mlp_gradient<true>;
  VPD_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGradSmem));
  kernel<<<(unsigned)mlp_gradient_blocks(B), kGradThreads, kGradSmem, s>>>(w, batch, B, partials, err);
  VPD_CUDA(cudaGetLastError());
  return VPD_OK;
}

constexpr unsigned kParamBlocks = (unsigned)((kMlpParams + 127) / 128);

int mlp_sum_partials(const float *partials, int64_t blocks, float *grad, bool first, cudaStream_t s) {
  k_sum_partials<<<kParamBlocks, 128, 0, s>>>(partials, (int)blocks, grad, first);
  VPD_CUDA(cudaGetLastError());
  return VPD_OK;
}

int mlp_adam(const float *partials, int64_t blocks, float *p, float *m, float *v, __nv_bfloat16 *wb, float lr,
             int step, cudaStream_t s) {
  const float b1 = 0.9f, b2 = 0.999f;
  const float c1 = 1.0f - powf(b1, (float)step), c2 = 1.0f - powf(b2, (float)step);
  k_adam<<<kParamBlocks, 128, 0, s>>>(partials, (int)blocks, p, m, v, wb, lr, b1, b2, 1e-8f, c1, c2);
  VPD_CUDA(cudaGetLastError());
  return VPD_OK;
}

}  // namespace vpd

// ------------------------------------------------------------------ C ABI (device pointers)
namespace {
// The end of a call: its timeout word (in ws) read, its work done.
int check_err(unsigned *derr, vpd::Workspace &ws, cudaStream_t s) {
  unsigned e = 0;
  VPD_CUDA(cudaMemcpyAsync(&e, derr, sizeof e, cudaMemcpyDeviceToHost, s));
  ws.finish();
  VPD_CUDA(cudaStreamSynchronize(s));
  if (e)
    return vpd::set_error(VPD_ERR_CUDA, "surrogate network: tensor-core wait timed out");
  return VPD_OK;
}
}  // namespace

using namespace vpd;

extern "C" int vpd_mlp_forward(const uint16_t *weights, const float *biases, const float *x, int64_t batch,
                               float *out, void *stream) {
  if (!weights || !biases || !x || !out || batch < 1)
    return set_error(VPD_ERR_INVALID, "vpd_mlp_forward: invalid argument");
  cudaStream_t s = (cudaStream_t)stream;
  Workspace ws(s);
  unsigned *derr = nullptr;
  int rc = ws.alloc(&derr, 1);
  if (rc)
    return rc;
  VPD_CUDA(cudaMemsetAsync(derr, 0, sizeof(unsigned), s));
  const MlpWeights w = mlp_weights(reinterpret_cast<const __nv_bfloat16 *>(weights), biases);
  rc = mlp_forward(w, x, batch, out, derr, s);
  return rc == VPD_OK ? check_err(derr, ws, s) : rc;
}

extern "C" int vpd_mlp_gradients(const uint16_t *weights, const float *biases, const float *x,
                                 const float *gout, int64_t batch, float *grad, void *stream) {
  if (!weights || !biases || !x || !gout || !grad || batch < 1)
    return set_error(VPD_ERR_INVALID, "vpd_mlp_gradients: invalid argument");
  cudaStream_t s = (cudaStream_t)stream;
  const MlpWeights w = mlp_weights(reinterpret_cast<const __nv_bfloat16 *>(weights), biases);
  // in parts of at most kPartBlocks blocks, whose partials (154 MB) stay within what the pool keeps; the sum runs on over
  // the parts in block order
  constexpr int64_t kPartBlocks = 7 * 148;
  const int64_t blocks = mlp_gradient_blocks(batch);
  Workspace ws(s);
  unsigned *derr = nullptr;
  float *partials = nullptr;
  int rc;
  if ((rc = ws.alloc(&derr, 1)) || (rc = ws.alloc(&partials, (size_t)std::min(blocks, kPartBlocks) * kMlpParams)))
    return rc;
  VPD_CUDA(cudaMemsetAsync(derr, 0, sizeof(unsigned), s));
  for (int64_t b = 0; b < blocks; b += kPartBlocks) {
    const int64_t row = 128 * b, count = std::min(kPartBlocks, blocks - b);
    MlpBatch rows{};
    rows.x = x + row * kMlpIn, rows.gout = gout + row * kMlpOut;
    if ((rc = mlp_gradient_partials(w, rows, std::min(batch - row, 128 * count), partials, derr, s)) ||
        (rc = mlp_sum_partials(partials, count, grad, b == 0, s)))
      return rc;
  }
  return check_err(derr, ws, s);
}
