// Surrogate network: sizes, parameter/activation/gradient views and launchers (vpd_mlp.cu).
#pragma once

#include "vpd_internal.h"

#include <cuda_bf16.h>

namespace vpd {

constexpr int kMlpIn = 16;      // 10 features, zero padded
constexpr int kMlpHidden = 128;
constexpr int kMlpOut = 16;     // 7 targets, zero padded
constexpr int kMlpFeatures = 10;
constexpr int kMlpTargets = 7;
// flat parameter order: w1 [128][16], w2 [128][128], w3 [128][128], w4 [16][128] (row-major
// [out][in]), then b1 [128], b2 [128], b3 [128], b4 [16]
constexpr int64_t kMlpWeights = 128 * 16 + 128 * 128 * 2 + 16 * 128;
constexpr int64_t kMlpParams = kMlpWeights + 128 * 3 + 16;

struct MlpWeights {
  const __nv_bfloat16 *w1, *w2, *w3, *w4;
  const float *b1, *b2, *b3, *b4;
  // the four matrices, one after the other, stored as the operand tiles (mlp_tile_index) instead of row-major: a
  // block then stages all of them with one bulk copy
  bool tiled = false;
};
// Where the flat parameter i (< kMlpWeights) stands in tiled storage: in its matrix, core matrices of 8 rows x 8
// columns follow one another along a row.
__host__ __device__ inline int mlp_tile_index(int i) {
  const int base = i < 2048 ? 0 : (i < 2048 + 32768 ? 2048 + ((i - 2048) & ~16383) : 2048 + 32768);
  const int cols = i < 2048 ? 16 : 128, r = (i - base) / cols, c = (i - base) % cols;
  return base + (r >> 3) * 8 * cols + (c >> 3) * 64 + (r & 7) * 8 + (c & 7);
}

struct MlpGrads {  // FP32 accumulators, same shapes as the parameters
  float *w1, *w2, *w3, *w4, *b1, *b2, *b3, *b4;
};

__host__ __device__ inline MlpWeights mlp_weights(const __nv_bfloat16 *wb, const float *bias) {
  return MlpWeights{wb, wb + 2048, wb + 2048 + 16384, wb + 2048 + 32768,
                    bias, bias + 128, bias + 256, bias + 384};
}
__host__ __device__ inline MlpGrads mlp_grads(float *g) {
  return MlpGrads{g, g + 2048, g + 2048 + 16384, g + 2048 + 32768,
                  g + kMlpWeights, g + kMlpWeights + 128, g + kMlpWeights + 256, g + kMlpWeights + 384};
}

// out [B][16] = network(x [B][16]).
int mlp_forward(const MlpWeights &w, const float *x, int64_t B, float *out, unsigned *err, cudaStream_t s);

// One pass for the gradient of a batch: partial gradients of sum(out * gout) per 128-row block into `partials`
// (mlp_gradient_blocks(B) x kMlpParams floats). Rows are x's own, with gout given, or gathered from the training
// set with gout of the weighted MSE (MlpBatch).
int64_t mlp_gradient_blocks(int64_t B);
struct MlpBatch {
  const float *x, *gout;  // [B][16]; gout null: training rows, and the rest of this struct
  const float *target;    // [rows][16], row weight in column 15; x is then [rows][16] too
  int64_t rows, first;    // row r of the batch is row (mul (first + r) + add) % rows
  uint64_t mul, add;
  float *loss;            // += the batch's mean loss
};
int mlp_gradient_partials(const MlpWeights &w, const MlpBatch &batch, int64_t B, float *partials, unsigned *err,
                          cudaStream_t s);
// grad [kMlpParams] = the partials' sum in block order (first: from 0, else from what grad holds).
int mlp_sum_partials(const float *partials, int64_t blocks, float *grad, bool first, cudaStream_t s);
// The same sum taken straight into one Adam step on the parameters p (m, v: moments); wb: the weights' BF16 copy
// (tiled storage).
int mlp_adam(const float *partials, int64_t blocks, float *p, float *m, float *v, __nv_bfloat16 *wb, float lr,
             int step, cudaStream_t s);

}  // namespace vpd
