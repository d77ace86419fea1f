// HBM-bound normalisation kernels (declarations).
#pragma once
#include "common.cuh"

namespace kfb {

// Output row order of a (rows, n) shard written as the send buffer of a shard transpose: row (i, q * rows + j) goes to
// block q, [q][i][j].  rows == 0: rows keep their order.
struct RowPerm {
  int rows = 0;
  int n = 0;
};

// Weights of a projection with the LayerNorm before it folded in (see layernorm.cu): wf[n][k] = bf16(gamma[k] w[n][k]),
// s1[n] = sum_k wf[n][k], s0[n] = sum_k beta[k] w[n][k].
struct LnFold {
  const __nv_bfloat16* w;
  const float *gamma, *beta;
  __nv_bfloat16* wf;
  float *s1, *s0;
  int n, k;
};
int launch_ln_fold_weights(cudaStream_t stream, const LnFold& f);

// Row-wise LayerNorm, one warp per row, fp32 statistics.  in/out dtype KFB_BF16 or KFB_FP32.
int launch_layernorm(cudaStream_t stream, const void* x, void* y, const float* w, const float* b, long long rows, int c,
                     long long xs, long long ys, float eps, int in_dtype, int out_dtype, RowPerm perm = RowPerm());

// LayerNorm of bf16 rows (128 or 256 channels, contiguous, 16-byte aligned) and projection to heads <= 16 values in one pass: the pair
// bias.  w [heads][c] bf16; row (b, o, n) of batch x o_extent x n_extent, head h -> out + b s_b + o s_o + n s_n + h s_h (elements).
struct HeadsOut {
  __nv_bfloat16* out;
  long long s_b, s_o, s_n, s_h;
};
bool ln_heads_ok(const void* z, const void* w, int c, int heads, long long rows);
int launch_ln_heads(cudaStream_t stream, const void* z, const float* ln_w, const float* ln_b, const void* w, const HeadsOut& o, int batch,
                    int o_extent, int n_extent, int c, int heads, float eps);

// fp32 -> bf16 (round to nearest), n elements.
int launch_to_bf16(cudaStream_t stream, const float* x, __nv_bfloat16* y, long long n);

// Row-wise LayerNorm of fp32 rows written as the bf16 triple split [x0 . x1 . . x2] (six blocks of c columns,
// row stride 6c): the A operand of the fp32-accurate GEMMs.  With w == b == nullptr and `normalise` == 0 it only
// splits (used for operands that are not normalised).
int launch_layernorm_split(cudaStream_t stream, const float* x, __nv_bfloat16* y6, const float* w, const float* b, long long rows,
                           int c, long long xs, float eps, int normalise);
int launch_layernorm_split(cudaStream_t stream, const __nv_bfloat16* x, __nv_bfloat16* y6, const float* w, const float* b, long long rows,
                           int c, long long xs, float eps, int normalise);

// LayerNorm over channels of a CHANNEL-major tensor t[batch][c][pos] (pos contiguous, channel stride
// `chan_stride`, batch stride `batch_stride`), written POSITION-major y[batch*npos + pos][c] in bf16.
// `in_dtype` is the element type of t.  Used on the triangle contraction's output.
int launch_layernorm_cm(cudaStream_t stream, const void* t, __nv_bfloat16* y, const float* w, const float* b, int batch,
                        long long npos, int c, long long chan_stride, long long batch_stride, float eps, int in_dtype,
                        int split_out = 0);  // split_out: y is the [x0 . x1 . . x2] split, row stride 6c

// Adaptive LayerNorm: y[r] = sigmoid(g[s(r)]) * LN(a[r]) + v[s(r)], LN without affine, fp32 statistics.
// a, y: `rows` rows of c channels; gv: rows_s rows of [2c] (gate logits | shift), bf16.  Row r of a uses row
// (r / (samples * l)) * l + r % l of gv: the conditioning is shared by the `samples` diffusion samples.
// gv_static: a launch of this library lies between the last write of gv and this call.  gv_ld: elements between consecutive gv rows
// (0 = 2c), for rows that are slices of a wider table.  in_dtype KFB_FP32_PRECISE: a and gv fp32, y fp32 rows, or (out_dtype
// KFB_FP32_PRECISE) bf16 triple-split rows of 6c.
int launch_adaln(cudaStream_t stream, const void* a, void* y, const void* gv, long long rows, int c, int samples,
                 int l, float eps, int in_dtype, int out_dtype, long long gv_ld = 0, int gv_static = 0);
// ... of bf16 or fp32 rows with two sets of gates and shifts (bf16, rows gv_ld apart in either) into two bf16 tensors; one launch where the
// kernel takes the shape.
int launch_adaln_two(cudaStream_t stream, const void* a, void* y, void* y2, const void* gv, const void* gv2, long long rows, int c, int samples, int l,
                     float eps, int in_dtype, long long gv_ld, int gv_static);

// LayerNorm folded into the following GEMM (see layernorm.cu): per-position (mean, rstd) of a channel-major tensor.
int launch_cm_stats(cudaStream_t stream, const __nv_bfloat16* t, float2* stats, long long npos, int c, long long chan_stride,
                    float eps);

// LayerNorm over c (16, 32 or 64) channels and projection to nh values per position: x [npos][c], w [nh][c] of `dtype`
// (KFB_BF16 or KFB_FP32), y [nh][npos] of the same type.  normalise == 0: projection only.
int launch_window_bias(cudaStream_t stream, const void* x, const float* ln_w, const float* ln_b, const void* w, void* y,
                       long long npos, int c, int nh, float eps, int normalise, int dtype);

}  // namespace kfb
