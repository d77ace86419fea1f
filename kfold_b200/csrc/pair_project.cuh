// LayerNorm and projections of the pair track in one kernel (declarations).
#pragma once
#include "layernorm.cuh"

namespace kfb {

// The rows x (bf16, c channels; strides in elements) walked as (batch, o, n), o and n of the same extent.
struct PairRows {
  const void* x;
  const float *ln_w, *ln_b;
  long long s_n, s_o, s_b;
  int batch, n, c;
  float eps;
  int w_static;            // the weights were written before the launch before this one
};

// Triangle multiplication: ab[ch][b][o][n] = GLU(LN(x) . w_in) * mask (2 c channels, rows of `pitch`), gl (laid out as x) = LN(x) . w_gout;
// fold: the output projection's weights, folded along the way (or null).
bool trimul_pair_project_ok(const PairRows& r, const void* w_in, const void* w_gout, const void* ab, const void* gl, int dtype);
int launch_trimul_pair_project(cudaStream_t stream, const PairRows& r, const void* w_in, const void* w_gout, __nv_bfloat16* ab, int pitch,
                               __nv_bfloat16* gl, const unsigned char* mask, long long m_n, long long m_o, long long m_b, const LnFold* fold);

// Triangle attention of 128 channels: qkg [b][o][n][384], vt [b][o][128][pitch], bias [b][heads][o][pitch] (times bias_scale).
bool triatt_pair_project_ok(const PairRows& r, const void* w, int heads, int hdp, const void* qkg, const void* vt, const void* bias, int dtype);
int launch_triatt_pair_project(cudaStream_t stream, const PairRows& r, const void* w, int heads, __nv_bfloat16* qkg, __nv_bfloat16* vt,
                               __nv_bfloat16* bias, int pitch, float bias_scale);

}  // namespace kfb
