// Token <-> atom maps around the atom transformers: a row gather (token features broadcast to their atoms) and a
// masked mean over the atoms of every token.  Both are pure data movement, HBM/L2-bound and tiny next to the
// transformers; they exist so that a caller never has to leave the library between the atom and the token level.
#include <cuda_bf16.h>

#include "ops_common.cuh"
#include "ptx.cuh"

namespace kfb {
namespace {

__device__ __forceinline__ float ld_f(const __nv_bfloat16* p) { return __bfloat162float(*p); }
__device__ __forceinline__ float ld_f(const float* p) { return *p; }
__device__ __forceinline__ void st_f(__nv_bfloat16* p, float v) { *p = __float2bfloat16_rn(v); }
__device__ __forceinline__ void st_f(float* p, float v) { *p = v; }
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <int VEC>
__device__ __forceinline__ void ld_vec(const float* p, float (&v)[VEC]) {
  if constexpr (VEC == 4) {
    const float4 f = *reinterpret_cast<const float4*>(p);
    v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
  } else {
    v[0] = *p;
  }
}
template <int VEC>
__device__ __forceinline__ void ld_vec(const __nv_bfloat16* p, float (&v)[VEC]) {
  if constexpr (VEC == 8) {
    const uint4 u = *reinterpret_cast<const uint4*>(p);
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      v[2 * i] = __uint_as_float(w[i] << 16);
      v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
  } else if constexpr (VEC == 4) {
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    v[0] = __uint_as_float(u.x << 16); v[1] = __uint_as_float(u.x & 0xffff0000u);
    v[2] = __uint_as_float(u.y << 16); v[3] = __uint_as_float(u.y & 0xffff0000u);
  } else {
    v[0] = ld_f(p);
  }
}

template <int VEC>
__device__ __forceinline__ void st_vec(float* p, const float (&v)[VEC]) {
  if constexpr (VEC == 4)
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  else
    *p = v[0];
}
template <int VEC>
__device__ __forceinline__ void st_vec(__nv_bfloat16* p, const float (&v)[VEC]) {
  if constexpr (VEC == 8)
    *reinterpret_cast<uint4*>(p) = make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
  else if constexpr (VEC == 4)
    *reinterpret_cast<uint2*>(p) = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]));
  else
    *p = __float2bfloat16_rn(v[0]);
}

// out[b][a][:] = x[b][index[b / index_div][a]][:] (+ addend[b][a][:]); one warp per atom row, 16-byte pieces when the
// types agree and nothing is added.  An index outside [0, n_token) yields a zero row (plus the addend) and records
// code 900 in the device status word instead of reading out of bounds.
static constexpr int kBadIndexCode = 900;
template <typename TX, typename TO>
__global__ void __launch_bounds__(256) tokens_to_atoms_kernel(const TX* x, const long long* index, const TO* addend, TO* out, long long rows,
                                                              int n_atom, int n_token, int d, int index_div) {
  grid_dependency_enter();
  const long long row = static_cast<long long>(blockIdx.x) * 8 + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int lane = threadIdx.x & 31;
  const long long b = row / n_atom;
  const int a = static_cast<int>(row - b * n_atom);
  const long long t = index[(b / index_div) * n_atom + a];
  const bool ok = t >= 0 && t < n_token;
  if (!ok && lane == 0) atomicCAS(&g_data_status, 0, kBadIndexCode);
  const TX* src = x + (b * n_token + (ok ? t : 0)) * d;
  TO* dst = out + row * d;
  if constexpr (sizeof(TX) == sizeof(TO)) {
    constexpr int kVec = 16 / sizeof(TX);
    if (addend == nullptr && d % kVec == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(out)) & 15) == 0) {
      for (int i0 = lane * kVec; i0 < d; i0 += 4 * 32 * kVec) {       // (four loads before the first store)
        uint4 piece[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int i = i0 + u * 32 * kVec;
          piece[u] = ok && i < d ? *reinterpret_cast<const uint4*>(src + i) : make_uint4(0, 0, 0, 0);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int i = i0 + u * 32 * kVec;
          if (i < d) *reinterpret_cast<uint4*>(dst + i) = piece[u];
        }
      }
      return;
    }
  }
  const TO* add = addend == nullptr ? nullptr : addend + row * d;
  for (int i0 = lane; i0 < d; i0 += 128) {
    float v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = min(i0 + 32 * u, d - 1);
      v[u] = (ok ? ld_f(src + i) : 0.f) + (add != nullptr ? ld_f(add + i) : 0.f);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (i0 + 32 * u < d) st_f(dst + i0 + 32 * u, v[u]);
  }
}

// out[row][:] = q[qrow][:] + sum_k w[:, k] r[row][k], fp32 out: the coordinate embedding added to the atom features
// (row r of out uses row (r / (samples * l)) * l + r % l of q and of the optional atom mask: the samples share them).
// One warp per row.
template <typename TQ>
__global__ void __launch_bounds__(256) coord_embed_kernel(const TQ* q, const float* r, const float* w, const unsigned char* mask, float* out,
                                                          long long rows, int c, int kc, int samples, int l) {
  grid_dependency_enter();
  const long long row = static_cast<long long>(blockIdx.x) * 8 + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int lane = threadIdx.x & 31;
  const long long qrow = (row / (static_cast<long long>(samples) * l)) * l + row % l;
  float rv[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  const bool keep = mask == nullptr || mask[qrow] != 0;   // coordinates of padding atoms count as zero
  for (int k = 0; k < kc; ++k) rv[k] = keep ? r[row * kc + k] : 0.f;
  for (int i0 = lane; i0 < c; i0 += 128) {
    float v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = min(i0 + 32 * u, c - 1);
      float acc = 0.f;
      for (int k = 0; k < kc; ++k) acc = fmaf(rv[k], w[i * kc + k], acc);   // same order as a dot product over k
      v[u] = ld_f(q + qrow * c + i) + acc;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (i0 + 32 * u < c) out[row * c + i0 + 32 * u] = v[u];
  }
}

// The same for 128 channels (the atom transformers') and KC coordinates: the general kernel asks for 12 weights 12 bytes apart and divides
// in 64 bits for every row; here a lane keeps the weights of its four neighbouring channels, and a warp goes from row to row, two at a time.
// 30 080 rows 35.5 -> 13.3 us between events.  Same bits.
template <typename TQ, int KC>
__global__ void __launch_bounds__(256) coord_embed128_kernel(const TQ* q, const float* r, const float* w, const unsigned char* mask, float* out,
                                                             unsigned rows, unsigned samples, unsigned l) {
  grid_dependency_enter();
  const unsigned lane = threadIdx.x & 31, warps = gridDim.x * 8;
  float wv[4][KC];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int k = 0; k < KC; ++k) wv[i][k] = w[(lane * 4 + i) * KC + k];
  for (unsigned row0 = blockIdx.x * 8 + (threadIdx.x >> 5); row0 < rows; row0 += 2 * warps) {
    float rv[2][KC], qv[2][4];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const unsigned row = min(row0 + j * warps, rows - 1), qrow = row / (samples * l) * l + row % l;
      const bool keep = mask == nullptr || mask[qrow] != 0;
#pragma unroll
      for (int k = 0; k < KC; ++k) rv[j][k] = keep ? r[static_cast<size_t>(row) * KC + k] : 0.f;
      ld_vec<4>(q + static_cast<size_t>(qrow) * 128 + lane * 4, qv[j]);
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      float v[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float acc = 0.f;
#pragma unroll
        for (int k = 0; k < KC; ++k) acc = fmaf(rv[j][k], wv[i][k], acc);
        v[i] = qv[j][i] + acc;
      }
      if (row0 + j * warps < rows)
        *reinterpret_cast<float4*>(out + static_cast<size_t>(row0 + j * warps) * 128 + lane * 4) = make_float4(v[0], v[1], v[2], v[3]);
    }
  }
}

// out[row][j] = sum_i LayerNorm(x[row])[i] w[j][i], j < n_out <= 8, everything fp32 after the load: the projection of the
// atom features to coordinate updates.  One warp per row; the row is re-read from L1 for the three passes.
template <typename T>
__global__ void __launch_bounds__(256) ln_project_kernel(const T* x, const float* ln_w, const float* ln_b, const float* w,
                                                         const unsigned char* mask, float* out, long long rows, int c, int n_out, float eps, int samples, int l) {
  grid_dependency_enter();
  const long long row = static_cast<long long>(blockIdx.x) * 8 + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int lane = threadIdx.x & 31;
  if (mask != nullptr && mask[(row / (static_cast<long long>(samples) * l)) * l + row % l] == 0) {
    if (lane < n_out) out[row * n_out + lane] = 0.f;   // padding atoms get a zero update
    return;
  }
  const T* xr = x + row * c;
  float s = 0.f;
  for (int i = lane; i < c; i += 32) s += ld_f(xr + i);
  const float mean = warp_sum(s) / static_cast<float>(c);
  float q = 0.f;
  for (int i = lane; i < c; i += 32) {
    const float dlt = ld_f(xr + i) - mean;
    q += dlt * dlt;
  }
  const float rstd = rsqrtf(warp_sum(q) / static_cast<float>(c) + eps);
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  for (int i = lane; i < c; i += 32) {
    const float xn = (ld_f(xr + i) - mean) * rstd * (ln_w != nullptr ? ln_w[i] : 1.f) + (ln_b != nullptr ? ln_b[i] : 0.f);
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (j < n_out) acc[j] = fmaf(xn, w[j * c + i], acc[j]);
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    if (j < n_out) {
      const float v = warp_sum(acc[j]);
      if (lane == 0) out[row * n_out + j] = v;
    }
  }
}

// The same for 128 channels and up to NOUT outputs: the general kernel loads a row three times and the weights again for every row; here a lane
// keeps the weights of its four channels (every 32nd, as there), and a warp goes from row to row, two at a time.  30 080 rows 29.0 -> 12.7 us between events.
// Same bits.
template <typename T, int NOUT>
__global__ void __launch_bounds__(256) ln_project128_kernel(const T* x, const float* ln_w, const float* ln_b, const float* w, const unsigned char* mask,
                                                            float* out, unsigned rows, float eps, unsigned samples, unsigned l) {
  grid_dependency_enter();
  const unsigned lane = threadIdx.x & 31, warps = gridDim.x * 8;
  float lw[4], lb[4], wv[NOUT][4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    lw[u] = ln_w != nullptr ? ln_w[lane + 32 * u] : 1.f;
    lb[u] = ln_b != nullptr ? ln_b[lane + 32 * u] : 0.f;
#pragma unroll
    for (int j = 0; j < NOUT; ++j) wv[j][u] = w[j * 128 + lane + 32 * u];
  }
  for (unsigned row0 = blockIdx.x * 8 + (threadIdx.x >> 5); row0 < rows; row0 += 2 * warps) {
    float v[2][4], acc[2][NOUT], sum[2], sq[2];
    bool keep[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const unsigned row = min(row0 + j * warps, rows - 1);
      keep[j] = mask == nullptr || mask[row / (samples * l) * l + row % l] != 0;   // padding atoms get a zero update
#pragma unroll
      for (int u = 0; u < 4; ++u) v[j][u] = ld_f(x + static_cast<size_t>(row) * 128 + lane + 32 * u);
      sum[j] = 0.f;
#pragma unroll
      for (int u = 0; u < 4; ++u) sum[j] += v[j][u];
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const float mean = warp_sum(sum[j]) / 128.f;
      sq[j] = 0.f;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        v[j][u] -= mean;
        sq[j] += v[j][u] * v[j][u];
      }
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const float rstd = rsqrtf(warp_sum(sq[j]) / 128.f + eps);
#pragma unroll
      for (int i = 0; i < NOUT; ++i) acc[j][i] = 0.f;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float xn = v[j][u] * rstd * lw[u] + lb[u];
#pragma unroll
        for (int i = 0; i < NOUT; ++i) acc[j][i] = fmaf(xn, wv[i][u], acc[j][i]);
      }
    }
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int i = 0; i < NOUT; ++i) acc[j][i] = warp_sum(acc[j][i]);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const unsigned row = row0 + j * warps;
      if (row >= rows) continue;
#pragma unroll
      for (int i = 0; i < NOUT; ++i)
        if (lane == static_cast<unsigned>(i)) out[static_cast<size_t>(row) * NOUT + i] = keep[j] ? acc[j][i] : 0.f;
    }
  }
}

// Per (index row, token): the first and last valid atom that maps to the token (first > last: none).  The mean below
// then scans only that range; it still tests every atom in it, so unsorted indices stay correct, and for the usual
// sorted atom order the range is just the token's own atoms.
__global__ void __launch_bounds__(256) token_range_init_kernel(int2* range, long long n) {
  grid_dependency_enter();
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < n) range[i] = make_int2(0x7fffffff, -1);
}
__global__ void __launch_bounds__(256) token_range_kernel(const long long* index, const unsigned char* mask, int2* range, long long total,
                                                          int n_atom, int n_token) {
  grid_dependency_enter();
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= total) return;
  const long long t = index[i];
  if (mask[i] == 0 || t < 0 || t >= n_token) return;
  const long long row = i / n_atom;
  const int a = static_cast<int>(i - row * n_atom);
  int* r = reinterpret_cast<int*>(range + row * n_token + t);
  atomicMin(r, a);
  atomicMax(r + 1, a);
}

// out[b][t][:] = mean over the atoms a of batch entry b with mask[a] and index[a] == t of x[b][a][:] (0 for a token
// without atoms); with `relu` the features pass through max(., 0) first.  One warp per (b, t, 32 * VEC channels): the warp scans
// the atom indices 32 at a time and adds the matching rows in atom order with fp32 accumulators, so the result does not depend on
// scheduling.  Latency-bound (a token has about eight atoms): rows are loaded four at a time, and the channels are spread over
// warps, where one warp walked 768 channels in three passes, a row at a time (55 us for 96 tokens).
template <typename T, int VEC>
__global__ void __launch_bounds__(256) atoms_to_tokens_kernel(const T* x, const long long* index, const unsigned char* mask, T* out,
                                                              long long rows, int n_atom, int n_token, int d, int index_div,
                                                              int relu, const int2* range, int pieces, int out_vec) {
  grid_dependency_enter();
  const long long item = static_cast<long long>(blockIdx.x) * 8 + (threadIdx.x >> 5);
  const long long row = item / pieces;
  if (row >= rows) return;
  const int lane = threadIdx.x & 31;
  const int col = (static_cast<int>(item - row * pieces) * 32 + lane) * VEC;
  const bool in = col < d;               // d is a multiple of VEC
  const long long b = row / n_token;
  const int t = static_cast<int>(row - b * n_token);
  const long long* idx = index + (b / index_div) * n_atom;
  const unsigned char* mk = mask + (b / index_div) * n_atom;
  const T* xb = x + b * n_atom * d + (in ? col : 0);
  int a_begin = 0, a_end = n_atom;
  if (range != nullptr) {
    const int2 rg = range[(b / index_div) * n_token + t];
    a_begin = rg.x <= rg.y ? rg.x : 0;
    a_end = rg.x <= rg.y ? rg.y + 1 : 0;
  }
  float acc[VEC];
#pragma unroll
  for (int i = 0; i < VEC; ++i) acc[i] = 0.f;
  int count = 0;
  for (int a0 = a_begin; a0 < a_end; a0 += 32) {
    const int a = a0 + lane;
    const bool hit = a < a_end && mk[a] != 0 && idx[a] == t;
    unsigned m = __ballot_sync(0xffffffffu, hit);
    count += __popc(m);
    while (m) {
      float v[4][VEC];
      bool some[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        some[u] = m != 0;
        const int j = some[u] ? __ffs(m) - 1 : 0;
        m &= m - 1;      // (zero stays zero)
        if (some[u]) ld_vec<VEC>(xb + static_cast<long long>(a0 + j) * d, v[u]);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (some[u]) {
#pragma unroll
          for (int i = 0; i < VEC; ++i) acc[i] += relu ? fmaxf(v[u][i], 0.f) : v[u][i];
        }
      }
    }
  }
  if (!in) return;
#pragma unroll
  for (int i = 0; i < VEC; ++i)
    // the reference divides the sum by the count (scatter_reduce "mean"): a division, not a multiplication
    acc[i] = count > 0 ? acc[i] / static_cast<float>(count) : 0.f;
  if (out_vec) {
    st_vec<VEC>(out + row * d + col, acc);
  } else {
#pragma unroll
    for (int i = 0; i < VEC; ++i) st_f(out + row * d + col + i, acc[i]);
  }
}

}  // namespace
}  // namespace kfb

using namespace kfb;

extern "C" {

KFB_API int kfb_tokens_to_atoms(const void* x, const long long* token_index, const void* addend, void* out, int batch,
                                int n_token, int n_atom, int d, int index_div, int x_dtype, int out_dtype, void* stream_) {
  KFB_CHECK_ARG(x && token_index && out, "tokens_to_atoms: null pointer");
  KFB_CHECK_ARG((x_dtype == KFB_BF16 || x_dtype == KFB_FP32) && (out_dtype == KFB_BF16 || out_dtype == KFB_FP32) &&
                    !(x_dtype == KFB_FP32 && out_dtype == KFB_BF16),
                "tokens_to_atoms: dtypes %d -> %d (bf16 -> bf16, bf16 -> fp32 or fp32 -> fp32)", x_dtype, out_dtype);
  KFB_CHECK_ARG(batch >= 1 && n_token >= 1 && n_atom >= 1 && d >= 1 && index_div >= 1 && batch % index_div == 0,
                "tokens_to_atoms: batch %d tokens %d atoms %d d %d index_div %d", batch, n_token, n_atom, d, index_div);
  cudaStream_t stream = as_stream(stream_);
  const long long rows = static_cast<long long>(batch) * n_atom;
  const unsigned blocks = static_cast<unsigned>((rows + 7) / 8);
  LaunchScope scope(stream, "tokens_to_atoms");
  using bf = __nv_bfloat16;
  if (x_dtype == KFB_BF16 && out_dtype == KFB_BF16)
    KFB_TRY(launch_kernel(stream, tokens_to_atoms_kernel<bf, bf>, blocks, 256, 0, static_cast<const bf*>(x), token_index,
        static_cast<const bf*>(addend),
                                                               static_cast<bf*>(out), rows, n_atom, n_token, d, index_div));
  else if (x_dtype == KFB_BF16)
    KFB_TRY(launch_kernel(stream, tokens_to_atoms_kernel<bf, float>, blocks, 256, 0, static_cast<const bf*>(x), token_index,
                                                                  static_cast<const float*>(addend), static_cast<float*>(out), rows,
                                                                  n_atom, n_token, d, index_div));
  else
    KFB_TRY(launch_kernel(stream, tokens_to_atoms_kernel<float, float>, blocks, 256, 0, static_cast<const float*>(x), token_index,
                                                                     static_cast<const float*>(addend), static_cast<float*>(out),
                                                                     rows, n_atom, n_token, d, index_div));
  KFB_CUDA(cudaGetLastError());
  return KFB_OK;
}

KFB_API size_t kfb_atoms_to_tokens_workspace_bytes(int batch, int n_token, int index_div) {
  return align_up(static_cast<size_t>(batch / (index_div > 0 ? index_div : 1)) * n_token * sizeof(int2), 256);
}

KFB_API int kfb_atoms_to_tokens(const void* x, const long long* token_index, const unsigned char* mask, void* out, void* workspace,
                                size_t workspace_bytes, int batch, int n_atom, int n_token, int d, int index_div, int relu,
                                int dtype, void* stream_) {
  KFB_CHECK_ARG(x && token_index && mask && out, "atoms_to_tokens: null pointer");
  KFB_CHECK_ARG(dtype == KFB_BF16 || dtype == KFB_FP32, "atoms_to_tokens: dtype %d (bf16 or fp32)", dtype);
  KFB_CHECK_ARG(batch >= 1 && n_token >= 1 && n_atom >= 1 && d >= 1 && index_div >= 1 && batch % index_div == 0,
                "atoms_to_tokens: batch %d tokens %d atoms %d d %d index_div %d", batch, n_token, n_atom, d, index_div);
  cudaStream_t stream = as_stream(stream_);
  const long long rows = static_cast<long long>(batch) * n_token;
  int2* range = nullptr;
  if (workspace != nullptr) {
    KFB_CHECK_ARG(workspace_bytes >= kfb_atoms_to_tokens_workspace_bytes(batch, n_token, index_div) &&
                      (reinterpret_cast<uintptr_t>(workspace) & 7) == 0,
                  "atoms_to_tokens: workspace too small or misaligned");
    range = static_cast<int2*>(workspace);
    const long long nr = static_cast<long long>(batch / index_div) * n_token, na = static_cast<long long>(batch / index_div) * n_atom;
    {
      LaunchScope scope(stream, "atoms_to_tokens_ranges");
      KFB_TRY(launch_kernel(stream, token_range_init_kernel, static_cast<unsigned>((nr + 255) / 256), 256, 0, range, nr));
    }
    {
      LaunchScope scope(stream, "atoms_to_tokens_ranges");
      KFB_TRY(launch_kernel(stream, token_range_kernel, static_cast<unsigned>((na + 255) / 256), 256, 0, token_index, mask, range, na, n_atom,
                            n_token));
    }
    KFB_CUDA(cudaGetLastError());
  }
  LaunchScope scope(stream, "atoms_to_tokens");
  // 16-byte pieces of bf16 where a row then needs fewer warps, 8-byte ones where its channels are whole fours; results by themselves where
  // they start between pieces.  5 x 768 tokens of eight atoms, us by pieces of 16 / 8 bytes: 768 channels 17.2 / 21.3, 136 9.4 / 10.7, 128
  // 9.4 / 6.7; single channels / 8 bytes: 124 12.8 / 6.6, 260 22.1 / 13.6.
  const bool x_ok = (reinterpret_cast<uintptr_t>(x) & 15) == 0;
  const int vec = x_ok && dtype == KFB_BF16 && d % 8 == 0 && d > 128 ? 8 : x_ok && d % 4 == 0 ? 4 : 1;
  const int out_vec = (reinterpret_cast<uintptr_t>(out) & (vec * (dtype == KFB_BF16 ? 2 : 4) - 1)) == 0;
  const int pieces = cdiv(d, 32 * vec);
  const unsigned blocks = static_cast<unsigned>((rows * pieces + 7) / 8);
  auto launch = [&](auto kernel, auto* xt, auto* ot) {
    return launch_kernel(stream, kernel, blocks, 256, 0, xt, token_index, mask, ot, rows, n_atom, n_token, d, index_div, relu, range, pieces, out_vec);
  };
  if (dtype == KFB_BF16) {
    using T = __nv_bfloat16;
    KFB_TRY(launch(vec == 8 ? atoms_to_tokens_kernel<T, 8> : vec == 4 ? atoms_to_tokens_kernel<T, 4> : atoms_to_tokens_kernel<T, 1>,
                   static_cast<const T*>(x), static_cast<T*>(out)));
  } else {
    KFB_TRY(launch(vec == 4 ? atoms_to_tokens_kernel<float, 4> : atoms_to_tokens_kernel<float, 1>, static_cast<const float*>(x),
                   static_cast<float*>(out)));
  }
  KFB_CUDA(cudaGetLastError());
  return KFB_OK;
}

KFB_API int kfb_coord_embed(const void* q, const float* r, const float* w, const unsigned char* mask, float* out, long long rows,
                            int c, int kc, int samples, int l, int q_dtype, void* stream_) {
  KFB_CHECK_ARG(q && r && w && out, "coord_embed: null pointer");
  KFB_CHECK_ARG(q_dtype == KFB_BF16 || q_dtype == KFB_FP32, "coord_embed: dtype %d (bf16 or fp32)", q_dtype);
  KFB_CHECK_ARG(rows >= 1 && c >= 1 && kc >= 1 && kc <= 8 && samples >= 1 && l >= 1 &&
                    rows % (static_cast<long long>(samples) * l) == 0,
                "coord_embed: rows %lld c %d coordinates %d samples %d l %d", rows, c, kc, samples, l);
  cudaStream_t stream = as_stream(stream_);
  const unsigned blocks = static_cast<unsigned>((rows + 7) / 8);
  LaunchScope scope(stream, "coord_embed");
  if (c == 128 && (kc == 3 || kc == 6) && rows < (1ll << 31) && ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(out)) & 15) == 0) {
    const unsigned few = rows < 16ll * 4 * sm_count() ? blocks : static_cast<unsigned>(4 * sm_count());
    auto launch = [&](auto kernel, auto* qt) {
      return launch_kernel(stream, kernel, few, 256, 0, qt, r, w, mask, out, static_cast<unsigned>(rows), static_cast<unsigned>(samples),
                           static_cast<unsigned>(l));
    };
    using bf = __nv_bfloat16;
    if (q_dtype == KFB_BF16) return launch(kc == 3 ? coord_embed128_kernel<bf, 3> : coord_embed128_kernel<bf, 6>, static_cast<const bf*>(q));
    return launch(kc == 3 ? coord_embed128_kernel<float, 3> : coord_embed128_kernel<float, 6>, static_cast<const float*>(q));
  }
  if (q_dtype == KFB_BF16)
    KFB_TRY(launch_kernel(stream, coord_embed_kernel<__nv_bfloat16>, blocks, 256, 0, static_cast<const __nv_bfloat16*>(q), r,
        w, mask, out, rows, c, kc,
                                                                   samples, l));
  else
    KFB_TRY(launch_kernel(stream, coord_embed_kernel<float>, blocks, 256, 0, static_cast<const float*>(q), r, w, mask, out,
        rows, c, kc, samples, l));
  KFB_CUDA(cudaGetLastError());
  return KFB_OK;
}

KFB_API int kfb_ln_project(const void* x, const float* ln_w, const float* ln_b, const float* w, const unsigned char* mask,
                           float* out, long long rows, int c, int n_out, float eps, int samples, int l, int dtype, void* stream_) {
  KFB_CHECK_ARG(x && w && out, "ln_project: null pointer");
  KFB_CHECK_ARG(dtype == KFB_BF16 || dtype == KFB_FP32, "ln_project: dtype %d (bf16 or fp32)", dtype);
  KFB_CHECK_ARG(rows >= 1 && c >= 1 && n_out >= 1 && n_out <= 8, "ln_project: rows %lld c %d outputs %d (at most 8)", rows, c, n_out);
  if (mask == nullptr) samples = l = 1;
  KFB_CHECK_ARG(samples >= 1 && l >= 1 && rows % (static_cast<long long>(samples) * l) == 0,
                "ln_project: rows %lld are not a multiple of samples %d x l %d", rows, samples, l);
  cudaStream_t stream = as_stream(stream_);
  const unsigned blocks = static_cast<unsigned>((rows + 7) / 8);
  LaunchScope scope(stream, "ln_project");
  if (c == 128 && n_out == 3 && rows < (1ll << 31)) {
    const unsigned few = rows < 16ll * 4 * sm_count() ? blocks : static_cast<unsigned>(4 * sm_count());
    auto launch = [&](auto kernel, auto* xt) {
      return launch_kernel(stream, kernel, few, 256, 0, xt, ln_w, ln_b, w, mask, out, static_cast<unsigned>(rows), eps, static_cast<unsigned>(samples),
                           static_cast<unsigned>(l));
    };
    if (dtype == KFB_BF16) return launch(ln_project128_kernel<__nv_bfloat16, 3>, static_cast<const __nv_bfloat16*>(x));
    return launch(ln_project128_kernel<float, 3>, static_cast<const float*>(x));
  }
  if (dtype == KFB_BF16)
    KFB_TRY(launch_kernel(stream, ln_project_kernel<__nv_bfloat16>, blocks, 256, 0, static_cast<const __nv_bfloat16*>(x),
        ln_w, ln_b, w, mask, out, rows,
                                                                  c, n_out, eps, samples, l));
  else
    KFB_TRY(launch_kernel(stream, ln_project_kernel<float>, blocks, 256, 0, static_cast<const float*>(x), ln_w, ln_b, w,
        mask, out, rows, c, n_out, eps,
                                                         samples, l));
  KFB_CUDA(cudaGetLastError());
  return KFB_OK;
}

}  // extern "C"
