// LayerNorm kernels.  Pure HBM traffic: every element is read once and written once,
// statistics are taken in fp32 with warp-shuffle reductions (two-pass: mean, then
// variance of the centred values, which is what torch's layer_norm computes).
#include "layernorm.cuh"

#include "gemm.cuh"  // part_a

#include <type_traits>

namespace kfb {

template <typename T>
__device__ __forceinline__ float2 load2(const T* p);
template <>
__device__ __forceinline__ float2 load2<float>(const float* p) {
  return *reinterpret_cast<const float2*>(p);
}
template <>
__device__ __forceinline__ float2 load2<__nv_bfloat16>(const __nv_bfloat16* p) {
  return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p));
}
__device__ __forceinline__ float load1(const float* p) { return *p; }
__device__ __forceinline__ float load1(const __nv_bfloat16* p) { return __bfloat162float(*p); }
__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
}
template <typename T>
__device__ __forceinline__ void store2(T* p, float a, float b);
template <>
__device__ __forceinline__ void store2<float>(float* p, float a, float b) {
  *reinterpret_cast<float2*>(p) = make_float2(a, b);
}
template <>
__device__ __forceinline__ void store2<__nv_bfloat16>(__nv_bfloat16* p, float a, float b) {
  *reinterpret_cast<__nv_bfloat162*>(p) = __floats2bfloat162_rn(a, b);
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// One warp per row; lane l holds channel pairs (l + 32 g) * 2, g < G.
template <typename TI, typename TO, int G, bool PERM>
__global__ void __launch_bounds__(256) layernorm_rows_kernel(const TI* x, TO* y, const float* w, const float* b, long long rows, int c,
                                                             long long xs, long long ys, float eps, RowPerm perm) {
  grid_dependency_enter();
  const int lane = threadIdx.x & 31;
  const long long warps_per_grid = static_cast<long long>(gridDim.x) * (blockDim.x >> 5);
  for (long long row = static_cast<long long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5); row < rows;
       row += warps_per_grid) {
    const TI* xr = x + row * xs;
    float2 v[G];
    float s = 0.f;
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const int ch = (lane + 32 * g) * 2;
      v[g] = ch < c ? load2<TI>(xr + ch) : make_float2(0.f, 0.f);
      s += v[g].x + v[g].y;
    }
    const float mean = warp_sum(s) / static_cast<float>(c);
    float q = 0.f;
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const int ch = (lane + 32 * g) * 2;
      if (ch < c) {
        v[g].x -= mean;
        v[g].y -= mean;
        q += v[g].x * v[g].x + v[g].y * v[g].y;
      }
    }
    const float rstd = rsqrtf(warp_sum(q) / static_cast<float>(c) + eps);
    long long orow = row;
    if (PERM) {   // (i, q, j) -> (q, i, j): the send buffer of a shard transpose, one block per destination rank
      const long long i = row / perm.n;
      const int rest = static_cast<int>(row - i * perm.n);
      const int q = rest / perm.rows;
      orow = (static_cast<long long>(q) * perm.rows + i) * perm.rows + (rest - q * perm.rows);
    }
    TO* yr = y + orow * ys;
    // (scale and offset of the whole row before its first store: behind one, a load waits for it)
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const int ch = (lane + 32 * g) * 2;
      if (ch < c) {
        const float2 ww = w != nullptr ? *reinterpret_cast<const float2*>(w + ch) : make_float2(1.f, 1.f);
        const float2 bb = b != nullptr ? *reinterpret_cast<const float2*>(b + ch) : make_float2(0.f, 0.f);
        v[g].x = fmaf(v[g].x * rstd, ww.x, bb.x);
        v[g].y = fmaf(v[g].y * rstd, ww.y, bb.y);
      }
    }
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const int ch = (lane + 32 * g) * 2;
      if (ch < c) store2<TO>(yr + ch, v[g].x, v[g].y);
    }
  }
}

// Folded weights (see LnFold), kFoldRows rows per block of 256 threads: W' rounded to bf16, s1 of the rounded values.  (A launch of 3.3 us,
// whatever the size; pair_project_kernel does the same beside its projections.)
constexpr int kFoldRows = 8;
__device__ __forceinline__ void ln_fold_rows(const LnFold& f, int block) {
  constexpr int kPer = kFoldRows / 2;                       // rows of each half of the block
  const int half = threadIdx.x >> 7, tid = threadIdx.x & 127, w4 = tid >> 5;
  const int n0 = block * kFoldRows + half * kPer;
  float a1[kPer], a0[kPer];
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    a1[j] = a0[j] = 0.f;
    const long long row = static_cast<long long>(min(n0 + j, f.n - 1)) * f.k;
    for (int i = tid; i < f.k; i += 128) {
      const float wv = __bfloat162float(f.w[row + i]);
      const __nv_bfloat16 wr = __float2bfloat16_rn(wv * (f.gamma != nullptr ? f.gamma[i] : 1.0f));
      if (n0 + j < f.n) f.wf[row + i] = wr;
      a1[j] += __bfloat162float(wr);
      a0[j] += (f.beta != nullptr ? f.beta[i] : 0.0f) * wv;
    }
  }
  __shared__ float red[2][kFoldRows][4];
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const float r1 = warp_sum(a1[j]), r0 = warp_sum(a0[j]);
    if ((tid & 31) == 0) {
      red[0][half * kPer + j][w4] = r1;
      red[1][half * kPer + j][w4] = r0;
    }
  }
  __syncthreads();
  const int j = threadIdx.x % kFoldRows, n = block * kFoldRows + j;
  if (threadIdx.x < 2 * kFoldRows && n < f.n) {
    const float* r = red[threadIdx.x / kFoldRows][j];
    (threadIdx.x < kFoldRows ? f.s1 : f.s0)[n] = (r[0] + r[1]) + (r[2] + r[3]);
  }
}
__global__ void __launch_bounds__(256) ln_fold_weights_kernel(const LnFold f) {
  grid_dependency_enter();
  ln_fold_rows(f, blockIdx.x);
}
int launch_ln_fold_weights(cudaStream_t stream, const LnFold& f) {
  KFB_CHECK_ARG(f.n > 0 && f.k > 0, "ln_fold_weights: n %d k %d", f.n, f.k);
  LaunchScope scope(stream, "layernorm_fold_weights");
  return launch_kernel(stream, ln_fold_weights_kernel, cdiv(f.n, kFoldRows), 256, 0, f);
}

// The pair track's shape: 128 bf16 channels, contiguous rows.  A row is 256 bytes = 16 lanes x 16 bytes, so a warp takes two
// rows per step and two steps per iteration: four rows (1 KB) in flight per warp, 16-byte loads and stores, the statistics
// reduced over the 16 lanes of a row.  Same arithmetic as layernorm_rows_kernel (two passes, fp32).
__global__ void __launch_bounds__(256) layernorm_c128_bf16_kernel(const __nv_bfloat16* x, __nv_bfloat16* y, const float* w, const float* b,
                                                                  long long rows, float eps) {
  constexpr int LANES = 16, STEPS = 2, C = LANES * 8, kRows = 32 / LANES;
  grid_dependency_enter();
  const int lane = threadIdx.x & 31;
  const int sub = lane % LANES;              // 16-byte chunk of the row
  const int half = lane / LANES;             // which of the step's rows
  float g[8], o[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    g[i] = w != nullptr ? w[sub * 8 + i] : 1.0f;
    o[i] = b != nullptr ? b[sub * 8 + i] : 0.0f;
  }
  const long long warps = static_cast<long long>(gridDim.x) * (blockDim.x >> 5);
  const long long warp_id = static_cast<long long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  for (long long base = warp_id * (kRows * STEPS); base < rows; base += warps * (kRows * STEPS)) {
    uint4 raw[STEPS];
    bool live[STEPS];
#pragma unroll
    for (int s = 0; s < STEPS; ++s) {
      const long long row = base + s * kRows + half;
      live[s] = row < rows;
      raw[s] = live[s] ? *reinterpret_cast<const uint4*>(x + row * C + sub * 8) : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int s = 0; s < STEPS; ++s) {
      const uint32_t wv[4] = {raw[s].x, raw[s].y, raw[s].z, raw[s].w};
      float v[8];
      float sum = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        v[2 * i] = __uint_as_float(wv[i] << 16);
        v[2 * i + 1] = __uint_as_float(wv[i] & 0xffff0000u);
        sum += v[2 * i] + v[2 * i + 1];
      }
#pragma unroll
      for (int m = LANES / 2; m > 0; m >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, m);
      const float mean = sum * (1.0f / C);
      float sq = 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        v[i] -= mean;
        sq = fmaf(v[i], v[i], sq);
      }
#pragma unroll
      for (int m = LANES / 2; m > 0; m >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, m);
      const float rstd = rsqrtf(sq * (1.0f / C) + eps);
      uint4 out;
      uint32_t* ov = reinterpret_cast<uint32_t*>(&out);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const __nv_bfloat162 pr = __floats2bfloat162_rn(fmaf(v[2 * i] * rstd, g[2 * i], o[2 * i]),
                                                        fmaf(v[2 * i + 1] * rstd, g[2 * i + 1], o[2 * i + 1]));
        ov[i] = *reinterpret_cast<const uint32_t*>(&pr);
      }
      const long long row = base + s * kRows + half;
      if (live[s]) *reinterpret_cast<uint4*>(y + row * C + sub * 8) = out;
    }
  }
}

// 256 bf16 channels, contiguous rows: layernorm_rows_kernel's lane layout, expressions and bits, with the weights kept in registers
// and four rows in flight per warp.  That kernel, one row at a time with the weights fetched for each, took 150 us for 768 x 768
// rows; this one 130 (92 at the memory's rate; 16-byte accesses gave 96, but another order of summation: a last-bit difference that
// four blocks of bf16 rounding turn into 0.8 % of the result).
constexpr int kC256Rows = 4;
__global__ void __launch_bounds__(256) layernorm_c256_bf16_kernel(const __nv_bfloat16* x, __nv_bfloat16* y, const float* w, const float* b,
                                                                  long long rows, float eps) {
  constexpr int G = 4, C = 256;
  grid_dependency_enter();
  const int lane = threadIdx.x & 31;
  float2 ww[G], bb[G];
#pragma unroll
  for (int g = 0; g < G; ++g) {
    ww[g] = w != nullptr ? *reinterpret_cast<const float2*>(w + (lane + 32 * g) * 2) : make_float2(1.f, 1.f);
    bb[g] = b != nullptr ? *reinterpret_cast<const float2*>(b + (lane + 32 * g) * 2) : make_float2(0.f, 0.f);
  }
  const long long warps = static_cast<long long>(gridDim.x) * (blockDim.x >> 5);
  const long long warp_id = static_cast<long long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  for (long long base = warp_id * kC256Rows; base < rows; base += warps * kC256Rows) {
    float2 v[kC256Rows][G];
#pragma unroll
    for (int r = 0; r < kC256Rows; ++r) {
      const __nv_bfloat16* xr = x + (base + r < rows ? base + r : rows - 1) * C;
#pragma unroll
      for (int g = 0; g < G; ++g) v[r][g] = load2<__nv_bfloat16>(xr + (lane + 32 * g) * 2);
    }
#pragma unroll
    for (int r = 0; r < kC256Rows; ++r) {
      float s = 0.f;
#pragma unroll
      for (int g = 0; g < G; ++g) s += v[r][g].x + v[r][g].y;
      const float mean = warp_sum(s) / static_cast<float>(C);
      float q = 0.f;
#pragma unroll
      for (int g = 0; g < G; ++g) {
        v[r][g].x -= mean;
        v[r][g].y -= mean;
        q += v[r][g].x * v[r][g].x + v[r][g].y * v[r][g].y;
      }
      const float rstd = rsqrtf(warp_sum(q) / static_cast<float>(C) + eps);
      if (base + r >= rows) break;
      __nv_bfloat16* yr = y + (base + r) * C;
#pragma unroll
      for (int g = 0; g < G; ++g) {
        store2<__nv_bfloat16>(yr + (lane + 32 * g) * 2, fmaf(v[r][g].x * rstd, ww[g].x, bb[g].x), fmaf(v[r][g].y * rstd, ww[g].y, bb[g].y));
      }
    }
  }
}

template <typename TI, typename TO, int G>
static int launch_rows(cudaStream_t stream, const void* x, void* y, const float* w, const float* b, long long rows, int c,
                       long long xs, long long ys, float eps, RowPerm perm) {
  const int warps = 8;
  long long blocks = (rows + warps - 1) / warps;
  const long long cap = static_cast<long long>(sm_count()) * 16;
  if (blocks > cap) blocks = cap;
  LaunchScope scope(stream, "layernorm_rows");
  if (perm.rows) {
    if constexpr (std::is_same<TO, __nv_bfloat16>::value) {   // the exchange order is only ever written in bf16
      KFB_TRY(launch_kernel(stream, layernorm_rows_kernel<TI, TO, G, true>, static_cast<unsigned>(blocks), warps * 32, 0,
          static_cast<const TI*>(x), static_cast<TO*>(y), w, b, rows, c, xs, ys, eps, perm));
    } else {
      set_error("layernorm: the exchange order is written in bf16 only");
      return KFB_ERR_UNSUPPORTED;
    }
  } else {
    KFB_TRY(launch_kernel(stream, layernorm_rows_kernel<TI, TO, G, false>, static_cast<unsigned>(blocks), warps * 32, 0,
        static_cast<const TI*>(x), static_cast<TO*>(y), w, b, rows, c, xs, ys, eps, perm));
  }
  KFB_CUDA(cudaGetLastError());
  return KFB_OK;
}

template <typename TI, typename TO>
static int dispatch_g(cudaStream_t stream, const void* x, void* y, const float* w, const float* b, long long rows, int c,
                      long long xs, long long ys, float eps, RowPerm perm) {
  const int g = cdiv(c, 64);
  if (g <= 1) return launch_rows<TI, TO, 1>(stream, x, y, w, b, rows, c, xs, ys, eps, perm);
  if (g <= 2) return launch_rows<TI, TO, 2>(stream, x, y, w, b, rows, c, xs, ys, eps, perm);
  if (g <= 4) return launch_rows<TI, TO, 4>(stream, x, y, w, b, rows, c, xs, ys, eps, perm);
  if (g <= 6) return launch_rows<TI, TO, 6>(stream, x, y, w, b, rows, c, xs, ys, eps, perm);
  if (g <= 12) return launch_rows<TI, TO, 12>(stream, x, y, w, b, rows, c, xs, ys, eps, perm);
  if (g <= 16) return launch_rows<TI, TO, 16>(stream, x, y, w, b, rows, c, xs, ys, eps, perm);
  set_error("layernorm: channel count %d above 1024 is not supported", c);
  return KFB_ERR_UNSUPPORTED;
}

int launch_layernorm(cudaStream_t stream, const void* x, void* y, const float* w, const float* b, long long rows, int c,
                     long long xs, long long ys, float eps, int in_dtype, int out_dtype, RowPerm perm) {
  KFB_CHECK_ARG(rows >= 0 && c > 0 && c % 2 == 0, "layernorm: rows %lld, channels %d (must be even)", rows, c);
  KFB_CHECK_ARG(perm.rows == 0 || (perm.n % perm.rows == 0 && rows == static_cast<long long>(perm.rows) * perm.n),
                "layernorm: exchange order needs a (%d, %d) shard, got %lld rows", perm.rows, perm.n, rows);
  KFB_CHECK_ARG(xs % 2 == 0 && ys % 2 == 0, "layernorm: row strides must be even");
  if (rows == 0) return KFB_OK;
  if (in_dtype == KFB_BF16 && out_dtype == KFB_BF16 && (c == 128 || c == 256) && xs == c && ys == c && perm.rows == 0 &&
      ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15) == 0) {
    long long blocks = (rows + 31) / 32;      // 8 warps x 4 rows per iteration
    const long long cap = static_cast<long long>(sm_count()) * 16;
    if (blocks > cap) blocks = cap;
    LaunchScope scope(stream, "layernorm_rows");
    KFB_TRY(launch_kernel(stream, c == 128 ? layernorm_c128_bf16_kernel : layernorm_c256_bf16_kernel,
                          static_cast<unsigned>(blocks), 256, 0, static_cast<const __nv_bfloat16*>(x),
                          static_cast<__nv_bfloat16*>(y), w, b, rows, eps));
    KFB_CUDA(cudaGetLastError());
    return KFB_OK;
  }
  if (in_dtype == KFB_BF16 && out_dtype == KFB_BF16)
    return dispatch_g<__nv_bfloat16, __nv_bfloat16>(stream, x, y, w, b, rows, c, xs, ys, eps, perm);
  if (in_dtype == KFB_FP32 && out_dtype == KFB_BF16)
    return dispatch_g<float, __nv_bfloat16>(stream, x, y, w, b, rows, c, xs, ys, eps, perm);
  if (in_dtype == KFB_FP32 && out_dtype == KFB_FP32)
    return dispatch_g<float, float>(stream, x, y, w, b, rows, c, xs, ys, eps, perm);
  if (in_dtype == KFB_BF16 && out_dtype == KFB_FP32)
    return dispatch_g<__nv_bfloat16, float>(stream, x, y, w, b, rows, c, xs, ys, eps, perm);
  set_error("layernorm: bad dtype");
  return KFB_ERR_INVALID_ARGUMENT;
}

// LayerNorm and projection to at most 16 heads.  What bounds it: the rows, read once; written normalised and read again by a GEMM of 16
// columns they had moved three times.  A warp takes 16 rows: four lanes share a row (a lane has 8 channels of every 32, 16-byte loads),
// the statistics take two shuffles, and the normalised bf16 pairs are already the A fragments of 16 x 8 x 16 products -- a product does
// not care which channel is called k, so the weights' fragments follow the lanes' channels.  (Sixteen columns are too few for a tile of
// the tensor memory kernels to be anything but latency; the products are 5 % of the time here.)
// 768 x 768 rows of 128 channels, between CUDA events: LayerNorm 56 + GEMM 44 us -> 54 in one launch; 400 x 400 of 256: 45 + 28 -> 43.
// (The unpacked rows live in registers, 128 and 254 of them; held to 64 or 80 they spill: 72 us.)
template <int C>
__global__ void __launch_bounds__(256) ln_heads_kernel(const __nv_bfloat16* z, const float* ln_w, const float* ln_b,
                                                       const __nv_bfloat16* w, const HeadsOut out, int rows, int o_extent, int n_extent,
                                                       int heads, float eps) {
  constexpr int Q = C / 32, kWLd = C + 8;       // (rows of the weights 16 bytes off: eight of them cover the banks)
  __shared__ __align__(16) __nv_bfloat16 s_w[16 * kWLd];
  __shared__ __align__(16) float s_g[C], s_b[C];
  grid_dependency_enter();
  for (int i = threadIdx.x; i < 16 * (C / 8); i += 256) {
    const int h = i / (C / 8), ch = (i % (C / 8)) * 8;
    *reinterpret_cast<uint4*>(s_w + h * kWLd + ch) = h < heads ? *reinterpret_cast<const uint4*>(w + h * C + ch) : make_uint4(0, 0, 0, 0);
  }
  for (int i = threadIdx.x; i < C; i += 256) {
    s_g[i] = ln_w != nullptr ? ln_w[i] : 1.0f;
    s_b[i] = ln_b != nullptr ? ln_b[i] : 0.0f;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int warps = gridDim.x * 8;
  for (int base = (blockIdx.x * 8 + (threadIdx.x >> 5)) * 16; base < rows; base += warps * 16) {
    uint4 raw[2][Q];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const __nv_bfloat16* zr = z + static_cast<long long>(min(base + g + 8 * r, rows - 1)) * C + t * 8;
#pragma unroll
      for (int q = 0; q < Q; ++q) raw[r][q] = *reinterpret_cast<const uint4*>(zr + q * 32);
    }
    float mean[2], rstd[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      float s = 0.f;
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const uint32_t u[4] = {raw[r][q].x, raw[r][q].y, raw[r][q].z, raw[r][q].w};
#pragma unroll
        for (int i = 0; i < 4; ++i) s += __uint_as_float(u[i] << 16) + __uint_as_float(u[i] & 0xffff0000u);
      }
      s += __shfl_xor_sync(0xffffffffu, s, 1);
      s += __shfl_xor_sync(0xffffffffu, s, 2);
      mean[r] = s * (1.0f / C);
      float v = 0.f;
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const uint32_t u[4] = {raw[r][q].x, raw[r][q].y, raw[r][q].z, raw[r][q].w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float d0 = __uint_as_float(u[i] << 16) - mean[r], d1 = __uint_as_float(u[i] & 0xffff0000u) - mean[r];
          v = fmaf(d0, d0, v);
          v = fmaf(d1, d1, v);
        }
      }
      v += __shfl_xor_sync(0xffffffffu, v, 1);
      v += __shfl_xor_sync(0xffffffffu, v, 2);
      rstd[r] = rsqrtf(v * (1.0f / C) + eps);
    }
    float acc[2][4] = {};       // [heads 0-7, 8-15][row g: heads 2t, 2t + 1; row g + 8: the same]
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int ch = q * 32 + t * 8;
      uint32_t a[2][4];         // the rows' normalised pairs
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 gg = *reinterpret_cast<const float2*>(s_g + ch + 2 * i), bb = *reinterpret_cast<const float2*>(s_b + ch + 2 * i);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const uint32_t u = i == 0 ? raw[r][q].x : i == 1 ? raw[r][q].y : i == 2 ? raw[r][q].z : raw[r][q].w;
          const __nv_bfloat162 pr = __floats2bfloat162_rn(fmaf((__uint_as_float(u << 16) - mean[r]) * rstd[r], gg.x, bb.x),
                                                          fmaf((__uint_as_float(u & 0xffff0000u) - mean[r]) * rstd[r], gg.y, bb.y));
          a[r][i] = *reinterpret_cast<const uint32_t*>(&pr);
        }
      }
#pragma unroll
      for (int h8 = 0; h8 < 2; ++h8) {
        const uint4 wv = *reinterpret_cast<const uint4*>(s_w + (h8 * 8 + g) * kWLd + ch);
        const uint32_t wb[4] = {wv.x, wv.y, wv.z, wv.w};
#pragma unroll
        for (int k = 0; k < 4; k += 2)
          asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
              : "+f"(acc[h8][0]), "+f"(acc[h8][1]), "+f"(acc[h8][2]), "+f"(acc[h8][3])
              : "r"(a[0][k]), "r"(a[1][k]), "r"(a[0][k + 1]), "r"(a[1][k + 1]), "r"(wb[k]), "r"(wb[k + 1]));
      }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int row = base + g + 8 * r;
      if (row >= rows) break;
      const int n = row % n_extent, rest = row / n_extent;
      __nv_bfloat16* dst = out.out + static_cast<long long>(rest / o_extent) * out.s_b + static_cast<long long>(rest % o_extent) * out.s_o +
                           static_cast<long long>(n) * out.s_n;
#pragma unroll
      for (int h8 = 0; h8 < 2; ++h8)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int h = h8 * 8 + 2 * t + i;
          if (h < heads) dst[h * out.s_h] = __float2bfloat16_rn(acc[h8][2 * r + i]);
        }
    }
  }
}

bool ln_heads_ok(const void* z, const void* w, int c, int heads, long long rows) {
  return (c == 128 || c == 256) && heads <= 16 && rows > 0 && rows < (1ll << 31) - 64 &&
         ((reinterpret_cast<uintptr_t>(z) | reinterpret_cast<uintptr_t>(w)) & 15) == 0;
}
int launch_ln_heads(cudaStream_t stream, const void* z, const float* ln_w, const float* ln_b, const void* w, const HeadsOut& o, int batch,
                    int o_extent, int n_extent, int c, int heads, float eps) {
  const long long rows = static_cast<long long>(batch) * o_extent * n_extent;
  KFB_CHECK_ARG(ln_heads_ok(z, w, c, heads, rows), "ln_heads: c %d heads %d rows %lld", c, heads, rows);
  long long blocks = (rows + 127) / 128;
  const long long cap = static_cast<long long>(sm_count()) * 8;
  if (blocks > cap) blocks = cap;
  LaunchScope scope(stream, "pair_bias_proj");
  return launch_kernel(stream, c == 128 ? ln_heads_kernel<128> : ln_heads_kernel<256>, static_cast<unsigned>(blocks), 256, 0,
                       static_cast<const __nv_bfloat16*>(z), ln_w, ln_b, static_cast<const __nv_bfloat16*>(w), o, static_cast<int>(rows), o_extent,
                       n_extent, heads, eps);
}

// fp32 -> bf16 conversion, eight elements per thread (HBM-bound; the conditioning rows of a stack: one small launch).
__global__ void __launch_bounds__(256) to_bf16_kernel(const float* x, __nv_bfloat16* y, long long n) {
  grid_dependency_enter();
  const long long i = (static_cast<long long>(blockIdx.x) * 256 + threadIdx.x) * 8;
  if (i + 8 <= n) {
    const float4 a = *reinterpret_cast<const float4*>(x + i), b = *reinterpret_cast<const float4*>(x + i + 4);
    const __nv_bfloat162 p[4] = {__floats2bfloat162_rn(a.x, a.y), __floats2bfloat162_rn(a.z, a.w), __floats2bfloat162_rn(b.x, b.y),
                                 __floats2bfloat162_rn(b.z, b.w)};
    *reinterpret_cast<uint4*>(y + i) = *reinterpret_cast<const uint4*>(p);
  } else {
    for (long long k = i; k < n; ++k) y[k] = __float2bfloat16_rn(x[k]);
  }
}

int launch_to_bf16(cudaStream_t stream, const float* x, __nv_bfloat16* y, long long n) {
  if (n <= 0) return KFB_OK;
  KFB_CHECK_ARG(((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15) == 0, "to_bf16: pointers must be 16-byte aligned");
  LaunchScope scope(stream, "to_bf16");
  KFB_TRY(launch_kernel(stream, to_bf16_kernel, static_cast<unsigned>((n + 2047) / 2048), 256, 0, x, y, n));
  KFB_CUDA(cudaGetLastError());
  return KFB_OK;
}

// ------------------------------------------------------------------------------------------------
// fp32-accurate mode: LayerNorm (or a plain copy) of fp32 rows, written as the bf16 triple split.
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ void split3_store(__nv_bfloat16* y6, int c, int ch, float v) {
  const __nv_bfloat16 x0 = __float2bfloat16_rn(v);
  const float r1 = v - __bfloat162float(x0);
  const __nv_bfloat16 x1 = __float2bfloat16_rn(r1);
  const __nv_bfloat16 x2 = __float2bfloat16_rn(r1 - __bfloat162float(x1));
  y6[part_a(0) * c + ch] = x0;
  y6[part_a(1) * c + ch] = x1;
  y6[part_a(2) * c + ch] = x2;
}

// One warp per row, G pieces of 128 channels held in registers: four channels of a lane per load and per part's store.
// HBM-bound; 25 600 rows of 128 float32 channels 13 -> 6 us against the form below, which reads a row three times, channel by
// channel, and remains for rows that are not whole aligned pieces of four.
template <typename TI, int G>
__global__ void __launch_bounds__(256) layernorm_split_vec_kernel(const TI* x, __nv_bfloat16* y6, const float* w, const float* b,
                                                                  long long rows, int c, long long xs, float eps, int normalise) {
  grid_dependency_enter();
  const int lane = threadIdx.x & 31;
  const long long warps_per_grid = static_cast<long long>(gridDim.x) * (blockDim.x >> 5);
  for (long long row = static_cast<long long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5); row < rows;
       row += warps_per_grid) {
    const TI* xr = x + row * xs;
    float v[G][4];
    float s = 0.f;
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const int ch = (lane + 32 * g) * 4;
      v[g][0] = v[g][1] = v[g][2] = v[g][3] = 0.f;
      if (ch < c) {
        const float4 f = load4(xr + ch);
        v[g][0] = f.x; v[g][1] = f.y; v[g][2] = f.z; v[g][3] = f.w;
      }
      s += (v[g][0] + v[g][1]) + (v[g][2] + v[g][3]);
    }
    float mean = 0.f, rstd = 1.f;
    if (normalise) {
      mean = warp_sum(s) / static_cast<float>(c);
      float q = 0.f;
#pragma unroll
      for (int g = 0; g < G; ++g)
        if ((lane + 32 * g) * 4 < c) {
#pragma unroll
          for (int i = 0; i < 4; ++i) q += (v[g][i] - mean) * (v[g][i] - mean);
        }
      rstd = 1.0f / sqrtf(warp_sum(q) / static_cast<float>(c) + eps);
    }
    __nv_bfloat16* yr = y6 + row * 6 * c;
#pragma unroll
    for (int g = 0; g < G; ++g) {      // (before the row's first store, as above)
      const int ch = (lane + 32 * g) * 4;
#pragma unroll
      for (int i = 0; i < 4; ++i)
        v[g][i] = fmaf((v[g][i] - mean) * rstd, w != nullptr && ch < c ? w[ch + i] : 1.f, b != nullptr && ch < c ? b[ch + i] : 0.f);
    }
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const int ch = (lane + 32 * g) * 4;
      if (ch >= c) continue;
      uint16_t parts[3][4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        __nv_bfloat16 x0, x1, x2;
        split3(v[g][i], x0, x1, x2);
        parts[0][i] = __bfloat16_as_ushort(x0);
        parts[1][i] = __bfloat16_as_ushort(x1);
        parts[2][i] = __bfloat16_as_ushort(x2);
      }
#pragma unroll
      for (int q = 0; q < 3; ++q)
        *reinterpret_cast<uint2*>(yr + part_a(q) * c + ch) =
            make_uint2(parts[q][0] | (static_cast<uint32_t>(parts[q][1]) << 16), parts[q][2] | (static_cast<uint32_t>(parts[q][3]) << 16));
    }
  }
}

template <typename TI>
__global__ void __launch_bounds__(256) layernorm_split_kernel(const TI* x, __nv_bfloat16* y6, const float* w, const float* b,
                                                              long long rows, int c, long long xs, float eps, int normalise) {
  grid_dependency_enter();
  const int lane = threadIdx.x & 31;
  const long long warps_per_grid = static_cast<long long>(gridDim.x) * (blockDim.x >> 5);
  for (long long row = static_cast<long long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5); row < rows;
       row += warps_per_grid) {
    const TI* xr = x + row * xs;
    float mean = 0.f, rstd = 1.f;
    if (normalise) {
      float s = 0.f;
      for (int ch = lane; ch < c; ch += 32) s += load1(xr + ch);
      mean = warp_sum(s) / static_cast<float>(c);
      float q = 0.f;
      for (int ch = lane; ch < c; ch += 32) {
        const float d = load1(xr + ch) - mean;
        q += d * d;
      }
      rstd = 1.0f / sqrtf(warp_sum(q) / static_cast<float>(c) + eps);
    }
    __nv_bfloat16* yr = y6 + row * 6 * c;
    for (int c0 = lane; c0 < c; c0 += 128) {
      float v[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int ch = min(c0 + 32 * k, c - 1);
        v[k] = fmaf((load1(xr + ch) - mean) * rstd, w != nullptr ? w[ch] : 1.f, b != nullptr ? b[ch] : 0.f);
      }
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (c0 + 32 * k < c) split3_store(yr, c, c0 + 32 * k, v[k]);
    }
  }
}

template <typename TI>
static int launch_split(cudaStream_t stream, const TI* x, __nv_bfloat16* y6, const float* w, const float* b, long long rows, int c,
                        long long xs, float eps, int normalise) {
  KFB_CHECK_ARG(rows >= 0 && c > 0, "layernorm_split: rows %lld, channels %d", rows, c);
  if (rows == 0) return KFB_OK;
  const int warps = 8;
  long long blocks = (rows + warps - 1) / warps;
  const long long cap = static_cast<long long>(sm_count()) * 16;
  if (blocks > cap) blocks = cap;
  LaunchScope scope(stream, "layernorm_split");
  auto launch = [&](auto kernel) {
    return launch_kernel(stream, kernel, static_cast<unsigned>(blocks), warps * 32, 0, x, y6, w, b, rows, c, xs, eps, normalise);
  };
  if (c % 4 != 0 || c > 1024 || xs % 4 != 0 || (reinterpret_cast<uintptr_t>(x) & 15) != 0 || (reinterpret_cast<uintptr_t>(y6) & 7) != 0)
    return launch(layernorm_split_kernel<TI>);
  if (c <= 128) return launch(layernorm_split_vec_kernel<TI, 1>);
  if (c <= 256) return launch(layernorm_split_vec_kernel<TI, 2>);
  if (c <= 512) return launch(layernorm_split_vec_kernel<TI, 4>);
  return launch(layernorm_split_vec_kernel<TI, 8>);
}

int launch_layernorm_split(cudaStream_t stream, const float* x, __nv_bfloat16* y6, const float* w, const float* b, long long rows,
                           int c, long long xs, float eps, int normalise) {
  return launch_split(stream, x, y6, w, b, rows, c, xs, eps, normalise);
}
int launch_layernorm_split(cudaStream_t stream, const __nv_bfloat16* x, __nv_bfloat16* y6, const float* w, const float* b, long long rows,
                           int c, long long xs, float eps, int normalise) {
  return launch_split(stream, x, y6, w, b, rows, c, xs, eps, normalise);
}

// Channel-major fp32 in, position-major triple split out (fp32-accurate mode).  A block turns 32 positions around through shared
// memory: a warp reads 128 bytes of a channel, then normalises one position at a time with the lanes on neighbouring channels, so
// that loads and all six stores are whole sectors.  (One thread per position, two-byte stores 6 C apart, took 300 us for 160 x 160
// positions of 128 channels; the 4 + 12 bytes per element take 8 at the memory's rate.)
constexpr int kCmSplitPos = 32;
__global__ void __launch_bounds__(256) layernorm_cm_split_kernel(const float* t, __nv_bfloat16* y6, const float* w, const float* b,
                                                                 long long npos, int c, long long chan_stride,
                                                                 long long batch_stride, float eps, int blocks_per_batch) {
  grid_dependency_enter();
  extern __shared__ __align__(16) unsigned char slab_raw_f[];
  float* slab = reinterpret_cast<float*>(slab_raw_f);  // [c][33]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int batch = blockIdx.x / blocks_per_batch;
  const long long p0 = static_cast<long long>(blockIdx.x % blocks_per_batch) * kCmSplitPos;
  const float* tb = t + batch * batch_stride + p0 + lane;
  const bool in = p0 + lane < npos;
#pragma unroll 8
  for (int ch = warp; ch < c; ch += 8) slab[ch * (kCmSplitPos + 1) + lane] = in ? tb[ch * chan_stride] : 0.f;
  float gamma[8], beta[8];        // of the lane's channels (at most 256 in all)
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int ch = lane + 32 * k;
    gamma[k] = w != nullptr && ch < c ? w[ch] : 1.f;
    beta[k] = b != nullptr && ch < c ? b[ch] : 0.f;
  }
  __syncthreads();
  for (int pp = warp; pp < kCmSplitPos && p0 + pp < npos; pp += 8) {
    const float* col = slab + pp;
    float s = 0.f;
    for (int ch = lane; ch < c; ch += 32) s += col[ch * (kCmSplitPos + 1)];
    const float mean = warp_sum(s) / static_cast<float>(c);
    float q = 0.f;
    for (int ch = lane; ch < c; ch += 32) {
      const float d = col[ch * (kCmSplitPos + 1)] - mean;
      q += d * d;
    }
    const float rstd = 1.0f / sqrtf(warp_sum(q) / static_cast<float>(c) + eps);
    __nv_bfloat16* yr = y6 + (static_cast<long long>(batch) * npos + p0 + pp) * 6 * c;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int ch = lane + 32 * k;
      if (ch < c) split3_store(yr, c, ch, fmaf((col[ch * (kCmSplitPos + 1)] - mean) * rstd, gamma[k], beta[k]));
    }
  }
}

// ------------------------------------------------------------------------------------------------
// Adaptive LayerNorm (AdaLN): one warp per row, same register layout as layernorm_rows_kernel.
// ------------------------------------------------------------------------------------------------
// SPLIT: the result as a bf16 triple split (an A operand's row of six times c, see part_a) for the fp32-accurate projections.
template <typename TI, typename TO, typename TG, int G, bool SPLIT>
__global__ void __launch_bounds__(256) adaln_rows_kernel(const TI* a, TO* y, const TG* gv, long long gv_ld, long long rows, int c,
                                                         int samples, int l, float eps) {
  grid_dependency_enter();
  const int lane = threadIdx.x & 31;
  const long long warps_per_grid = static_cast<long long>(gridDim.x) * (blockDim.x >> 5);
  for (long long row = static_cast<long long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5); row < rows;
       row += warps_per_grid) {
    const TI* xr = a + row * c;
    const long long srow = (row / (static_cast<long long>(samples) * l)) * l + row % l;
    const TG* gr = gv + srow * gv_ld;
    float2 v[G], gate[G], shift[G];
    float s = 0.f;
    // the gate / shift rows do not depend on the statistics: their loads are issued together with the row's own
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const int ch = (lane + 32 * g) * 2;
      v[g] = ch < c ? load2<TI>(xr + ch) : make_float2(0.f, 0.f);
      gate[g] = ch < c ? load2<TG>(gr + ch) : make_float2(0.f, 0.f);
      shift[g] = ch < c ? load2<TG>(gr + c + ch) : make_float2(0.f, 0.f);
      s += v[g].x + v[g].y;
    }
    const float mean = warp_sum(s) / static_cast<float>(c);
    float q = 0.f;
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const int ch = (lane + 32 * g) * 2;
      if (ch < c) {
        v[g].x -= mean;
        v[g].y -= mean;
        q += v[g].x * v[g].x + v[g].y * v[g].y;
      }
    }
    const float rstd = rsqrtf(warp_sum(q) / static_cast<float>(c) + eps);
    TO* yr = y + row * (SPLIT ? 6 * c : c);
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const int ch = (lane + 32 * g) * 2;
      if (ch < c) {
        const float s0 = 1.f / (1.f + __expf(-gate[g].x)), s1 = 1.f / (1.f + __expf(-gate[g].y));
        const float r0 = s0 * (v[g].x * rstd) + shift[g].x, r1 = s1 * (v[g].y * rstd) + shift[g].y;
        if constexpr (SPLIT) {
          __nv_bfloat16 x[2][3];
          split3(r0, x[0][0], x[0][1], x[0][2]);
          split3(r1, x[1][0], x[1][1], x[1][2]);
#pragma unroll
          for (int q = 0; q < 3; ++q) *reinterpret_cast<__nv_bfloat162*>(yr + part_a(q) * c + ch) = __halves2bfloat162(x[0][q], x[1][q]);
        } else {
          store2<TO>(yr + ch, r0, r1);
        }
      }
    }
  }
}

// bf16 rows of 256 * CH channels (the token transformer's 768, 1024): 16-byte accesses, CH per lane for each of the row,
// its gate row and its shift row (3 * CH loads in flight per lane instead of 36 four-byte ones at c = 768); the sigmoid as
// 0.5 + 0.5 tanh(g / 2) on the MUFU (one op instead of an exponential and a reciprocal; relative error 5e-4, below the
// bf16 rounding of the result).  LANES = 32: one row per warp; LANES = 16 (CH = 1, c = 128: the atom transformer):
// two rows per warp.
// `gv` stands behind the wait where the launch before may be the one that writes it (an AdaLN by itself: its gate / shift projection).
__device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[2 * i] = __uint_as_float(w[i] << 16);
    f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}
__device__ __forceinline__ void load8(const __nv_bfloat16* p, float (&f)[8]) {
  unpack8(*reinterpret_cast<const uint4*>(p), f);
}
__device__ __forceinline__ void load8(const float* p, float (&f)[8]) {
  const float4 lo = *reinterpret_cast<const float4*>(p), hi = *reinterpret_cast<const float4*>(p + 4);
  f[0] = lo.x; f[1] = lo.y; f[2] = lo.z; f[3] = lo.w; f[4] = hi.x; f[5] = hi.y; f[6] = hi.z; f[7] = hi.w;
}
// OUTS = 2: a second set of gates and shifts (`gv2`, rows as far apart) from the same statistics into `y2`: the queries' and the keys' AdaLN of
// an atom block in one launch (66 launches a step become 60; 5 x 768 tokens: 705 -> 672 us of AdaLN between events).
template <typename TI, int CH, int LANES, int OUTS>
__global__ void __launch_bounds__(256) adaln_vec_kernel(const TI* a, __nv_bfloat16* y, __nv_bfloat16* y2, const __nv_bfloat16* gv,
                                                        const __nv_bfloat16* gv2, long long gv_ld, long long rows, int samples, int l, float eps,
                                                        int gv_static) {
  constexpr int c = 8 * LANES * CH;
  constexpr int kRowsPerWarp = 32 / LANES;
  const int lane = threadIdx.x & 31;
  const int sub = lane % LANES;
  const long long warps_per_grid = static_cast<long long>(gridDim.x) * (blockDim.x >> 5);
  bool waited = false;
  for (long long base = (static_cast<long long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5)) * kRowsPerWarp; base < rows;
       base += warps_per_grid * kRowsPerWarp) {
    const long long row = base + lane / LANES;
    const bool live = row < rows;
    const long long rr = live ? row : 0;
    const unsigned r32 = static_cast<unsigned>(rr);     // (the launcher sends 2^31 rows and more elsewhere; a 64-bit division is 400 cycles)
    const long long srow = static_cast<long long>(r32 / (static_cast<unsigned>(samples) * static_cast<unsigned>(l))) * l + r32 % static_cast<unsigned>(l);
    const TI* xr = a + rr * c;
    uint4 gt[OUTS][CH], sh[OUTS][CH];
    float v[CH][8];
    // the conditioning rows of a stack's tables are there long before the rows to be normalised: fetched under the launch before
    // this one, which is writing those
    if (!gv_static && !waited) grid_dependency_enter();
#pragma unroll
    for (int o = 0; o < OUTS; ++o) {
      const __nv_bfloat16* gr = (o == 0 ? gv : gv2) + srow * gv_ld;
#pragma unroll
      for (int k = 0; k < CH; ++k) {
        const int ch = (sub + LANES * k) * 8;
        gt[o][k] = *reinterpret_cast<const uint4*>(gr + ch);
        sh[o][k] = *reinterpret_cast<const uint4*>(gr + c + ch);
      }
    }
    if (gv_static && !waited) grid_dependency_enter();
    waited = true;
#pragma unroll
    for (int k = 0; k < CH; ++k) load8(xr + (sub + LANES * k) * 8, v[k]);
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < CH; ++k)
#pragma unroll
      for (int i = 0; i < 8; ++i) s += v[k][i];
#pragma unroll
    for (int m = LANES / 2; m > 0; m >>= 1) s += __shfl_xor_sync(0xffffffffu, s, m);
    const float mean = s * (1.0f / c);
    float q = 0.f;
#pragma unroll
    for (int k = 0; k < CH; ++k)
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        v[k][i] -= mean;
        q = fmaf(v[k][i], v[k][i], q);
      }
#pragma unroll
    for (int m = LANES / 2; m > 0; m >>= 1) q += __shfl_xor_sync(0xffffffffu, q, m);
    const float rstd = rsqrtf(q * (1.0f / c) + eps);
    if (live) {
#pragma unroll
      for (int ok = 0; ok < OUTS * CH; ++ok) {
        const int out = ok / CH, k = ok % CH;
        __nv_bfloat16* yr = (out == 0 ? y : y2) + row * c;
        float g[8], t[8];
        unpack8(gt[out][k], g);
        unpack8(sh[out][k], t);
        uint32_t o[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float t0, t1;
          asm("tanh.approx.f32 %0, %1;" : "=f"(t0) : "f"(0.5f * g[2 * i]));
          asm("tanh.approx.f32 %0, %1;" : "=f"(t1) : "f"(0.5f * g[2 * i + 1]));
          const __nv_bfloat162 pr = __floats2bfloat162_rn(fmaf(fmaf(t0, 0.5f, 0.5f), v[k][2 * i] * rstd, t[2 * i]),
                                                          fmaf(fmaf(t1, 0.5f, 0.5f), v[k][2 * i + 1] * rstd, t[2 * i + 1]));
          o[i] = *reinterpret_cast<const uint32_t*>(&pr);
        }
        *reinterpret_cast<uint4*>(yr + (sub + LANES * k) * 8) = make_uint4(o[0], o[1], o[2], o[3]);
      }
    }
  }
}

template <typename TI, int CH, int LANES, int OUTS = 1>
static int launch_adaln_vec(cudaStream_t stream, const void* a, void* y, const void* gv, long long gv_ld, long long rows, int samples,
                            int l, float eps, int gv_static, void* y2 = nullptr, const void* gv2 = nullptr) {
  const long long rows_per_block = 8 * (32 / LANES);
  long long blocks = (rows + rows_per_block - 1) / rows_per_block;
  const long long cap = static_cast<long long>(sm_count()) * 16;
  if (blocks > cap) blocks = cap;
  LaunchScope scope(stream, "adaln_rows");
  KFB_TRY(launch_kernel(stream, adaln_vec_kernel<TI, CH, LANES, OUTS>, static_cast<unsigned>(blocks), 256, 0,
      static_cast<const TI*>(a), static_cast<__nv_bfloat16*>(y), static_cast<__nv_bfloat16*>(y2), static_cast<const __nv_bfloat16*>(gv),
      static_cast<const __nv_bfloat16*>(gv2), gv_ld, rows, samples, l, eps, gv_static));
  KFB_CUDA(cudaGetLastError());
  return KFB_OK;
}

template <typename TI, typename TO, typename TG, bool SPLIT = false>
static int adaln_dispatch(cudaStream_t stream, const void* a, void* y, const void* gv_, long long gv_ld, long long rows, int c,
                          int samples, int l, float eps) {
  const TG* gv = static_cast<const TG*>(gv_);
  const int warps = 8;
  long long blocks = (rows + warps - 1) / warps;
  const long long cap = static_cast<long long>(sm_count()) * 16;
  if (blocks > cap) blocks = cap;
  const int g = cdiv(c, 64);
  LaunchScope scope(stream, "adaln_rows");
#define KFB_ADALN(GG)                                                                                          \
  KFB_TRY(launch_kernel(stream, adaln_rows_kernel<TI, TO, TG, GG, SPLIT>, static_cast<unsigned>(blocks), warps * 32, 0, \
      static_cast<const TI*>(a), static_cast<TO*>(y), gv, gv_ld, rows, c, samples, l, eps))
  if (g <= 2) KFB_ADALN(2);
  else if (g <= 6) KFB_ADALN(6);
  else if (g <= 12) KFB_ADALN(12);
  else if (g <= 16) KFB_ADALN(16);
  else {
    set_error("adaln: channel count %d above 1024 is not supported", c);
    return KFB_ERR_UNSUPPORTED;
  }
#undef KFB_ADALN
  KFB_CUDA(cudaGetLastError());
  return KFB_OK;
}

int launch_adaln(cudaStream_t stream, const void* a, void* y, const void* gv, long long rows, int c, int samples,
                 int l, float eps, int in_dtype, int out_dtype, long long gv_ld, int gv_static) {
  if (gv_ld <= 0) gv_ld = 2ll * c;
  KFB_CHECK_ARG(gv_ld >= 2ll * c && gv_ld % 2 == 0 && (reinterpret_cast<uintptr_t>(gv) & 7) == 0,
                "adaln: gate/shift row stride %lld (at least 2c, even) or misaligned pointer", gv_ld);
  KFB_CHECK_ARG(rows >= 0 && c > 0 && c % 2 == 0 && samples >= 1 && l >= 1, "adaln: rows %lld c %d samples %d l %d", rows, c,
                samples, l);
  KFB_CHECK_ARG(rows % (static_cast<long long>(samples) * l) == 0, "adaln: rows %lld is not a multiple of samples*l", rows);
  if (rows == 0) return KFB_OK;
  if ((in_dtype == KFB_BF16 || in_dtype == KFB_FP32) && out_dtype == KFB_BF16 && gv_ld % 8 == 0 && rows < (1ll << 31) &&
      ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(gv)) & 15) == 0) {
#define KFB_ADALN_VEC(CH, LANES)                                                                                          \
  return in_dtype == KFB_BF16 ? launch_adaln_vec<__nv_bfloat16, CH, LANES>(stream, a, y, gv, gv_ld, rows, samples, l, eps, gv_static) \
                              : launch_adaln_vec<float, CH, LANES>(stream, a, y, gv, gv_ld, rows, samples, l, eps, gv_static)
    switch (c) {
      case 128: KFB_ADALN_VEC(1, 16);
      case 256: KFB_ADALN_VEC(1, 32);
      case 512: KFB_ADALN_VEC(2, 32);
      case 768: KFB_ADALN_VEC(3, 32);
      case 1024: KFB_ADALN_VEC(4, 32);
      default: break;
    }
#undef KFB_ADALN_VEC
  }
  if (in_dtype == KFB_BF16 && out_dtype == KFB_BF16)
    return adaln_dispatch<__nv_bfloat16, __nv_bfloat16, __nv_bfloat16>(stream, a, y, gv, gv_ld, rows, c, samples, l, eps);
  if (in_dtype == KFB_FP32 && out_dtype == KFB_BF16)
    return adaln_dispatch<float, __nv_bfloat16, __nv_bfloat16>(stream, a, y, gv, gv_ld, rows, c, samples, l, eps);
  if (in_dtype == KFB_FP32_PRECISE && out_dtype == KFB_FP32_PRECISE)  // fp32 in, triple split out: no pass of its own for the split
    return adaln_dispatch<float, __nv_bfloat16, float, true>(stream, a, y, gv, gv_ld, rows, c, samples, l, eps);
  if (in_dtype == KFB_FP32_PRECISE && out_dtype == KFB_FP32)  // everything fp32, gate / shift rows included
    return adaln_dispatch<float, float, float>(stream, a, y, gv, gv_ld, rows, c, samples, l, eps);
  set_error("adaln: unsupported dtype combination");
  return KFB_ERR_INVALID_ARGUMENT;
}

int launch_adaln_two(cudaStream_t stream, const void* a, void* y, void* y2, const void* gv, const void* gv2, long long rows, int c, int samples, int l,
                     float eps, int in_dtype, long long gv_ld, int gv_static) {
  const uintptr_t all = reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(y2) |
                        reinterpret_cast<uintptr_t>(gv) | reinterpret_cast<uintptr_t>(gv2);
  if (c == 128 && rows > 0 && rows < (1ll << 31) && rows % (static_cast<long long>(samples) * l) == 0 && gv_ld % 8 == 0 && gv_ld >= 2ll * c && (all & 15) == 0)
    return in_dtype == KFB_BF16 ? launch_adaln_vec<__nv_bfloat16, 1, 16, 2>(stream, a, y, gv, gv_ld, rows, samples, l, eps, gv_static, y2, gv2)
                                : launch_adaln_vec<float, 1, 16, 2>(stream, a, y, gv, gv_ld, rows, samples, l, eps, gv_static, y2, gv2);
  KFB_TRY(launch_adaln(stream, a, y, gv, rows, c, samples, l, eps, in_dtype, KFB_BF16, gv_ld, gv_static));
  return launch_adaln(stream, a, y2, gv2, rows, c, samples, l, eps, in_dtype, KFB_BF16, gv_ld, gv_static);
}

// ------------------------------------------------------------------------------------------------
// Channel-major in, position-major out.  A block of 128 threads stages a [c][128 positions] slab in shared
// memory as bf16 (each warp copies whole channel rows: 256 contiguous bytes per row), then every thread
// owns ONE position: it walks down its column of the slab (neighbouring lanes read neighbouring 2-byte
// cells, so the column walk is bank-conflict free), takes mean and variance in two passes and writes its
// normalised row of c channels with 16-byte stores.
// ------------------------------------------------------------------------------------------------
static constexpr int kCmPos = 128;

__device__ __forceinline__ float cm_to_float(__nv_bfloat16 v) { return __bfloat162float(v); }
__device__ __forceinline__ float cm_to_float(float v) { return v; }
__device__ __forceinline__ uint32_t cm_pack(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}

template <typename TI>
__global__ void __launch_bounds__(kCmPos) layernorm_cm_kernel(const TI* t, __nv_bfloat16* y, const float* w, const float* b, long long npos, int c,
                                                              long long chan_stride, long long batch_stride, float eps, int blocks_per_batch) {
  grid_dependency_enter();
  extern __shared__ __align__(16) unsigned char slab_raw[];
  __nv_bfloat16* slab = reinterpret_cast<__nv_bfloat16*>(slab_raw);  // [c][128]
  const int batch = blockIdx.x / blocks_per_batch;
  const long long p0 = static_cast<long long>(blockIdx.x % blocks_per_batch) * kCmPos;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const TI* tb = t + batch * batch_stride + p0;
  const bool full = (p0 + kCmPos <= npos) && ((chan_stride & 3) == 0) && ((reinterpret_cast<uintptr_t>(tb) & 7) == 0);
  for (int ch = warp; ch < c; ch += kCmPos / 32) {
    const TI* src = tb + ch * chan_stride + lane * 4;
    __nv_bfloat16* dst = slab + ch * kCmPos + lane * 4;
    if (full && sizeof(TI) == 2) {
      *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(src);
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        dst[i] = (p0 + lane * 4 + i < npos) ? __float2bfloat16_rn(cm_to_float(src[i])) : __float2bfloat16_rn(0.f);
    }
  }
  __syncthreads();
  const long long p = p0 + threadIdx.x;
  if (p >= npos) return;
  const __nv_bfloat16* col = slab + threadIdx.x;
  // mean and variance in one walk down the column, as sums of (x - x0) and (x - x0)^2 with x0 the first channel:
  // the shift keeps the subtraction of the squared mean harmless
  const float x0 = __bfloat162float(col[0]);
  float s = 0.f, q2 = 0.f;
#pragma unroll 8
  for (int ch = 0; ch < c; ++ch) {
    const float d = __bfloat162float(col[ch * kCmPos]) - x0;
    s += d;
    q2 = fmaf(d, d, q2);
  }
  const float ms = s / static_cast<float>(c);
  const float mean = x0 + ms;
  const float q = fmaxf(q2 - s * ms, 0.f);
  const float rstd = rsqrtf(q / static_cast<float>(c) + eps);
  __nv_bfloat16* yr = y + (static_cast<long long>(batch) * npos + p) * c;
  if ((c & 15) == 0 && (reinterpret_cast<uintptr_t>(yr) & 31) == 0) {
    for (int ch = 0; ch < c; ch += 16) {   // 32-byte stores: one full sector per instruction
      uint32_t o[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        float a0 = (__bfloat162float(col[(ch + 2 * i) * kCmPos]) - mean) * rstd;
        float a1 = (__bfloat162float(col[(ch + 2 * i + 1) * kCmPos]) - mean) * rstd;
        if (w != nullptr) { a0 *= w[ch + 2 * i]; a1 *= w[ch + 2 * i + 1]; }
        if (b != nullptr) { a0 += b[ch + 2 * i]; a1 += b[ch + 2 * i + 1]; }
        o[i] = cm_pack(a0, a1);
      }
      asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(yr + ch), "r"(o[0]), "r"(o[1]), "r"(o[2]),
                   "r"(o[3]), "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7])
                   : "memory");
    }
    return;
  }
  for (int ch = 0; ch < c; ch += 8) {
    float a[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      a[i] = (__bfloat162float(col[(ch + i) * kCmPos]) - mean) * rstd;
      if (w != nullptr) a[i] *= w[ch + i];
      if (b != nullptr) a[i] += b[ch + i];
    }
    *reinterpret_cast<uint4*>(yr + ch) = make_uint4(cm_pack(a[0], a[1]), cm_pack(a[2], a[3]), cm_pack(a[4], a[5]), cm_pack(a[6], a[7]));
  }
}

// ------------------------------------------------------------------------------------------------
// LayerNorm folded into the GEMM that follows it.  For rows x (c channels) and a projection W,
//   LN(x) W^T = rstd * (x W'^T - mean * s1) + s0,   W' = gamma * W,  s1[n] = sum_k W'[n][k],  s0[n] = sum_k beta[k] W[n][k],
// so the GEMM can read the raw rows (here: channel-major, as the triangle contraction leaves them) and the epilogue
// applies the per-row (mean, rstd) and the per-column s1, s0.  The projection's kernel takes the statistics itself where it has the
// warps for it (gemm.cuh, STATS); cm_stats does where it has not.
// ------------------------------------------------------------------------------------------------
// (mean, rstd) over the channels of every position of a channel-major tensor t[c][npos]; two positions per thread
__global__ void __launch_bounds__(256) cm_stats_kernel(const __nv_bfloat16* t, float2* stats, long long npos, int c, long long chan_stride,
                                                       float eps) {
  grid_dependency_enter();
  const long long p2 = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) * 2;
  if (p2 >= npos) return;
  const bool pair = p2 + 1 < npos;
  float s0 = 0.f, s1 = 0.f, q0 = 0.f, q1 = 0.f;
  // shifted sums (by the first channel's value) keep E[x^2] - E[x]^2 harmless
  float x00, x01;
  {
    const __nv_bfloat16* src = t + p2;
    x00 = __bfloat162float(src[0]);
    x01 = pair ? __bfloat162float(src[1]) : 0.f;
  }
#pragma unroll 8
  for (int ch = 0; ch < c; ++ch) {
    const __nv_bfloat16* src = t + ch * chan_stride + p2;
    float a, b2;
    if (pair) {
      const uint32_t w = *reinterpret_cast<const uint32_t*>(src);
      a = __uint_as_float(w << 16);
      b2 = __uint_as_float(w & 0xffff0000u);
    } else {
      a = __bfloat162float(src[0]);
      b2 = 0.f;
    }
    const float d0 = a - x00, d1 = b2 - x01;
    s0 += d0; q0 = fmaf(d0, d0, q0);
    s1 += d1; q1 = fmaf(d1, d1, q1);
  }
  const float inv_c = 1.0f / static_cast<float>(c);
  const float m0 = s0 * inv_c, m1 = s1 * inv_c;
  stats[p2] = make_float2(x00 + m0, rsqrtf(fmaxf(q0 - s0 * m0, 0.f) * inv_c + eps));
  if (pair) stats[p2 + 1] = make_float2(x01 + m1, rsqrtf(fmaxf(q1 - s1 * m1, 0.f) * inv_c + eps));
}

// The same with four positions per thread (8-byte loads): half as many CTAs, all resident at once for a 768 x 768 pair
// tensor, and twice the bytes in flight per thread.  npos and the channel stride multiples of 4, t 8-byte aligned.
__global__ void __launch_bounds__(128) cm_stats4_kernel(const __nv_bfloat16* t, float2* stats, long long npos, int c, long long chan_stride,
                                                        float eps) {
  grid_dependency_enter();
  const long long p4 = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) * 4;
  if (p4 >= npos) return;
  float s[4] = {0.f, 0.f, 0.f, 0.f}, q[4] = {0.f, 0.f, 0.f, 0.f}, x0[4];
  {
    const uint2 w = *reinterpret_cast<const uint2*>(t + p4);
    x0[0] = __uint_as_float(w.x << 16);
    x0[1] = __uint_as_float(w.x & 0xffff0000u);
    x0[2] = __uint_as_float(w.y << 16);
    x0[3] = __uint_as_float(w.y & 0xffff0000u);
  }
#pragma unroll 8
  for (int ch = 0; ch < c; ++ch) {
    const uint2 w = *reinterpret_cast<const uint2*>(t + ch * chan_stride + p4);
    const float v[4] = {__uint_as_float(w.x << 16), __uint_as_float(w.x & 0xffff0000u), __uint_as_float(w.y << 16),
                        __uint_as_float(w.y & 0xffff0000u)};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float d = v[i] - x0[i];
      s[i] += d;
      q[i] = fmaf(d, d, q[i]);
    }
  }
  const float inv_c = 1.0f / static_cast<float>(c);
  float4 o[2];
  float* of = reinterpret_cast<float*>(o);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float m = s[i] * inv_c;
    of[2 * i] = x0[i] + m;
    of[2 * i + 1] = rsqrtf(fmaxf(q[i] - s[i] * m, 0.f) * inv_c + eps);
  }
  float4* dst = reinterpret_cast<float4*>(stats + p4);
  dst[0] = o[0];
  dst[1] = o[1];
}

int launch_cm_stats(cudaStream_t stream, const __nv_bfloat16* t, float2* stats, long long npos, int c, long long chan_stride,
                    float eps) {
  KFB_CHECK_ARG(npos > 0 && npos % 2 == 0 && c > 0 && chan_stride % 2 == 0 && (reinterpret_cast<uintptr_t>(t) & 3) == 0,
                "cm_stats: npos %lld (even), c %d, channel stride %lld (even)", npos, c, chan_stride);
  LaunchScope scope(stream, "layernorm_cm_stats");
  if (npos % 4 == 0 && chan_stride % 4 == 0 && (reinterpret_cast<uintptr_t>(t) & 7) == 0 &&
      (reinterpret_cast<uintptr_t>(stats) & 15) == 0) {
    const long long threads4 = npos / 4;
    KFB_TRY(launch_kernel(stream, cm_stats4_kernel, static_cast<unsigned>((threads4 + 127) / 128), 128, 0, t, stats, npos, c,
        chan_stride, eps));
    KFB_CUDA(cudaGetLastError());
    return KFB_OK;
  }
  const long long threads = npos / 2;
  KFB_TRY(launch_kernel(stream, cm_stats_kernel, static_cast<unsigned>((threads + 255) / 256), 256, 0, t, stats, npos, c,
      chan_stride, eps));
  KFB_CUDA(cudaGetLastError());
  return KFB_OK;
}

__device__ __forceinline__ float to_float(__nv_bfloat16 v) { return __bfloat162float(v); }
__device__ __forceinline__ float to_float(float v) { return v; }
template <typename T> __device__ __forceinline__ T from_float(float v);
template <> __device__ __forceinline__ __nv_bfloat16 from_float<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
template <> __device__ __forceinline__ float from_float<float>(float v) { return v; }

// LayerNorm over a few channels followed by a projection to `nh` head values, one thread per position: the pair
// bias of the atom windows (16 channels in, heads x layers out).  x [npos][C]; w [nh][C]; y [nh][npos] (head-major,
// positions contiguous).  bf16 mode rounds the normalised value to bf16 as the reference's LayerNorm does and
// accumulates in fp32; fp32 mode keeps everything in fp32.
template <int C, typename T>
__global__ void __launch_bounds__(256) window_bias_kernel(const T* x, const float* ln_w, const float* ln_b, const T* w, T* y, long long npos,
                                                          int nh, float eps, int normalise) {
  grid_dependency_enter();
  extern __shared__ float s_w[];  // [nh][C] fp32, then gamma[C], beta[C]
  float* s_g = s_w + nh * C;
  float* s_b = s_g + C;
  for (int i = threadIdx.x; i < nh * C; i += blockDim.x) s_w[i] = to_float(w[i]);
  for (int i = threadIdx.x; i < C; i += blockDim.x) {
    s_g[i] = ln_w != nullptr ? ln_w[i] : 1.0f;
    s_b[i] = ln_b != nullptr ? ln_b[i] : 0.0f;
  }
  __syncthreads();
  const long long pos = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (pos >= npos) return;
  float v[C];
  const T* xr = x + pos * C;
  constexpr int kVec = 16 / sizeof(T);
#pragma unroll
  for (int i = 0; i < C; i += kVec) {
    const uint4 raw = *reinterpret_cast<const uint4*>(xr + i);
    const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
    for (int j = 0; j < kVec; ++j) v[i + j] = to_float(e[j]);
  }
  if (normalise) {
    float mean = 0.f;
#pragma unroll
    for (int i = 0; i < C; ++i) mean += v[i];
    mean *= 1.0f / C;
    float var = 0.f;
#pragma unroll
    for (int i = 0; i < C; ++i) var += (v[i] - mean) * (v[i] - mean);
    const float rstd = rsqrtf(var * (1.0f / C) + eps);
#pragma unroll
    for (int i = 0; i < C; ++i) v[i] = to_float(from_float<T>((v[i] - mean) * rstd * s_g[i] + s_b[i]));
  }
  for (int h = 0; h < nh; ++h) {
    float acc = 0.f;
#pragma unroll
    for (int i = 0; i < C; ++i) acc = fmaf(v[i], s_w[h * C + i], acc);
    y[static_cast<long long>(h) * npos + pos] = from_float<T>(acc);
  }
}

template <int C>
static int launch_window_bias_c(cudaStream_t stream, const void* x, const float* ln_w, const float* ln_b, const void* w, void* y,
                                long long npos, int nh, float eps, int normalise, int dtype) {
  const size_t smem = (static_cast<size_t>(nh) * C + 2 * C) * sizeof(float);
  const unsigned blocks = static_cast<unsigned>((npos + 255) / 256);
  LaunchScope scope(stream, "window_bias");
  if (dtype == KFB_BF16)
    KFB_TRY(launch_kernel(stream, window_bias_kernel<C, __nv_bfloat16>, blocks, 256, smem,
        static_cast<const __nv_bfloat16*>(x), ln_w, ln_b, static_cast<const __nv_bfloat16*>(w), static_cast<__nv_bfloat16*>(y),
        npos, nh, eps, normalise));
  else
    KFB_TRY(launch_kernel(stream, window_bias_kernel<C, float>, blocks, 256, smem, static_cast<const float*>(x), ln_w, ln_b,
                                                                static_cast<const float*>(w), static_cast<float*>(y), npos, nh, eps,
                                                                normalise));
  KFB_CUDA(cudaGetLastError());
  return KFB_OK;
}

int launch_window_bias(cudaStream_t stream, const void* x, const float* ln_w, const float* ln_b, const void* w, void* y,
                       long long npos, int c, int nh, float eps, int normalise, int dtype) {
  KFB_CHECK_ARG(dtype == KFB_BF16 || dtype == KFB_FP32, "window_bias: dtype %d (bf16 or fp32)", dtype);
  KFB_CHECK_ARG(nh >= 1 && nh * c <= 8192, "window_bias: %d heads x %d channels exceed the shared-memory weight table", nh, c);
  KFB_CHECK_ARG(npos < (1ll << 31) * 256, "window_bias: too many positions");
  if (npos == 0) return KFB_OK;
  switch (c) {
    case 16: return launch_window_bias_c<16>(stream, x, ln_w, ln_b, w, y, npos, nh, eps, normalise, dtype);
    case 32: return launch_window_bias_c<32>(stream, x, ln_w, ln_b, w, y, npos, nh, eps, normalise, dtype);
    case 64: return launch_window_bias_c<64>(stream, x, ln_w, ln_b, w, y, npos, nh, eps, normalise, dtype);
    default:
      set_error("window_bias: %d channels not supported (16, 32 or 64)", c);
      return KFB_ERR_UNSUPPORTED;
  }
}

int launch_layernorm_cm(cudaStream_t stream, const void* t, __nv_bfloat16* y, const float* w, const float* b, int batch,
                        long long npos, int c, long long chan_stride, long long batch_stride, float eps, int in_dtype,
                        int split_out) {
  KFB_CHECK_ARG(c > 0 && c % 8 == 0 && c <= 512, "layernorm_cm: channels %d (multiple of 8, at most 512)", c);
  if (split_out) {
    KFB_CHECK_ARG(in_dtype == KFB_FP32 && c <= 256, "layernorm_cm: the split output takes fp32 input and at most 256 channels");
    if (npos == 0 || batch == 0) return KFB_OK;
    const int bpb = static_cast<int>((npos + kCmSplitPos - 1) / kCmSplitPos);
    const size_t smem = static_cast<size_t>(c) * (kCmSplitPos + 1) * sizeof(float);   // at most 33 KB
    LaunchScope scope(stream, "layernorm_cm_split");
    KFB_TRY(launch_kernel(stream, layernorm_cm_split_kernel, bpb * batch, 256, smem, static_cast<const float*>(t), y, w, b, npos, c,
                          chan_stride, batch_stride, eps, bpb));
    KFB_CUDA(cudaGetLastError());
    return KFB_OK;
  }
  KFB_CHECK_ARG((reinterpret_cast<uintptr_t>(y) & 15) == 0, "layernorm_cm: output must be 16-byte aligned");
  if (npos == 0 || batch == 0) return KFB_OK;
  const int bpb = static_cast<int>((npos + kCmPos - 1) / kCmPos);
  const size_t smem = static_cast<size_t>(c) * kCmPos * sizeof(__nv_bfloat16);
  LaunchScope scope(stream, "layernorm_cm");
  if (in_dtype == KFB_BF16) {
    if (smem > 48 * 1024)
      KFB_CUDA(cudaFuncSetAttribute(layernorm_cm_kernel<__nv_bfloat16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    KFB_TRY(launch_kernel(stream, layernorm_cm_kernel<__nv_bfloat16>, bpb * batch, kCmPos, smem,
        static_cast<const __nv_bfloat16*>(t), y, w, b, npos,
                                                                           c, chan_stride, batch_stride, eps, bpb));
  } else {
    if (smem > 48 * 1024)
      KFB_CUDA(cudaFuncSetAttribute(layernorm_cm_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    KFB_TRY(launch_kernel(stream, layernorm_cm_kernel<float>, bpb * batch, kCmPos, smem, static_cast<const float*>(t), y, w,
        b, npos, c, chan_stride,
                                                                   batch_stride, eps, bpb));
  }
  KFB_CUDA(cudaGetLastError());
  return KFB_OK;
}

}  // namespace kfb
