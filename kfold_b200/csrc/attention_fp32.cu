// fp32 attention with pair bias and key mask for the fp32-accurate mode.
//
// CUDA cores, float32 throughout, an online softmax (the L x L x H logits are never stored).  Same semantics as attention.cu:
// additive pair bias, masked keys get -1e9 (finite, as the reference does), optional sigmoid gate, and the result is written as the
// bf16 triple split (an A operand's row, see part_a) that the fp32-accurate output projection consumes.
//
// A block takes 32 or 64 queries of one head and splits the keys over its eight or four warps, eight keys at a time; a lane owns one
// or two query rows, and the warps' (maximum, sum, accumulator) are merged at the end.  The single-track problems (a few hundred queries,
// one batch entry, 16 heads) have too few rows to fill the chip with one thread per row and all keys each: 301 queries x 16 heads x 48
// took 250 us that way.  A warp stages its own keys in a two-slot ring with cp.async, so nothing but the merge waits for another
// warp; K and V are read as broadcast 16-byte pieces, which bounds the loop (one load feeds four multiply-adds per query row: two
// rows per lane where there are enough blocks without it).
#include "attention.cuh"
#include "gemm.cuh"  // part_a
#include "ptx.cuh"

#include <mutex>

namespace kfb {
namespace {

constexpr int kKeys = 8;    // keys per warp and step

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(ptx::smem_u32(smem)), "l"(gmem) : "memory");
}

template <int D, int QPT, int kWarps>
struct F32Cfg {
  static constexpr int kQ = 32 * QPT;
  static constexpr int kRing = kWarps * 2 * 2 * kKeys * D;             // floats: [warp][slot][K | V][key][D]
  static constexpr int kMerge = (kWarps / 2) * kQ * (D + 1);           // the same memory after the loop
  static constexpr int kMain = kRing > kMerge ? kRing : kMerge;
  static constexpr int kBias = kWarps * kQ * (kKeys + 1);
  static constexpr int kSmem = (kMain + kBias + 2 * kWarps * kQ) * 4;
};

template <int D, int QPT, int kWarps>
__global__ void __launch_bounds__(kWarps * 32) attention_fp32_kernel(const AttnFp32Params p) {
  using Cfg = F32Cfg<D, QPT, kWarps>;
  constexpr int kQ = Cfg::kQ;
  grid_dependency_enter();
  extern __shared__ __align__(16) float smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* ring = smem + warp * (4 * kKeys * D);
  float* s_bias = smem + Cfg::kMain + warp * kQ * (kKeys + 1);
  float* s_m = smem + Cfg::kMain + Cfg::kBias;      // [warp][query]
  float* s_l = s_m + kWarps * kQ;
  const int q0 = blockIdx.x * kQ, h = blockIdx.y, b = blockIdx.z;
  const int b_hi = b / p.mask_lo_extent, b_lo = b - b_hi * p.mask_lo_extent;
  const unsigned char* mrow =
      p.mask == nullptr ? nullptr : p.mask + static_cast<long long>(b_hi) * p.m_hi + static_cast<long long>(b_lo) * p.m_lo;
  const int bias_b = p.bias_mod > 0 ? (b / p.bias_div) * p.bias_mod + b % p.bias_mod : b / p.bias_div;
  const long long bias_z = p.bias_head_major > 0 ? static_cast<long long>(h) * p.bias_head_major + bias_b
                                                 : static_cast<long long>(bias_b) * p.heads + h;
  const float* bias_base = p.bias + bias_z * (p.bias_hs > 0 ? p.bias_hs : p.lq * p.ldb);
  const long long ld_kv = p.ld_kv > 0 ? p.ld_kv : p.ld;
  const float* k_base = p.k + static_cast<long long>(b) * p.lk * ld_kv + p.k_col0 + h * D;
  const float* v_base = p.v + static_cast<long long>(b) * p.lk * ld_kv + p.v_col0 + h * D;

  float q[QPT][D], acc[QPT][D], m_run[QPT], l_run[QPT];
#pragma unroll
  for (int i = 0; i < QPT; ++i) {
    const long long row = static_cast<long long>(b) * p.lq + min(q0 + i * 32 + lane, p.lq - 1);
    const float4* src = reinterpret_cast<const float4*>(p.q + row * p.ld + p.q_col0 + h * D);
#pragma unroll
    for (int d = 0; d < D / 4; ++d) {
      const float4 f = src[d];
      q[i][4 * d] = f.x; q[i][4 * d + 1] = f.y; q[i][4 * d + 2] = f.z; q[i][4 * d + 3] = f.w;
    }
#pragma unroll
    for (int d = 0; d < D; ++d) acc[i][d] = 0.f;
    m_run[i] = -INFINITY;
    l_run[i] = 0.f;
  }

  const int groups = (p.lk + kKeys - 1) / kKeys;
  // bias and mask of a group are fetched a step ahead: lane = (row of four, key), which reads whole sectors
  float bias_r[8 * QPT], mask_r = 0.f;
  auto fetch = [&](int g, int slot) {
    float* dst = ring + slot * (2 * kKeys * D);
#pragma unroll
    for (int idx = lane; idx < kKeys * D / 4; idx += 32) {
      const int kk = idx / (D / 4), c = idx - kk * (D / 4);
      const long long off = static_cast<long long>(min(g * kKeys + kk, p.lk - 1)) * ld_kv + c * 4;
      cp_async16(dst + idx * 4, k_base + off);
      cp_async16(dst + kKeys * D + idx * 4, v_base + off);
    }
    const int key = g * kKeys + (lane & 7);
    mask_r = key < p.lk ? ((mrow == nullptr || mrow[static_cast<long long>(key) * p.m_k]) ? 0.f : -1e9f) : -INFINITY;
#pragma unroll
    for (int i = 0; i < 8 * QPT; ++i) {
      const int row = min(q0 + i * 4 + (lane >> 3), p.lq - 1);
      bias_r[i] = key < p.lk ? bias_base[static_cast<long long>(row) * p.ldb + key] : 0.f;
    }
  };
  if (warp < groups) fetch(warp, 0);
  asm volatile("cp.async.commit_group;" ::: "memory");
  int slot = 0;
  for (int g = warp; g < groups; g += kWarps, slot ^= 1) {
    const float mask_v = mask_r;
#pragma unroll
    for (int i = 0; i < 8 * QPT; ++i) s_bias[(i * 4 + (lane >> 3)) * (kKeys + 1) + (lane & 7)] = bias_r[i];
    if (g + kWarps < groups) fetch(g + kWarps, slot ^ 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();
    const float4* sk = reinterpret_cast<const float4*>(ring + slot * (2 * kKeys * D));
    const float4* sv = sk + kKeys * D / 4;
    float s[QPT][kKeys];
#pragma unroll
    for (int i = 0; i < QPT; ++i)
#pragma unroll
      for (int kk = 0; kk < kKeys; ++kk) s[i][kk] = 0.f;
#pragma unroll
    for (int d = 0; d < D / 4; ++d)
#pragma unroll
      for (int kk = 0; kk < kKeys; ++kk) {
        const float4 f = sk[kk * (D / 4) + d];
#pragma unroll
        for (int i = 0; i < QPT; ++i) {
          s[i][kk] = fmaf(q[i][4 * d], f.x, s[i][kk]);
          s[i][kk] = fmaf(q[i][4 * d + 1], f.y, s[i][kk]);
          s[i][kk] = fmaf(q[i][4 * d + 2], f.z, s[i][kk]);
          s[i][kk] = fmaf(q[i][4 * d + 3], f.w, s[i][kk]);
        }
      }
#pragma unroll
    for (int i = 0; i < QPT; ++i) {
      float mx = -INFINITY;
#pragma unroll
      for (int kk = 0; kk < kKeys; ++kk) {
        // same order of additions as the reference: (q k + mask) + bias
        s[i][kk] = (s[i][kk] + __shfl_sync(0xffffffffu, mask_v, kk)) + s_bias[(i * 32 + lane) * (kKeys + 1) + kk];
        mx = fmaxf(mx, s[i][kk]);
      }
      const float m_new = fmaxf(m_run[i], mx);
      const float alpha = expf(m_run[i] - m_new);
      l_run[i] *= alpha;
#pragma unroll
      for (int d = 0; d < D; ++d) acc[i][d] *= alpha;
#pragma unroll
      for (int kk = 0; kk < kKeys; ++kk) {
        s[i][kk] = expf(s[i][kk] - m_new);
        l_run[i] += s[i][kk];
      }
      m_run[i] = m_new;
    }
#pragma unroll
    for (int kk = 0; kk < kKeys; ++kk)
#pragma unroll
      for (int d = 0; d < D / 4; ++d) {
        const float4 f = sv[kk * (D / 4) + d];
#pragma unroll
        for (int i = 0; i < QPT; ++i) {
          acc[i][4 * d] = fmaf(s[i][kk], f.x, acc[i][4 * d]);
          acc[i][4 * d + 1] = fmaf(s[i][kk], f.y, acc[i][4 * d + 1]);
          acc[i][4 * d + 2] = fmaf(s[i][kk], f.z, acc[i][4 * d + 2]);
          acc[i][4 * d + 3] = fmaf(s[i][kk], f.w, acc[i][4 * d + 3]);
        }
      }
    __syncwarp();   // the slot and the bias tile may be written again
  }

  // merge the warps' softmax states; a warp without keys has m = -inf, l = 0
#pragma unroll
  for (int i = 0; i < QPT; ++i) {
    s_m[warp * kQ + i * 32 + lane] = m_run[i];
    s_l[warp * kQ + i * 32 + lane] = l_run[i];
  }
  __syncthreads();
  float inv_l[QPT];
#pragma unroll
  for (int i = 0; i < QPT; ++i) {
    float m = -INFINITY, l = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) m = fmaxf(m, s_m[w * kQ + i * 32 + lane]);
#pragma unroll
    for (int w = 0; w < kWarps; ++w) l += s_l[w * kQ + i * 32 + lane] * expf(s_m[w * kQ + i * 32 + lane] - m);
    inv_l[i] = 1.0f / l;
    const float scale = expf(m_run[i] - m);
#pragma unroll
    for (int d = 0; d < D; ++d) acc[i][d] *= scale;
  }
#pragma unroll 1
  for (int half = kWarps / 2; half >= 1; half >>= 1) {
    if (warp >= half && warp < 2 * half) {
#pragma unroll
      for (int i = 0; i < QPT; ++i)
#pragma unroll
        for (int d = 0; d < D; ++d) smem[((warp - half) * kQ + i * 32 + lane) * (D + 1) + d] = acc[i][d];
    }
    __syncthreads();
    if (warp < half) {
#pragma unroll
      for (int i = 0; i < QPT; ++i)
#pragma unroll
        for (int d = 0; d < D; ++d) acc[i][d] += smem[(warp * kQ + i * 32 + lane) * (D + 1) + d];
    }
    __syncthreads();
  }
  if (warp == 0) {
#pragma unroll
    for (int i = 0; i < QPT; ++i)
#pragma unroll
      for (int d = 0; d < D; ++d) smem[(i * 32 + lane) * (D + 1) + d] = acc[i][d] * inv_l[i];
  }
  __syncthreads();
  const int hd = p.heads * D;
  for (int idx = threadIdx.x; idx < kQ * D; idx += kWarps * 32) {
    const int qq = idx / D, d = idx - qq * D;
    if (q0 + qq >= p.lq) break;
    const long long qrow = static_cast<long long>(b) * p.lq + q0 + qq;
    float o = smem[qq * (D + 1) + d];
    if (p.g != nullptr) o *= 1.0f / (1.0f + expf(-p.g[qrow * p.ld + p.g_col0 + h * D + d]));
    __nv_bfloat16* o6 = p.out6 + qrow * 6 * hd;
    const int col = h * D + d;
    const __nv_bfloat16 x0 = __float2bfloat16_rn(o);
    const float r1 = o - __bfloat162float(x0);
    const __nv_bfloat16 x1 = __float2bfloat16_rn(r1);
    const __nv_bfloat16 x2 = __float2bfloat16_rn(r1 - __bfloat162float(x1));
    o6[part_a(0) * hd + col] = x0;
    o6[part_a(1) * hd + col] = x1;
    o6[part_a(2) * hd + col] = x2;
  }
}

template <int D, int QPT, int kWarps>
int launch(cudaStream_t stream, const AttnFp32Params& p) {
  using Cfg = F32Cfg<D, QPT, kWarps>;
  static std::once_flag once[64];
  int dev = 0;
  KFB_CUDA(cudaGetDevice(&dev));
  cudaError_t attr_err = cudaSuccess;
  std::call_once(once[dev & 63], [&] {
    attr_err = cudaFuncSetAttribute(attention_fp32_kernel<D, QPT, kWarps>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmem);
  });
  KFB_CUDA(attr_err);
  LaunchScope scope(stream, p.tag ? p.tag : "attention_fp32");
  const dim3 grid(cdiv(p.lq, Cfg::kQ), p.heads, p.batch);
  KFB_TRY(launch_kernel(stream, attention_fp32_kernel<D, QPT, kWarps>, grid, kWarps * 32, Cfg::kSmem, p));
  return KFB_OK;
}

}  // namespace

int launch_attention_fp32(cudaStream_t stream, const AttnFp32Params& p) {
  KFB_CHECK_ARG(p.batch > 0 && p.heads > 0 && p.lq > 0 && p.lk > 0, "attention_fp32: empty problem");
  KFB_CHECK_ARG(p.batch <= 65535 && p.heads <= 65535, "attention_fp32: batch %d / heads %d exceed the grid limits", p.batch, p.heads);
  // two query rows per lane: half the shared-memory reads per row, but half the blocks (and registers for head dims up to 32 only);
  // with that many blocks four warps share the keys, which halves what is merged (160 x 160 rows: 180 us with eight)
  const bool two = p.lq > 32 && static_cast<long long>(cdiv(p.lq, 64)) * p.heads * p.batch >= 2ll * sm_count();
  switch (p.d) {
    case 16: return two ? launch<16, 2, 4>(stream, p) : launch<16, 1, 8>(stream, p);
    case 24: return two ? launch<24, 2, 4>(stream, p) : launch<24, 1, 8>(stream, p);
    case 32: return two ? launch<32, 2, 4>(stream, p) : launch<32, 1, 8>(stream, p);
    case 48: return launch<48, 1, 8>(stream, p);
    case 64: return launch<64, 1, 8>(stream, p);
    default:
      set_error("attention_fp32: head dim %d not supported (16, 24, 32, 48, 64)", p.d);
      return KFB_ERR_UNSUPPORTED;
  }
}

}  // namespace kfb
