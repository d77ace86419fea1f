// fp32 attention with pair bias and key mask for the fp32-accurate mode.
//
// CUDA cores, float32 throughout, an online softmax (the L x L x H logits are never stored).  Same semantics as attention.cu:
// additive pair bias, masked keys get -1e9 (finite, as the reference does), optional sigmoid gate, and the result is written as the
// bf16 triple split (an A operand's row, see part_a) that the fp32-accurate output projection consumes.
//
// Few rows (attention_fp32_kernel): a block takes 16 queries of one head, two lanes a row, and splits the keys over its eight warps, eight keys
// at a time; where there are enough blocks without it, 64 queries, two rows a lane, over four warps.  The warps' (maximum, sum, accumulator)
// are merged at the end.  The single-track problems (a few hundred queries, one batch entry, 16 heads) have too few rows to fill the chip
// with one thread per row and all keys each: 301 queries x 16 heads x 48 took 250 us that way.  A warp stages its own keys in a two-slot ring
// with cp.async, so nothing but the merge waits for another warp; K and V are read as broadcast 16-byte pieces, which bounds the loop.
// Many rows: attention_fp32_rows_kernel below.
#include "attention.cuh"
#include "gemm.cuh"  // part_a
#include "ptx.cuh"

#include <mutex>

namespace kfb {
namespace {

constexpr int kKeys = 8;    // keys per warp and step

using ptx::fma2;
using ptx::mul2;

template <int D, int QPT, int LPR, int kWarps>
struct F32Cfg {
  static constexpr int kQ = 32 / LPR * QPT;
  static constexpr int kPitch = LPR == 2 ? D + 4 : D;                  // a row's halves 4 banks apart
  static constexpr int kRing = kWarps * 2 * 2 * kKeys * kPitch;        // floats: [warp][slot][K | V][key][kPitch]
  static constexpr int kMerge = (kWarps / 2) * kQ * (D + 1);           // the same memory after the loop
  static constexpr int kMain = kRing > kMerge ? kRing : kMerge;
  static constexpr int kBias = kWarps * kQ * (kKeys + 1);
  static constexpr int kSmem = (kMain + kBias + 2 * kWarps * kQ) * 4;
};

template <int D, int QPT, int LPR, int kWarps>
__global__ void __launch_bounds__(kWarps * 32, LPR == 2 ? 2 : 1) attention_fp32_kernel(const AttnFp32Params p) {
  using Cfg = F32Cfg<D, QPT, LPR, kWarps>;
  constexpr int kQ = Cfg::kQ, kPitch = Cfg::kPitch, kL = 32 / LPR, DL = D / LPR;    // rows side by side in a warp, channels of a lane
  grid_dependency_enter();
  extern __shared__ __align__(16) float smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, lrow = lane % kL, part = lane / kL;
  float* ring = smem + warp * (4 * kKeys * kPitch);
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

  uint64_t q[QPT][DL / 2], acc2[QPT][DL / 2];      // pairs of neighbouring channels
  float m_run[QPT], l_run[QPT];
#pragma unroll
  for (int i = 0; i < QPT; ++i) {
    const long long row = static_cast<long long>(b) * p.lq + min(q0 + i * kL + lrow, p.lq - 1);
    const ulonglong2* src = reinterpret_cast<const ulonglong2*>(p.q + row * p.ld + p.q_col0 + h * D + part * DL);
#pragma unroll
    for (int d = 0; d < DL / 4; ++d) {
      const ulonglong2 f = src[d];
      q[i][2 * d] = f.x;
      q[i][2 * d + 1] = f.y;
    }
#pragma unroll
    for (int d = 0; d < DL / 2; ++d) acc2[i][d] = 0;
    m_run[i] = -INFINITY;
    l_run[i] = 0.f;
  }

  const int groups = (p.lk + kKeys - 1) / kKeys;
  // bias and mask of a group are fetched a step ahead: lane = (row of four, key), which reads whole sectors
  constexpr int kFetch = kQ / 4;
  float bias_r[kFetch], mask_r = 0.f;
  auto fetch = [&](int g, int slot) {
    float* dst = ring + slot * (2 * kKeys * kPitch);
#pragma unroll
    for (int idx = lane; idx < kKeys * D / 4; idx += 32) {
      const int kk = idx / (D / 4), c = idx - kk * (D / 4);
      const long long off = static_cast<long long>(min(g * kKeys + kk, p.lk - 1)) * ld_kv + c * 4;
      const int at = kk * kPitch + c * 4 + (LPR == 2 && c >= DL / 4 ? 4 : 0);
      ptx::cp_async_16(dst + at, k_base + off);
      ptx::cp_async_16(dst + kKeys * kPitch + at, v_base + off);
    }
    const int key = g * kKeys + (lane & 7);
    mask_r = key < p.lk ? ((mrow == nullptr || mrow[static_cast<long long>(key) * p.m_k]) ? 0.f : -1e9f) : -INFINITY;
#pragma unroll
    for (int i = 0; i < kFetch; ++i) {
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
    for (int i = 0; i < kFetch; ++i) s_bias[(i * 4 + (lane >> 3)) * (kKeys + 1) + (lane & 7)] = bias_r[i];
    if (g + kWarps < groups) fetch(g + kWarps, slot ^ 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();
    const ulonglong2* sk = reinterpret_cast<const ulonglong2*>(ring + slot * (2 * kKeys * kPitch) + part * (DL + 4));
    const ulonglong2* sv = sk + kKeys * kPitch / 4;
    uint64_t s2[QPT][kKeys];
#pragma unroll
    for (int i = 0; i < QPT; ++i)
#pragma unroll
      for (int kk = 0; kk < kKeys; ++kk) s2[i][kk] = 0;
#pragma unroll
    for (int d = 0; d < DL / 4; ++d)
#pragma unroll
      for (int kk = 0; kk < kKeys; ++kk) {
        const ulonglong2 f = sk[kk * (kPitch / 4) + d];
#pragma unroll
        for (int i = 0; i < QPT; ++i) {
          s2[i][kk] = fma2(q[i][2 * d], f.x, s2[i][kk]);
          s2[i][kk] = fma2(q[i][2 * d + 1], f.y, s2[i][kk]);
        }
      }
    float s[QPT][kKeys];
#pragma unroll
    for (int i = 0; i < QPT; ++i) {
      float mx = -INFINITY;
#pragma unroll
      for (int kk = 0; kk < kKeys; ++kk) {
        // same order of additions as the reference: (q k + mask) + bias
        const float2 f = ptx::unpack2(s2[i][kk]);
        float qk = f.x + f.y;
        if constexpr (LPR == 2) qk += __shfl_xor_sync(0xffffffffu, qk, kL);
        s[i][kk] = (qk + __shfl_sync(0xffffffffu, mask_v, kk)) + s_bias[(i * kL + lrow) * (kKeys + 1) + kk];
        mx = fmaxf(mx, s[i][kk]);
      }
      const float m_new = fmaxf(m_run[i], mx);
      const float alpha = expf(m_run[i] - m_new);
      const uint64_t a2 = ptx::pack2(alpha, alpha);
      l_run[i] *= alpha;
#pragma unroll
      for (int d = 0; d < DL / 2; ++d) acc2[i][d] = mul2(acc2[i][d], a2);
#pragma unroll
      for (int kk = 0; kk < kKeys; ++kk) {
        s[i][kk] = expf(s[i][kk] - m_new);
        l_run[i] += s[i][kk];
      }
      m_run[i] = m_new;
    }
#pragma unroll
    for (int kk = 0; kk < kKeys; ++kk) {
      uint64_t p2[QPT];
#pragma unroll
      for (int i = 0; i < QPT; ++i) p2[i] = ptx::pack2(s[i][kk], s[i][kk]);
#pragma unroll
      for (int d = 0; d < DL / 4; ++d) {
        const ulonglong2 f = sv[kk * (kPitch / 4) + d];
#pragma unroll
        for (int i = 0; i < QPT; ++i) {
          acc2[i][2 * d] = fma2(p2[i], f.x, acc2[i][2 * d]);
          acc2[i][2 * d + 1] = fma2(p2[i], f.y, acc2[i][2 * d + 1]);
        }
      }
    }
    __syncwarp();   // the slot and the bias tile may be written again
  }

  float acc[QPT][DL];
#pragma unroll
  for (int i = 0; i < QPT; ++i)
#pragma unroll
    for (int d = 0; d < DL / 2; ++d) {
      const float2 f = ptx::unpack2(acc2[i][d]);
      acc[i][2 * d] = f.x;
      acc[i][2 * d + 1] = f.y;
    }

  // merge the warps' softmax states; a warp without keys has m = -inf, l = 0
#pragma unroll
  for (int i = 0; i < QPT; ++i) {
    s_m[warp * kQ + i * kL + lrow] = m_run[i];
    s_l[warp * kQ + i * kL + lrow] = l_run[i];
  }
  __syncthreads();
  float inv_l[QPT];
#pragma unroll
  for (int i = 0; i < QPT; ++i) {
    float m = -INFINITY, l = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) m = fmaxf(m, s_m[w * kQ + i * kL + lrow]);
#pragma unroll
    for (int w = 0; w < kWarps; ++w) l += s_l[w * kQ + i * kL + lrow] * expf(s_m[w * kQ + i * kL + lrow] - m);
    inv_l[i] = 1.0f / l;
    const float scale = expf(m_run[i] - m);
#pragma unroll
    for (int d = 0; d < DL; ++d) acc[i][d] *= scale;
  }
#pragma unroll 1
  for (int half = kWarps / 2; half >= 1; half >>= 1) {
    if (warp >= half && warp < 2 * half) {
#pragma unroll
      for (int i = 0; i < QPT; ++i)
#pragma unroll
        for (int d = 0; d < DL; ++d) smem[((warp - half) * kQ + i * kL + lrow) * (D + 1) + part * DL + d] = acc[i][d];
    }
    __syncthreads();
    if (warp < half) {
#pragma unroll
      for (int i = 0; i < QPT; ++i)
#pragma unroll
        for (int d = 0; d < DL; ++d) acc[i][d] += smem[(warp * kQ + i * kL + lrow) * (D + 1) + part * DL + d];
    }
    __syncthreads();
  }
  if (warp == 0) {
#pragma unroll
    for (int i = 0; i < QPT; ++i)
#pragma unroll
      for (int d = 0; d < DL; ++d) smem[(i * kL + lrow) * (D + 1) + part * DL + d] = acc[i][d] * inv_l[i];
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

// ------------------------------------------------------------------------------------------------
// Many rows (triangle attention): nothing split, nothing merged.
//
// The kernel above gives a warp of 160 keys forty, and then loads of queries, the merge and 2-byte stores are most of its time: 164 us for
// 160 x 160 rows of 4 heads, of which the multiply-adds take 28.  Here a block has 64 or 128 queries of one row and head, 64 for each warp
// (two rows a lane), and all keys go by in tiles of 32 that its warps share: one broadcast load of 16 bytes feeds eight multiply-adds of a
// row pair, issued two at a time (fma.rn.f32x2: the same IEEE operations, sums over even and over odd channels added at the end).  The bias
// comes with the keys by cp.async, 36 floats a row so that a lane's 16-byte pieces of its own row meet no bank conflict.
// Sums over keys are of eight by themselves, then added to the row's: in one accumulator for all keys the operator's error against 64 bits
// was 5.6e-7 at 160 tokens and 6.4e-7 at 400 (root mean square of the result), with the split keys above 5.1e-7 and 5.2e-7, and is 5.05e-7 and
// 5.15e-7 so, for 1 to 4 % of the time.
// Measured (events, 4 heads of 32): 96 x 96 rows 54 -> 39 us, 128 x 128 82 -> 52, 160 x 160 150 -> 107, 200 x 200 298 -> 185, 256 x 256 461 -> 261.
constexpr int kTile = 32, kBiasPitch = 36, kRowsWarp = 64;

__device__ __forceinline__ void cp_async4(void* smem, const void* gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(ptx::smem_u32(smem)), "l"(gmem) : "memory");
}

template <int D>
constexpr int rows_smem(int warps) { return 2 * (2 * kTile * D + warps * kRowsWarp * kBiasPitch + kTile) * 4; }

template <int D, int W>
__global__ void __launch_bounds__(W * 32, 8 / W) attention_fp32_rows_kernel(const AttnFp32Params p, int bias_vec) {
  grid_dependency_enter();
  extern __shared__ __align__(16) float smem[];
  constexpr int threads = W * 32, rows = threads * 2;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* s_kv = smem;                                   // [slot][K | V][key][D]
  float* s_bias = s_kv + 2 * 2 * kTile * D;             // [slot][query][kBiasPitch]
  float* s_mask = s_bias + 2 * rows * kBiasPitch;       // [slot][key]
  const int q0 = blockIdx.x * rows, h = blockIdx.y, b = blockIdx.z;
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

  // keys of a tile past the last are copies of it (masked), queries past the last copies of that one (not stored)
  auto fetch = [&](int k0, int slot) {
    float* kv = s_kv + slot * (2 * kTile * D);
    for (int idx = threadIdx.x; idx < kTile * D / 4; idx += threads) {
      const int kk = idx / (D / 4), c = idx - kk * (D / 4);
      const long long off = static_cast<long long>(min(k0 + kk, p.lk - 1)) * ld_kv + c * 4;
      ptx::cp_async_16(kv + idx * 4, k_base + off);
      ptx::cp_async_16(kv + kTile * D + idx * 4, v_base + off);
    }
    float* bias = s_bias + slot * rows * kBiasPitch;
    if (bias_vec && k0 + kTile <= p.lk) {
      for (int idx = threadIdx.x; idx < rows * (kTile / 4); idx += threads) {
        const int row = idx >> 3, c = idx & 7;
        if (q0 + row < p.lq) ptx::cp_async_16(bias + row * kBiasPitch + c * 4, bias_base + static_cast<long long>(q0 + row) * p.ldb + k0 + c * 4);
      }
    } else {
      for (int idx = threadIdx.x; idx < rows * kTile; idx += threads) {
        const int row = idx >> 5, c = idx & 31;
        if (q0 + row < p.lq && k0 + c < p.lk)
          cp_async4(bias + row * kBiasPitch + c, bias_base + static_cast<long long>(q0 + row) * p.ldb + k0 + c);
        else
          bias[row * kBiasPitch + c] = 0.f;
      }
    }
    if (threadIdx.x < kTile) {
      const int key = k0 + threadIdx.x;
      s_mask[slot * kTile + threadIdx.x] = key < p.lk ? ((mrow == nullptr || mrow[static_cast<long long>(key) * p.m_k]) ? 0.f : -1e9f) : -INFINITY;
    }
  };
  fetch(0, 0);
  asm volatile("cp.async.commit_group;" ::: "memory");

  const int row0 = q0 + warp * kRowsWarp + lane;          // this lane's rows: row0 and row0 + 32
  const bool busy = q0 + warp * kRowsWarp < p.lq;         // (of the warp)
  uint64_t q[2][D / 2], acc[2][D / 2];
  float m_run[2], l_run[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const long long row = static_cast<long long>(b) * p.lq + min(row0 + 32 * i, p.lq - 1);
    const ulonglong2* src = reinterpret_cast<const ulonglong2*>(p.q + row * p.ld + p.q_col0 + h * D);
#pragma unroll
    for (int d = 0; d < D / 4; ++d) {
      const ulonglong2 f = src[d];
      q[i][2 * d] = f.x;
      q[i][2 * d + 1] = f.y;
    }
#pragma unroll
    for (int d = 0; d < D / 2; ++d) acc[i][d] = 0;
    m_run[i] = -INFINITY;
    l_run[i] = 0.f;
  }

  int slot = 0;
  for (int k0 = 0; k0 < p.lk; k0 += kTile, slot ^= 1) {
    if (k0 + kTile < p.lk) fetch(k0 + kTile, slot ^ 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    const int groups = min(kTile / kKeys, (p.lk - k0 + kKeys - 1) / kKeys);
    for (int g = 0; busy && g < groups; ++g) {
      const ulonglong2* sk = reinterpret_cast<const ulonglong2*>(s_kv + slot * (2 * kTile * D)) + g * kKeys * (D / 4);
      const ulonglong2* sv = sk + kTile * D / 4;
      const float* bias = s_bias + (slot * rows + warp * kRowsWarp + lane) * kBiasPitch + g * kKeys;
      const float* mask = s_mask + slot * kTile + g * kKeys;
      uint64_t s2[2][kKeys];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int kk = 0; kk < kKeys; ++kk) s2[i][kk] = 0;
#pragma unroll
      for (int d = 0; d < D / 4; ++d)
#pragma unroll
        for (int kk = 0; kk < kKeys; ++kk) {
          const ulonglong2 f = sk[kk * (D / 4) + d];
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            s2[i][kk] = fma2(q[i][2 * d], f.x, s2[i][kk]);
            s2[i][kk] = fma2(q[i][2 * d + 1], f.y, s2[i][kk]);
          }
        }
      float s[2][kKeys], m_new[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        float bv[kKeys];
#pragma unroll
        for (int c = 0; c < kKeys / 4; ++c) {
          const float4 f = *reinterpret_cast<const float4*>(bias + i * 32 * kBiasPitch + c * 4);
          bv[4 * c] = f.x; bv[4 * c + 1] = f.y; bv[4 * c + 2] = f.z; bv[4 * c + 3] = f.w;
        }
        m_new[i] = m_run[i];
#pragma unroll
        for (int kk = 0; kk < kKeys; ++kk) {
          const float2 f = ptx::unpack2(s2[i][kk]);
          // same order of additions as the reference: (q k + mask) + bias
          s[i][kk] = ((f.x + f.y) + mask[kk]) + bv[kk];
          m_new[i] = fmaxf(m_new[i], s[i][kk]);
        }
      }
      if (__any_sync(0xffffffffu, m_new[0] > m_run[0] || m_new[1] > m_run[1])) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const float alpha = expf(m_run[i] - m_new[i]);
          const uint64_t a2 = ptx::pack2(alpha, alpha);
          l_run[i] *= alpha;
#pragma unroll
          for (int d = 0; d < D / 2; ++d) acc[i][d] = mul2(acc[i][d], a2);
          m_run[i] = m_new[i];
        }
      }
      // eight keys by themselves: 512 are 64 + 8 roundings of a sum, not 512
      uint64_t p2[2][kKeys];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        float sum = 0.f;
#pragma unroll
        for (int kk = 0; kk < kKeys; ++kk) {
          s[i][kk] = expf(s[i][kk] - m_run[i]);
          sum += s[i][kk];
          p2[i][kk] = ptx::pack2(s[i][kk], s[i][kk]);
        }
        l_run[i] += sum;
      }
#pragma unroll
      for (int d = 0; d < D / 4; ++d) {
        uint64_t t[2][2];
#pragma unroll
        for (int kk = 0; kk < kKeys; ++kk) {
          const ulonglong2 f = sv[kk * (D / 4) + d];
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            t[i][0] = kk == 0 ? mul2(p2[i][kk], f.x) : fma2(p2[i][kk], f.x, t[i][0]);
            t[i][1] = kk == 0 ? mul2(p2[i][kk], f.y) : fma2(p2[i][kk], f.y, t[i][1]);
          }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          acc[i][2 * d] = ptx::add2(acc[i][2 * d], t[i][0]);
          acc[i][2 * d + 1] = ptx::add2(acc[i][2 * d + 1], t[i][1]);
        }
      }
    }
    __syncthreads();      // the slot may be written again
  }

  const int hd = p.heads * D;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    if (row0 + 32 * i >= p.lq) continue;
    const long long qrow = static_cast<long long>(b) * p.lq + row0 + 32 * i;
    const float inv_l = 1.0f / l_run[i];
    __nv_bfloat16* o6 = p.out6 + qrow * 6 * hd + h * D;
#pragma unroll
    for (int d0 = 0; d0 < D; d0 += 8) {
      float o[8];
#pragma unroll
      for (int d = 0; d < 4; ++d) {
        const float2 f = ptx::unpack2(acc[i][d0 / 2 + d]);
        o[2 * d] = f.x * inv_l;
        o[2 * d + 1] = f.y * inv_l;
      }
      if (p.g != nullptr) {
        const float4* g = reinterpret_cast<const float4*>(p.g + qrow * p.ld + p.g_col0 + h * D + d0);
        const float4 lo = g[0], hi = g[1];
        const float gv[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
        for (int d = 0; d < 8; ++d) o[d] *= 1.0f / (1.0f + expf(-gv[d]));
      }
      uint32_t w[3][4];
#pragma unroll
      for (int d = 0; d < 4; ++d) {
        __nv_bfloat16 x[2][3];
        split3(o[2 * d], x[0][0], x[0][1], x[0][2]);
        split3(o[2 * d + 1], x[1][0], x[1][1], x[1][2]);
#pragma unroll
        for (int part = 0; part < 3; ++part)
          w[part][d] = static_cast<uint32_t>(__bfloat16_as_ushort(x[0][part])) | (static_cast<uint32_t>(__bfloat16_as_ushort(x[1][part])) << 16);
      }
#pragma unroll
      for (int part = 0; part < 3; ++part)
        *reinterpret_cast<uint4*>(o6 + part_a(part) * hd + d0) = make_uint4(w[part][0], w[part][1], w[part][2], w[part][3]);
    }
  }
}

template <int D, int W>
int launch_rows(cudaStream_t stream, const AttnFp32Params& p, int bias_vec) {
  static std::once_flag once[64];
  int dev = 0;
  KFB_CUDA(cudaGetDevice(&dev));
  cudaError_t attr_err = cudaSuccess;
  std::call_once(once[dev & 63], [&] {
    attr_err = cudaFuncSetAttribute(attention_fp32_rows_kernel<D, W>, cudaFuncAttributeMaxDynamicSharedMemorySize, rows_smem<D>(W));
  });
  KFB_CUDA(attr_err);
  LaunchScope scope(stream, p.tag ? p.tag : "attention_fp32");
  return launch_kernel(stream, attention_fp32_rows_kernel<D, W>, dim3(cdiv(p.lq, W * kRowsWarp), p.heads, p.batch), W * 32, rows_smem<D>(W), p, bias_vec);
}
template <int D>
int launch_rows(cudaStream_t stream, const AttnFp32Params& p) {
  const int bias_vec = (reinterpret_cast<uintptr_t>(p.bias) & 15) == 0 && p.ldb % 4 == 0 && (p.bias_hs > 0 ? p.bias_hs : p.lq * p.ldb) % 4 == 0;
  // two warps share a tile's copies; one where the second would have nothing to do in every other block (with one accumulator, 160 rows: 117 us
  // with two, 105 with one; 128: 50, 60; four: 80 and 118)
  const int tiles = cdiv(p.lq, kRowsWarp);
  return tiles == 1 || tiles == 3 ? launch_rows<D, 1>(stream, p, bias_vec) : launch_rows<D, 2>(stream, p, bias_vec);
}

// The operands' rows by 16 bytes, and two (entry, head) problems for every multiprocessor at least: below that (single-track problems) the keys
// of a row have to be split to fill the chip, and a warp of fewer than 48 rows wastes more than the split costs.
bool takes_rows(const AttnFp32Params& p) {
  const long long ld_kv = p.ld_kv > 0 ? p.ld_kv : p.ld;
  const uintptr_t all = reinterpret_cast<uintptr_t>(p.q) | reinterpret_cast<uintptr_t>(p.k) | reinterpret_cast<uintptr_t>(p.v) |
                        reinterpret_cast<uintptr_t>(p.g) | reinterpret_cast<uintptr_t>(p.out6);
  return p.lq >= 48 && static_cast<long long>(p.batch) * p.heads >= 2ll * sm_count() && (all & 15) == 0 && p.ld % 4 == 0 && ld_kv % 4 == 0 &&
         p.q_col0 % 4 == 0 && p.k_col0 % 4 == 0 && p.v_col0 % 4 == 0 && (p.g == nullptr || p.g_col0 % 4 == 0) && (p.heads * p.d) % 8 == 0;
}

template <int D, int QPT, int LPR, int kWarps>
int launch(cudaStream_t stream, const AttnFp32Params& p) {
  using Cfg = F32Cfg<D, QPT, LPR, kWarps>;
  static std::once_flag once[64];
  int dev = 0;
  KFB_CUDA(cudaGetDevice(&dev));
  cudaError_t attr_err = cudaSuccess;
  std::call_once(once[dev & 63], [&] {
    attr_err = cudaFuncSetAttribute(attention_fp32_kernel<D, QPT, LPR, kWarps>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmem);
  });
  KFB_CUDA(attr_err);
  LaunchScope scope(stream, p.tag ? p.tag : "attention_fp32");
  const dim3 grid(cdiv(p.lq, Cfg::kQ), p.heads, p.batch);
  KFB_TRY(launch_kernel(stream, attention_fp32_kernel<D, QPT, LPR, kWarps>, grid, kWarps * 32, Cfg::kSmem, p));
  return KFB_OK;
}

}  // namespace

int launch_attention_fp32(cudaStream_t stream, const AttnFp32Params& p) {
  KFB_CHECK_ARG(p.batch > 0 && p.heads > 0 && p.lq > 0 && p.lk > 0, "attention_fp32: empty problem");
  KFB_CHECK_ARG(p.batch <= 65535 && p.heads <= 65535, "attention_fp32: batch %d / heads %d exceed the grid limits", p.batch, p.heads);
  // two query rows per lane: half the shared-memory reads per row, but half the blocks (and registers for head dims up to 32 only);
  // with that many blocks four warps share the keys, which halves what is merged (160 x 160 rows: 180 us with eight)
  const bool two = p.lq > 32 && static_cast<long long>(cdiv(p.lq, 64)) * p.heads * p.batch >= 2ll * sm_count();
  if (takes_rows(p)) {
    switch (p.d) {
      case 16: return launch_rows<16>(stream, p);
      case 24: return launch_rows<24>(stream, p);
      case 32: return launch_rows<32>(stream, p);
      default: break;
    }
  }
  switch (p.d) {
    case 16: return two ? launch<16, 2, 1, 4>(stream, p) : launch<16, 1, 2, 8>(stream, p);
    case 24: return two ? launch<24, 2, 1, 4>(stream, p) : launch<24, 1, 2, 8>(stream, p);
    case 32: return two ? launch<32, 2, 1, 4>(stream, p) : launch<32, 1, 2, 8>(stream, p);
    case 48: return launch<48, 1, 2, 8>(stream, p);
    case 64: return launch<64, 1, 2, 8>(stream, p);
    default:
      set_error("attention_fp32: head dim %d not supported (16, 24, 32, 48, 64)", p.d);
      return KFB_ERR_UNSUPPORTED;
  }
}

}  // namespace kfb
