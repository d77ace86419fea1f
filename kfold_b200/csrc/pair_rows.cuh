// LayerNorm of the rows that a CTA's tile holds in shared memory, for the kernels that multiply them there.
#pragma once
#include <cuda_bf16.h>

#include "gemm.cuh"   // pack_bf16x2
#include "ptx.cuh"

namespace kfb {

static constexpr int kRowTile = 128;              // rows of a CTA's tile
static constexpr int kRowBox = kRowTile * 128;    // [128 rows][64 bf16], 128-byte swizzle: the tile is C / 64 of them

// A lane's eight channels' scale and offset in pairs (1 and 0 where there are none).
template <int C>
__device__ __forceinline__ void rows_affine(const float* ln_w, const float* ln_b, int lane, uint64_t (&lw)[4], uint64_t (&lb)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int ch = C == 128 ? (lane & 15) * 8 + 2 * i : (lane + 32 * i) * 2;
    lw[i] = ln_w != nullptr ? ptx::pack2(ln_w[ch], ln_w[ch + 1]) : ptx::pack2(1.0f, 1.0f);
    lb[i] = ln_b != nullptr ? ptx::pack2(ln_b[ch], ln_b[ch + 1]) : ptx::pack2(0.0f, 0.0f);
  }
}

// Rows first .. first + rows - 1 (a multiple of eight) in place, by one warp.  Lanes, expressions and their order are those of layernorm_c128_bf16_kernel and
// layernorm_c256_bf16_kernel: the same bits (four blocks of bf16 rounding turn a last bit into up to 1 % of the confidence head's result).
template <int C>
__device__ __forceinline__ void rows_layernorm(uint8_t* a, int first, int rows, int lane, const uint64_t (&lw)[4], const uint64_t (&lb)[4],
                                               float eps) {
  if constexpr (C == 128) {
    const int sub = lane & 15, half = lane >> 4;
    constexpr int kSteps = 4;        // of two rows each in flight
#pragma unroll 1
    for (int base = first; base < first + rows; base += 2 * kSteps) {
      uint64_t v[kSteps][4];
      float sum[kSteps], sq[kSteps];
      uint4* cell[kSteps];
#pragma unroll
      for (int s = 0; s < kSteps; ++s) {
        const int r = base + 2 * s + half;
        cell[s] = reinterpret_cast<uint4*>(a + (sub >> 3) * kRowBox + r * 128 + (((sub & 7) ^ (r & 7)) << 4));
        const uint4 raw = *cell[s];
        const uint32_t wv[4] = {raw.x, raw.y, raw.z, raw.w};
        sum[s] = 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          v[s][i] = ptx::pack2(wv[i] << 16, wv[i] & 0xffff0000u);
          sum[s] += __uint_as_float(wv[i] << 16) + __uint_as_float(wv[i] & 0xffff0000u);
        }
      }
#pragma unroll
      for (int m = 8; m > 0; m >>= 1)
#pragma unroll
        for (int s = 0; s < kSteps; ++s) sum[s] += __shfl_xor_sync(0xffffffffu, sum[s], m);
#pragma unroll
      for (int s = 0; s < kSteps; ++s) {
        const float mean = sum[s] * (1.0f / C);
        sq[s] = 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          v[s][i] = ptx::add2(v[s][i], ptx::pack2(-mean, -mean));
          const float2 d = ptx::unpack2(v[s][i]);
          sq[s] = fmaf(d.x, d.x, sq[s]);
          sq[s] = fmaf(d.y, d.y, sq[s]);
        }
      }
#pragma unroll
      for (int m = 8; m > 0; m >>= 1)
#pragma unroll
        for (int s = 0; s < kSteps; ++s) sq[s] += __shfl_xor_sync(0xffffffffu, sq[s], m);
#pragma unroll
      for (int s = 0; s < kSteps; ++s) {
        const float rstd = rsqrtf(sq[s] * (1.0f / C) + eps);
        uint32_t ov[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 y = ptx::unpack2(ptx::fma2(ptx::mul2(v[s][i], ptx::pack2(rstd, rstd)), lw[i], lb[i]));
          ov[i] = pack_bf16x2(y.x, y.y);
        }
        *cell[s] = make_uint4(ov[0], ov[1], ov[2], ov[3]);
      }
    }
  } else {
    constexpr int kStep = 4;         // rows in flight
#pragma unroll 1
    for (int base = first; base < first + rows; base += kStep) {
      uint64_t v[kStep][4];
      float s[kStep], q[kStep];
      uint32_t* cell[kStep];
#pragma unroll
      for (int r = 0; r < kStep; ++r) {
        cell[r] = reinterpret_cast<uint32_t*>(a + (base + r) * 128 + (((lane >> 2) ^ ((base + r) & 7)) << 4) + (lane & 3) * 4);
        s[r] = 0.f;
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          const uint32_t u = cell[r][g * (kRowBox / 4)];
          v[r][g] = ptx::pack2(u << 16, u & 0xffff0000u);
          s[r] += __uint_as_float(u << 16) + __uint_as_float(u & 0xffff0000u);
        }
      }
#pragma unroll
      for (int m = 16; m > 0; m >>= 1)
#pragma unroll
        for (int r = 0; r < kStep; ++r) s[r] += __shfl_xor_sync(0xffffffffu, s[r], m);
#pragma unroll
      for (int r = 0; r < kStep; ++r) {
        const float mean = s[r] / static_cast<float>(C);
        q[r] = 0.f;
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          v[r][g] = ptx::add2(v[r][g], ptx::pack2(-mean, -mean));
          const float2 d = ptx::unpack2(v[r][g]);
          q[r] += d.x * d.x + d.y * d.y;
        }
      }
#pragma unroll
      for (int m = 16; m > 0; m >>= 1)
#pragma unroll
        for (int r = 0; r < kStep; ++r) q[r] += __shfl_xor_sync(0xffffffffu, q[r], m);
#pragma unroll
      for (int r = 0; r < kStep; ++r) {
        const float rstd = rsqrtf(q[r] / static_cast<float>(C) + eps);
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          const float2 y = ptx::unpack2(ptx::fma2(ptx::mul2(v[r][g], ptx::pack2(rstd, rstd)), lw[g], lb[g]));
          cell[r][g * (kRowBox / 4)] = pack_bf16x2(y.x, y.y);
        }
      }
    }
  }
}

}  // namespace kfb
