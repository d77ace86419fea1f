// LayerNorm of the rows that a CTA's tile holds in shared memory, for the kernels that multiply them there.
#pragma once
#include <cuda_bf16.h>

#include "gemm.cuh"   // pack_bf16x2

namespace kfb {

static constexpr int kRowTile = 128;              // rows of a CTA's tile
static constexpr int kRowBox = kRowTile * 128;    // [128 rows][64 bf16], 128-byte swizzle: the tile is C / 64 of them

// A lane's eight channels' scale and offset (1 and 0 where there are none).
template <int C>
__device__ __forceinline__ void rows_affine(const float* ln_w, const float* ln_b, int lane, float (&lw)[8], float (&lb)[8]) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int ch = C == 128 ? (lane & 15) * 8 + i : (lane + 32 * (i >> 1)) * 2 + (i & 1);
    lw[i] = ln_w != nullptr ? ln_w[ch] : 1.0f;
    lb[i] = ln_b != nullptr ? ln_b[ch] : 0.0f;
  }
}

// Rows first .. first + rows - 1 (a multiple of eight) in place, by one warp.  Lanes, expressions and their order are those of layernorm_c128_bf16_kernel and
// layernorm_c256_bf16_kernel: the same bits (four blocks of bf16 rounding turn a last bit into up to 1 % of the confidence head's result).
template <int C>
__device__ __forceinline__ void rows_layernorm(uint8_t* a, int first, int rows, int lane, const float (&lw)[8], const float (&lb)[8], float eps) {
  constexpr int kPer = C == 128 ? 8 : 4;       // channels, or channel pairs, of a lane
  if constexpr (C == 128) {
    const int sub = lane & 15, half = lane >> 4;
    constexpr int kSteps = 4;        // of two rows each in flight
#pragma unroll 1
    for (int base = first; base < first + rows; base += 2 * kSteps) {
      float v[kSteps][8], sum[kSteps], sq[kSteps];
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
          v[s][2 * i] = __uint_as_float(wv[i] << 16);
          v[s][2 * i + 1] = __uint_as_float(wv[i] & 0xffff0000u);
          sum[s] += v[s][2 * i] + v[s][2 * i + 1];
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
        for (int i = 0; i < 8; ++i) {
          v[s][i] -= mean;
          sq[s] = fmaf(v[s][i], v[s][i], sq[s]);
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
        for (int i = 0; i < 4; ++i)
          ov[i] = pack_bf16x2(fmaf(v[s][2 * i] * rstd, lw[2 * i], lb[2 * i]), fmaf(v[s][2 * i + 1] * rstd, lw[2 * i + 1], lb[2 * i + 1]));
        *cell[s] = make_uint4(ov[0], ov[1], ov[2], ov[3]);
      }
    }
  } else {
    constexpr int kStep = 4;         // rows in flight
#pragma unroll 1
    for (int base = first; base < first + rows; base += kStep) {
      float2 v[kStep][kPer];
      float s[kStep], q[kStep];
      uint32_t* cell[kStep];
#pragma unroll
      for (int r = 0; r < kStep; ++r) {
        cell[r] = reinterpret_cast<uint32_t*>(a + (base + r) * 128 + (((lane >> 2) ^ ((base + r) & 7)) << 4) + (lane & 3) * 4);
        s[r] = 0.f;
#pragma unroll
        for (int g = 0; g < kPer; ++g) {
          const uint32_t u = cell[r][g * (kRowBox / 4)];
          v[r][g] = make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u));
          s[r] += v[r][g].x + v[r][g].y;
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
        for (int g = 0; g < kPer; ++g) {
          v[r][g].x -= mean;
          v[r][g].y -= mean;
          q[r] += v[r][g].x * v[r][g].x + v[r][g].y * v[r][g].y;
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
        for (int g = 0; g < kPer; ++g)
          cell[r][g * (kRowBox / 4)] = pack_bf16x2(fmaf(v[r][g].x * rstd, lw[2 * g], lb[2 * g]), fmaf(v[r][g].y * rstd, lw[2 * g + 1], lb[2 * g + 1]));
      }
    }
  }
}

}  // namespace kfb
