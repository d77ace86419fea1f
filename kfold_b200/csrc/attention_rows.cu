// Attention of batch entries that share their bias (see attention.cuh for the operator): triangle attention over pair rows, head dim
// <= 32, and the token transformer's samples, head dim <= 64.  A persistent kernel whose time is the softmax warps'.
//
// What bounds it.  A 128 x 64 tile of logits is 8 192 exponentials, 512 cycles of the SM's MUFU.  The kernel of attention.cu (two
// CTAs per SM, eight softmax warps each, a thread per row and 32 keys) took 1 100 cycles per tile plus 9 000 per CTA of fill and
// drain: around the 256 cycles of exponentials of 32 x 32 logits a warp spends 600 to 800 on bias loads, waits, votes and
// tensor-memory round trips, and warps that share barriers spend them at the same time.  Here:
//   * the bias, in log2 units, is added by the tensor core (bias tile x identity, accumulated under Q K^T in float32), so a softmax
//     thread does nothing per logit but exp2, a sum and half a conversion: 1 080 -> 910 cycles per tile;
//   * S runs two tiles ahead of the softmax in two buffers per row group: with one, the S of a group waited 1 200 to 2 000 cycles
//     behind the other groups' products on the one tensor core (910 -> 800);
//   * R row groups (pair rows with the same bias tile) per CTA, four softmax warps each, that share nothing but the ring of operand
//     tiles; one thread owns a query row and all 64 keys of a tile, so waits and arrivals come once per 64 keys;
//   * the groups take turns: at most R - 1 of them do their exponentials at a time, while the other one waits, loads, stores and
//     arrives.  Left alone, groups that are released by the same stage run in step (clock stamps, R = 3: all of them in 1 640 of a
//     tile's 2 400 cycles of exponentials, at the MUFU's rate, then all of them in 760 cycles of round trips).  Both halves of a
//     row's S are loaded before its turn, and one vote per tile decides about the stabiliser.  N = 251: 53.5 -> 48.6 us, 768: 660 ->
//     655, 2048: 12.3 -> 12.0 ms; 5 x 768 samples of 48-wide heads: 42.5 -> 40.5 us.  (One group at a time: 765 us at N = 768, as one
//     warp needs 14 cycles an exponential, not 8.  Loads ahead without turns: 700.  An eighth of the exponentials as polynomials on
//     the FMA pipe: another 0.5 %; a quarter: slower.)
//   * the stabiliser is zero unless a row needs another one: logits are in log2 units, and exp2(x) of a row whose first keys' sum
//     lies in [2^-40, 2^100] and whose later sums stay below 2^100 neither overflows nor loses accuracy, so the common path
//     subtracts nothing and keeps no maximum;
//   * the CTA is persistent over (R rows, head, 128 queries): loads and the first S of the next item run under the output of the
//     previous one;
//   * the key mask costs nothing where it masks nothing: a row's first masked and last valid key come from a scan kernel, the rank-1
//     mask product is issued for the tiles that hold masked keys, and tiles after the last valid key are skipped.
// N = 768 (4 heads): 1.15 -> 0.69 ms; N = 2048: 18.3 -> 11.4 ms (the exponentials alone: 0.40, 7.6), 790 cycles a tile.  The MUFU is
// busy 59 % of a launch at N = 768 (ncu); without exponentials a tile still takes 660 cycles, and neither the bias nor the value
// products change that.
// Warps: 4 g .. 4 g + 3 softmax and output of row group g (a warp reads the tensor-memory lanes warp % 4); then the TMA producer, which
// also writes the mask operands, and one MMA-issuing warp per group.
// Tensor memory per row group: two S tiles, 64 fp32 columns each, overwritten in place by their P (64 bf16 = 32 columns), and O, 32
// fp32 columns.
#include <cuda_bf16.h>

#include <mutex>
#include <type_traits>

#include "attention.cuh"
#include "gemm.cuh"  // sigmoidf_fast, pack_bf16x2
#include "ptx.cuh"

namespace kfb {
namespace {

constexpr int kQ = 128;            // queries per row group
constexpr int kT = 64;             // keys per tile
constexpr int kBiasBytes = kQ * kT * 2;
constexpr int kMaskBytes = kT * 32;            // a 64 x 16 bf16 K-major operand without swizzle
constexpr int kE0Bytes = kQ * 32;
constexpr int kEyeBytes = (48 + 16 + 48) * 32; // a 16 x 16 identity (times a factor) between 48 zero rows on either side: the four K
                                               // steps of a 64 x 64 one

// R row groups, padded head dim D (32 or 64)
template <int R, int D>
struct RowsCfg {
  static constexpr int kSoftWarps = 4 * R;
  static constexpr int kThreads = 32 * (kSoftWarps + 1 + R);
  static constexpr int kQBytes = kQ * D * 2, kKBytes = kT * D * 2, kVBytes = D * kT * 2;
  static constexpr int kStages = D == 64 ? 3 : (R == 3 ? 4 : 5);      // ring of tiles: bias, and K, V^T of all row groups
  static constexpr int kStageBytes = kBiasBytes + R * (kKBytes + kVBytes);
  static constexpr int kMaskSlots = R == 3 || D == 64 ? 1 : 2;   // mask operands per group (shared memory has no room for more)
  static constexpr int kTmemCols = 512;               // 128 + D per group are used: S 2 x 64, O D
  // identities: the bias of D = 32 (triangle attention) comes in log2 units; the other callers' does not, and log2(e) is applied
  // as two bf16 factors, high and low part (relative error 4e-6, below the bias' own bf16 rounding)
  static constexpr int kEyes = D == 64 ? 2 : 1;
  static constexpr int kSmem = kStages * kStageBytes + 2 * R * kQBytes + R * kMaskSlots * kMaskBytes + kE0Bytes + kEyes * kEyeBytes +
                               R * D * 4 + 1024 /*alignment*/ + 512 /*barriers*/;
  static_assert(kSmem <= 227 * 1024, "shared memory");
};
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kMasked = -1e9f * 1.4426950408889634f;   // a masked key: the reference's finite -1e9, in log2 units
constexpr float kAbsent = -1e30f;                         // keys beyond lk
constexpr float kHighSum = 1.2676506e30f;                 // 2^100: a tile's row sum above this moves the stabiliser
constexpr float kLowSum = 9.094947e-13f;                  // 2^-40: a first tile's row sum below this sets it

struct RowsParams {
  AttnParams a;
  const int2* rows;       // per batch row: (last valid key + 1, first masked key)
  int sets_per_bias;      // sets of R rows that share a bias batch: ceil(bias_div / R)
  int q_blocks, items;
};

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// One item: R consecutive rows of one bias batch, a head, 128 queries.  Everything a role needs to walk it.
template <int R>
struct Item {
  int qb, h, b0, bias_b;
  int rows;               // rows that exist (1..R); the groups past them repeat the last one and drop its result
  int first[R];           // first masked key of each row
  int tiles;              // key tiles to process; 0: no valid key in any row (the mean of V, see the output)
};
template <int R>
__device__ __forceinline__ Item<R> load_item(const RowsParams& p, int item) {
  Item<R> it;
  it.qb = item % p.q_blocks;
  const int rest = item / p.q_blocks;
  it.h = rest % p.a.heads;
  const int set = rest / p.a.heads;
  it.bias_b = set / p.sets_per_bias;
  const int in = R * (set - it.bias_b * p.sets_per_bias);
  it.b0 = it.bias_b * p.a.bias_div + in;
  it.rows = min(R, p.a.bias_div - in);
  int most = 0;
  bool empty = false;     // a row without valid keys: its result is the uniform average over all keys
#pragma unroll
  for (int g = 0; g < R; ++g) {
    const int2 r = p.rows[it.b0 + min(g, it.rows - 1)];
    it.first[g] = r.y;
    most = max(most, r.x);
    empty = empty || r.x == 0;
  }
  it.tiles = most == 0 ? 0 : ((empty ? p.a.lk : most) + kT - 1) / kT;
  return it;
}

template <int R, int kD>
__global__ void __launch_bounds__(RowsCfg<R, kD>::kThreads, 1)
attention_rows_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                      const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_b, const RowsParams p) {
  using Cfg = RowsCfg<R, kD>;
  constexpr int kQBytes = Cfg::kQBytes, kKBytes = Cfg::kKBytes, kVBytes = Cfg::kVBytes, kEyes = Cfg::kEyes;
  constexpr int kStages = Cfg::kStages, kStageBytes = Cfg::kStageBytes, kMaskSlots = Cfg::kMaskSlots;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* s_stage = smem;                                   // [stage][bias 16 KB | K0 | V0 | K1 | V1 | ...]
  uint8_t* s_q = s_stage + kStages * kStageBytes;            // [2 items][R]
  uint8_t* s_mask = s_q + 2 * R * kQBytes;                   // [R][slots]
  uint8_t* s_e0 = s_mask + R * kMaskSlots * kMaskBytes;
  uint8_t* s_eye = s_e0 + kE0Bytes;
  float* s_mean = reinterpret_cast<float*>(s_eye + kEyes * kEyeBytes); // [R][D]
  uint64_t* bars = reinterpret_cast<uint64_t*>(s_mean + R * kD);
  uint64_t* stage_full = bars;                    // [stages]
  uint64_t* stage_empty = stage_full + kStages;   // [stages]: a commit per group
  uint64_t* q_full = stage_empty + kStages;       // [2]
  uint64_t* q_empty = q_full + 2;                 // [2]: a commit per group
  uint64_t* s_full = q_empty + 2;                 // [R][2]
  uint64_t* p_ready = s_full + 2 * R;             // [R][2]: 4 warps (they can be two tiles ahead)
  uint64_t* m_full = p_ready + 2 * R;                 // [R][slots]: ring of mask operands
  uint64_t* m_empty = m_full + kMaskSlots * R;    // [R][slots]
  uint64_t* pv_done = m_empty + kMaskSlots * R;   // [R][2]
  uint64_t* turn = pv_done + 2 * R;               // [R][2 tiles][4]: a warp of the group has done a tile's exponentials
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(turn + 8 * R);
  static_assert((2 * kStages + 4 + 6 * R + 2 * kMaskSlots * R + 8 * R) * 8 + 4 <= 512, "barriers");

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int kProducer = Cfg::kSoftWarps, kMma = kProducer + 1;
  const AttnParams& a = p.a;

  if (threadIdx.x == 0) {
    ptx::prefetch_tmap(&tm_q);
    ptx::prefetch_tmap(&tm_k);
    ptx::prefetch_tmap(&tm_v);
    ptx::prefetch_tmap(&tm_b);
    for (int i = 0; i < kStages; ++i) {
      ptx::mbar_init(&stage_full[i], 1);
      ptx::mbar_init(&stage_empty[i], R);
    }
    for (int i = 0; i < 2; ++i) {
      ptx::mbar_init(&q_full[i], 1);
      ptx::mbar_init(&q_empty[i], R);
    }
    for (int i = 0; i < R; ++i) {
      ptx::mbar_init(&s_full[2 * i], 1);
      ptx::mbar_init(&s_full[2 * i + 1], 1);
      ptx::mbar_init(&p_ready[2 * i], 4);
      ptx::mbar_init(&p_ready[2 * i + 1], 4);
      ptx::mbar_init(&pv_done[2 * i], 1);
      ptx::mbar_init(&pv_done[2 * i + 1], 1);
      for (int w = 0; w < 8; ++w) ptx::mbar_init(&turn[8 * i + w], 1);
    }
    for (int i = 0; i < kMaskSlots * R; ++i) {
      ptx::mbar_init(&m_full[i], 1);
      ptx::mbar_init(&m_empty[i], 1);
    }
    ptx::fence_barrier_init();
  }
  if (warp == kMma) {
    ptx::tmem_alloc(tmem_slot, Cfg::kTmemCols);
    ptx::tmem_relinquish();
  }
  if (warp < 4) {   // constant operands: e0 (ones in column 0), the identity; the zero halves of the mask operands
    const int r = warp * 32 + lane;
    *reinterpret_cast<uint4*>(s_e0 + ptx::noswizzle_row_offset(r)) = make_uint4(0x3F80u, 0, 0, 0);
    *reinterpret_cast<uint4*>(s_e0 + ptx::noswizzle_row_offset(r) + 128) = make_uint4(0, 0, 0, 0);
    if (r < 112) {
#pragma unroll
      for (int e = 0; e < kEyes; ++e) {
        const float hi = __bfloat162float(__float2bfloat16_rn(kLog2e));
        const uint32_t one = __bfloat16_as_ushort(__float2bfloat16_rn(kEyes == 1 ? 1.f : (e == 0 ? hi : kLog2e - hi)));
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int at = r - 48 - h * 8;   // column of the row's factor within this half of the K step
          uint32_t w[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) w[i] = (at >> 1) == i ? ((at & 1) ? one << 16 : one) : 0u;
          *reinterpret_cast<uint4*>(s_eye + e * kEyeBytes + ptx::noswizzle_row_offset(r) + h * 128) = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
    }
    if (r < kT) {
#pragma unroll
      for (int u = 0; u < kMaskSlots * R; ++u) *reinterpret_cast<uint4*>(s_mask + u * kMaskBytes + ptx::noswizzle_row_offset(r) + 128) = make_uint4(0, 0, 0, 0);
    }
    ptx::fence_proxy_async_smem();
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  grid_dependency_enter();

  if (warp == kProducer) {
    // ---------------------------------------------------------------- TMA loads, and the mask operands of the tiles that hold masked
    // or absent keys.  (One warp for both: a 17th would leave the softmax warps 96 registers, as one scheduler would hold five.  A
    // tile's mask slot is free when the S before it has been computed, which is when the stage of the next tile is, too.)
    bool ok = true;
    int st = 0;
    uint32_t par = 0, k = 0;        // ring position; items so far
    uint32_t uses[R];               // mask ring position of each group
#pragma unroll
    for (int g = 0; g < R; ++g) uses[g] = 0;
    for (int item = blockIdx.x; ok && item < p.items; item += gridDim.x) {
      const Item<R> it = load_item<R>(p, item);
      if (it.tiles == 0) continue;
      const uint32_t qbuf = k & 1;
      ok = __all_sync(0xffffffffu, ptx::mbar_wait(&q_empty[qbuf], ((k >> 1) & 1) ^ 1, 301));
      if (!ok) break;
      if (ptx::elect_one()) {
        ptx::mbar_expect_tx(&q_full[qbuf], R * kQBytes);
        for (int g = 0; g < R; ++g)   // (a row that does not exist reads another one or zeros: its results are dropped)
          ptx::tma_load_3d(s_q + (qbuf * R + g) * kQBytes, &tm_q, &q_full[qbuf], a.q_col0 + it.h * kD, it.qb * kQ, it.b0 + g);
      }
      const int bias_z = a.bias_head_major > 0 ? it.h * a.bias_head_major + it.bias_b : it.bias_b * a.heads + it.h;
      int from = it.first[0];       // tiles before the first masked key of every row need no mask operand
#pragma unroll
      for (int g = 1; g < R; ++g) from = min(from, it.first[g]);
      for (int t = 0; t < it.tiles; ++t) {
        ok = __all_sync(0xffffffffu, ptx::mbar_wait(&stage_empty[st], par ^ 1, 302));
        if (!ok) break;
        if (ptx::elect_one()) {
          uint8_t* dst = s_stage + st * kStageBytes;
          ptx::mbar_expect_tx(&stage_full[st], kStageBytes);
          for (int g = 0; g < R; ++g) {
            uint8_t* kv = dst + kBiasBytes + g * (kKBytes + kVBytes);
            ptx::tma_load_3d(kv, &tm_k, &stage_full[st], a.k_col0 + it.h * kD, t * kT, it.b0 + g);
            ptx::tma_load_3d(kv + kKBytes, &tm_v, &stage_full[st], t * kT, it.h * kD, it.b0 + g);
          }
          ptx::tma_load_3d(dst, &tm_b, &stage_full[st], t * kT, it.qb * kQ, bias_z);
        }
        if (++st == kStages) { st = 0; par ^= 1u; }
        if (t * kT + kT <= from) continue;
#pragma unroll
        for (int g = 0; g < R; ++g) {
          if (!ok || t * kT + kT <= it.first[g]) continue;
          const int b = it.b0 + min(g, it.rows - 1);
          const int b_hi = b / a.mask_lo_extent, b_lo = b - b_hi * a.mask_lo_extent;
          const unsigned char* mrow = a.mask + static_cast<long long>(b_hi) * a.m_hi + static_cast<long long>(b_lo) * a.m_lo;
          uint32_t v[2];
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int key = t * kT + lane + 32 * i;
            const float m = key >= a.lk ? kAbsent : (mrow[static_cast<long long>(key) * a.m_k] ? 0.f : kMasked);
            v[i] = static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(m)));
          }
          const uint32_t slot = uses[g] % kMaskSlots, mpar = (uses[g] / kMaskSlots) & 1;
          ok = __all_sync(0xffffffffu, ptx::mbar_wait(&m_empty[g * kMaskSlots + slot], mpar ^ 1, 308));
          if (!ok) continue;
          uint8_t* dst = s_mask + (g * kMaskSlots + slot) * kMaskBytes;
#pragma unroll
          for (int i = 0; i < 2; ++i) *reinterpret_cast<uint4*>(dst + ptx::noswizzle_row_offset(lane + 32 * i)) = make_uint4(v[i], 0, 0, 0);
          ptx::fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(&m_full[g * kMaskSlots + slot]);
          ++uses[g];
        }
        if (!ok) break;
      }
      ++k;
    }
  } else if (warp >= kMma) {
    // ---------------------------------------------------------------- MMA issue of row group g
    if (ptx::elect_one()) {
      const int g = warp - kMma;
      constexpr uint32_t idesc_s = ptx::make_idesc(kQ, kT, 1);
      constexpr uint32_t idesc_o = ptx::make_idesc(kQ, kD, 1);
      const uint32_t kv_off = kBiasBytes + g * (kKBytes + kVBytes);
      const uint64_t e0_desc = ptx::make_noswizzle_desc(ptx::smem_u32(s_e0));
      const uint64_t eye_desc = ptx::make_noswizzle_desc(ptx::smem_u32(s_eye));
      const uint64_t bias_desc = ptx::make_kmajor_desc<128>(ptx::smem_u32(s_stage));
      const uint64_t q_desc = ptx::make_kmajor_desc<kD * 2>(ptx::smem_u32(s_q + g * kQBytes));
      const uint64_t k_desc = ptx::make_kmajor_desc<kD * 2>(ptx::smem_u32(s_stage + kv_off));
      const uint64_t v_desc = ptx::make_kmajor_desc<128>(ptx::smem_u32(s_stage + kv_off + kKBytes));
      const uint64_t m_desc = ptx::make_noswizzle_desc(ptx::smem_u32(s_mask + g * kMaskSlots * kMaskBytes));
      const uint32_t tmem_g = tmem_base + g * (128 + kD), tmem_o = tmem_g + 128;
      auto first_masked = [&](const Item<R>& it) {
        int f = it.first[0];
#pragma unroll
        for (int i = 1; i < R; ++i) f = g == i ? it.first[i] : f;
        return f;
      };
      auto next_item = [&](int item, Item<R>& it) -> int {
        for (; item < p.items; item += gridDim.x) {
          it = load_item<R>(p, item);
          if (it.tiles > 0) break;
        }
        return item;
      };
      // S runs two tiles ahead of the products with V, across items: a_* is its position
      Item<R> a_it;
      int a_item = next_item(blockIdx.x, a_it), a_t = 0, a_st = 0, m_slot = 0;
      int a_tiles = a_item < p.items ? a_it.tiles : 0, a_first = a_item < p.items ? first_masked(a_it) : 0;
      uint32_t a_par = 0, a_k = 0, a_n = 0, m_par = 0;
      auto issue_s = [&]() -> bool {
        if (a_t == a_tiles) return true;     // every item's S has been issued
        if (a_t == 0 && !ptx::mbar_wait(&q_full[a_k & 1], (a_k >> 1) & 1, 303)) return false;
        if (!ptx::mbar_wait(&stage_full[a_st], a_par, 304)) return false;
        const bool masked = a_t * kT + kT > a_first;
        if (masked && !ptx::mbar_wait(&m_full[g * kMaskSlots + m_slot], m_par, 305)) return false;
        ptx::tc_fence_after_sync();
        const uint64_t qd = q_desc + (a_k & 1) * ((R * kQBytes) >> 4), kd = k_desc + a_st * (kStageBytes >> 4);
        const uint64_t bd = bias_desc + a_st * (kStageBytes >> 4);
        const uint32_t d = tmem_g + (a_n & 1) * kT;
#pragma unroll
        for (int c = 0; c < 4; ++c)   // bias x identity: exact products, added in float32 like the rest
          ptx::mma_f16_ss(d, bd + c * 2, eye_desc + (48 - 16 * c) * 2, idesc_s, c > 0 ? 1u : 0u);
        if constexpr (kEyes == 2) {
#pragma unroll
          for (int c = 0; c < 4; ++c) ptx::mma_f16_ss(d, bd + c * 2, eye_desc + (kEyeBytes >> 4) + (48 - 16 * c) * 2, idesc_s, 1u);
        }
#pragma unroll
        for (int c = 0; c < kD / 16; ++c) ptx::mma_f16_ss(d, qd + c * 2, kd + c * 2, idesc_s, 1u);
        if (masked) {
          ptx::mma_f16_ss(d, e0_desc, m_desc + m_slot * (kMaskBytes >> 4), idesc_s, 1u);
          ptx::tc_commit(&m_empty[g * kMaskSlots + m_slot]);
          if (++m_slot == kMaskSlots) { m_slot = 0; m_par ^= 1u; }
        }
        ptx::tc_commit(&s_full[g * 2 + (a_n & 1)]);
        ++a_n;
        if (++a_st == kStages) { a_st = 0; a_par ^= 1u; }
        if (++a_t == a_tiles) {
          ptx::tc_commit(&q_empty[a_k & 1]);
          ++a_k;
          a_item = next_item(a_item + gridDim.x, a_it);
          a_t = 0;
          a_tiles = a_item < p.items ? a_it.tiles : 0;
          a_first = a_item < p.items ? first_masked(a_it) : 0;
        }
        return true;
      };
      Item<R> it;
      int st = 0;
      uint32_t n = 0;
      bool ok = issue_s() && issue_s();
      for (int item = next_item(blockIdx.x, it); ok && item < p.items; item = next_item(item + gridDim.x, it)) {
        for (int t = 0; t < it.tiles; ++t) {
          if (!ptx::mbar_wait(&p_ready[g * 2 + (n & 1)], (n >> 1) & 1, 306)) { ok = false; break; }
          ptx::tc_fence_after_sync();
          const uint64_t vd = v_desc + st * (kStageBytes >> 4);
          const uint32_t pt = tmem_g + (n & 1) * kT;
          // (the first product of an item overwrites an accumulator that has been read: P comes from the warps that read it)
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) ptx::mma_f16_ts(tmem_o, pt + kk * 8, vd + kk * 2, idesc_o, (t > 0 || kk > 0) ? 1u : 0u);
          ptx::tc_commit(&stage_empty[st]);
          ptx::tc_commit(&pv_done[g * 2 + (n & 1)]);
          if (++st == kStages) st = 0;
          ++n;
          // the S after the next goes over the P just multiplied: the tensor core executes in order
          ok = issue_s();
          if (!ok) break;
        }
      }
    }
  } else {
    // ---------------------------------------------------------------- softmax and output of row group g
    const int g = warp >> 2, quad = warp & 3;
    const int r = quad * 32 + lane;
    const uint32_t tmem_g = tmem_base + g * (128 + kD) + (static_cast<uint32_t>(quad * 32) << 16);
    const uint32_t tmem_o = tmem_g + 128;
    bool ok = true;
    uint32_t n = 0;                   // tiles so far
    float s_cur = 0.f, l_run = 0.f;   // the row's stabiliser and sum
    bool shifted = false;             // some lane of the warp has a stabiliser other than zero

    // exponentials of 32 logits of the row, packed in pairs, and their sum
    auto exps = [&](auto sub, const uint32_t (&x)[32], uint32_t (&out)[16]) -> float {
      float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int i = 0; i < 32; i += 2) {
        float y0 = __uint_as_float(x[i]), y1 = __uint_as_float(x[i + 1]);
        if constexpr (decltype(sub)::value) { y0 -= s_cur; y1 -= s_cur; }
        const float p0 = ex2(y0), p1 = ex2(y1);
        sum[i & 2] += p0;
        sum[(i & 2) + 1] += p1;
        out[i >> 1] = pack_bf16x2(p0, p1);
      }
      return (sum[0] + sum[1]) + (sum[2] + sum[3]);
    };
    // rare: a tile whose sums ask for another stabiliser (S is still whole).  It moves to the row's maximum of this tile's keys, and
    // the accumulator and the sum with it; writes P.
    auto rescale = [&](int t, uint32_t tmem_s, bool mine) {
      float mx = -INFINITY;
      uint32_t x[32], out[16];
#pragma unroll 1
      for (int half = 0; half < 2; ++half) {
        ptx::tmem_ld_32x32b_x32(tmem_s + half * 32, x);
        ptx::tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i) mx = fmaxf(mx, __uint_as_float(x[i]));
      }
      const float s_new = mine ? (t == 0 ? mx : fmaxf(mx, s_cur)) : s_cur;
      const float alpha = ex2(s_cur - s_new);      // 1 for the rows whose stabiliser stays
      if (t > 0) {
        if (!__all_sync(0xffffffffu, ptx::mbar_wait(&pv_done[g * 2 + ((n - 1) & 1)], ((n - 1) >> 1) & 1, 310))) ok = false;
        ptx::tc_fence_after_sync();
#pragma unroll 1
        for (int c = 0; c < kD / 16; ++c) {
          ptx::tmem_ld_32x32b_x16(tmem_o + c * 16, out);
          ptx::tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) out[i] = __float_as_uint(__uint_as_float(out[i]) * alpha);
          ptx::tmem_st_32x32b_x16(tmem_o + c * 16, out);
        }
        l_run *= alpha;
      }
      s_cur = s_new;
      shifted = __any_sync(0xffffffffu, s_cur != 0.f);
#pragma unroll 1
      for (int half = 0; half < 2; ++half) {       // (P of the second half goes over S columns that the first has read)
        ptx::tmem_ld_32x32b_x32(tmem_s + half * 32, x);
        ptx::tmem_ld_wait();
        l_run += exps(std::true_type(), x, out);
        ptx::tmem_st_32x32b_x16(tmem_s + half * 16, out);
      }
    };

    for (int item = blockIdx.x; ok && item < p.items; item += gridDim.x) {
      const Item<R> it = load_item<R>(p, item);
      s_cur = 0.f;
      l_run = 0.f;
      shifted = false;
      // S columns 32 h .. 32 h + 31 become P columns 16 h .. 16 h + 15.
#pragma unroll 1
      for (int t = 0; t < it.tiles; ++t) {
        const uint32_t tmem_s = tmem_g + (n & 1) * kT;
        ok = __all_sync(0xffffffffu, ptx::mbar_wait(&s_full[g * 2 + (n & 1)], (n >> 1) & 1, 309));
        if (!ok) break;
        ptx::tc_fence_after_sync();
        uint32_t xa[32], xb[32], oa[16], ob[16];
        ptx::tmem_ld_32x32b_x32(tmem_s, xa);
        ptx::tmem_ld_32x32b_x32(tmem_s + 32, xb);
        ptx::tmem_ld_wait();
        // the groups take turns (see above): in the order of tiles and groups, this one after the (R - 1)-th before it
        if (g == R - 1 || n > 0) {
          const uint32_t m = g == R - 1 ? n : n - 1;
          ok = __all_sync(0xffffffffu, ptx::mbar_wait(&turn[((g + 1) % R * 2 + (m & 1)) * 4 + quad], (m >> 1) & 1, 311));
          if (!ok) break;
        }
        const float l0 = shifted ? exps(std::true_type(), xa, oa) : exps(std::false_type(), xa, oa);
        const float l1 = shifted ? exps(std::true_type(), xb, ob) : exps(std::false_type(), xb, ob);
        if (lane == 0) ptx::mbar_arrive(&turn[(g * 2 + (n & 1)) * 4 + quad]);
        const bool mine = !(l0 < kHighSum) || !(l1 < kHighSum) || (t == 0 && l0 + l1 < kLowSum);
        if (__any_sync(0xffffffffu, mine)) {
          rescale(t, tmem_s, mine);
          if (!ok) break;
        } else {
          l_run += l0;
          l_run += l1;
          ptx::tmem_st_32x32b_x16(tmem_s, oa);
          ptx::tmem_st_32x32b_x16(tmem_s + 16, ob);
        }
        ptx::tmem_st_wait();
        ptx::tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&p_ready[g * 2 + (n & 1)]);
        ++n;
      }
      if (!ok) break;
      // output: O / row sum, gate, store
      const int q = it.qb * kQ + r;
      const bool live = q < a.lq && g < it.rows;
      const int b = it.b0 + min(g, it.rows - 1);
      const long long row = static_cast<long long>(b) * a.lq + (q < a.lq ? q : 0);
      const __nv_bfloat16* gp = a.g != nullptr ? reinterpret_cast<const __nv_bfloat16*>(a.g) + row * a.ldg + a.g_col0 + it.h * kD : nullptr;
      uint4 gate[kD / 8];
      if (gp != nullptr) {
#pragma unroll
        for (int i = 0; i < kD / 8; ++i) gate[i] = *reinterpret_cast<const uint4*>(gp + i * 8);
      }
      float scale = 1.0f;
      if (it.tiles == 0) {
        // no valid key in any row (padding): every logit is the same finite -1e9 in the reference's float32 arithmetic, the result
        // the mean of V over all keys
        const __nv_bfloat16* vrows = reinterpret_cast<const __nv_bfloat16*>(a.vt) + (static_cast<long long>(b) * a.heads + it.h) * kD * a.ldv;
        for (int dd = quad * (kD / 4); dd < (quad + 1) * (kD / 4); ++dd) {
          float acc = 0.f;
          for (int key = lane; key < a.lk; key += 32) acc += __bfloat162float(vrows[static_cast<long long>(dd) * a.ldv + key]);
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
          if (lane == 0) s_mean[g * kD + dd] = acc / static_cast<float>(a.lk);
        }
        asm volatile("bar.sync %0, 128;" ::"r"(1 + g) : "memory");
      } else {
        scale = 1.0f / l_run;
        ok = __all_sync(0xffffffffu, ptx::mbar_wait(&pv_done[g * 2 + ((n - 1) & 1)], ((n - 1) >> 1) & 1, 313));
        if (!ok) break;
        ptx::tc_fence_after_sync();
      }
      __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(a.out) + row * a.ldo + it.h * a.d;
#pragma unroll
      for (int half = 0; half < kD / 16; ++half) {
        float v[16];
        if (it.tiles == 0) {
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = s_mean[g * kD + half * 16 + i];
        } else {
          ptx::tmem_ld_32x32b_x16(tmem_o + half * 16, reinterpret_cast<uint32_t(&)[16]>(v));
          ptx::tmem_ld_wait();
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const uint4 gu = gate[half * 2 + i];
          const uint32_t gw[4] = {gu.x, gu.y, gu.z, gu.w};
          uint32_t ow[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            float v0 = v[i * 8 + j * 2] * scale, v1 = v[i * 8 + j * 2 + 1] * scale;
            if (gp != nullptr) {
              v0 *= sigmoidf_fast(__uint_as_float(gw[j] << 16));
              v1 *= sigmoidf_fast(__uint_as_float(gw[j] & 0xffff0000u));
            }
            ow[j] = pack_bf16x2(v0, v1);
          }
          // d is a multiple of 8
          if (live && half * 16 + i * 8 < a.d) *reinterpret_cast<uint4*>(o + half * 16 + i * 8) = make_uint4(ow[0], ow[1], ow[2], ow[3]);
        }
      }
      if (it.tiles == 0) {
        asm volatile("bar.sync %0, 128;" ::"r"(1 + g) : "memory");     // the means have been read
      } else {
        ptx::tc_fence_before_sync();     // (the next item's first P is what lets the accumulator be written again)
      }
    }
  }

  ptx::tc_fence_before_sync();
  __syncthreads();
  if (warp == kMma) {
    ptx::tc_fence_after_sync();
    ptx::tmem_dealloc(tmem_base, Cfg::kTmemCols);
  }
}

// (last valid key + 1, first masked key or lk) of every batch row, one block of 32 warps per 32 rows.  Keys are read along whichever
// of the two strides is contiguous.  A chain of loads: with 8 warps a block, each scanning four rows (or an eighth of the keys of 32
// rows), 13.8 us for 768 x 768 keys between CUDA events (about 4 of them the events'), twice a block; now 10.4, once.
constexpr int kMaskWarps = 32;
// blockIdx.y == 1: the same of the transposed mask (the ending node's), behind the first result.
__global__ void __launch_bounds__(32 * kMaskWarps) mask_rows_kernel(AttnParams a, int2* rows) {
  grid_dependency_enter();
  if (blockIdx.y == 1) {
    const long long m_lo = a.m_lo;
    a.m_lo = a.m_k;
    a.m_k = m_lo;
    rows += a.batch;
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  __shared__ int s_last[kMaskWarps][33], s_first[kMaskWarps][33];
  auto row_ptr = [&](int b) {
    const int b_hi = b / a.mask_lo_extent, b_lo = b - b_hi * a.mask_lo_extent;
    return a.mask + static_cast<long long>(b_hi) * a.m_hi + static_cast<long long>(b_lo) * a.m_lo;
  };
  if (a.m_k == 1) {   // a warp walks a row
    const int b = blockIdx.x * 32 + w;
    if (b >= a.batch) return;
    const unsigned char* m = row_ptr(b);
    int last = 0, first = a.lk;
#pragma unroll 16
    for (int k = lane; k < a.lk; k += 32) {
      if (m[k]) last = k + 1;
      else first = min(first, k);
    }
    last = __reduce_max_sync(0xffffffffu, last);
    first = __reduce_min_sync(0xffffffffu, first);
    if (lane == 0) rows[b] = make_int2(last, first);
    return;
  }
  // neighbouring rows lie next to each other: lane = row, the warps share the keys
  const int b = blockIdx.x * 32 + lane;
  int last = 0, first = a.lk;
  if (b < a.batch) {
    const unsigned char* m = row_ptr(b);
#pragma unroll 8
    for (int k = w; k < a.lk; k += kMaskWarps) {
      if (m[static_cast<long long>(k) * a.m_k]) last = k + 1;
      else first = min(first, k);
    }
  }
  s_last[w][lane] = last;
  s_first[w][lane] = first;
  __syncthreads();
  // a warp takes one row, a lane the result of one warp
  last = __reduce_max_sync(0xffffffffu, s_last[lane][w]);
  first = __reduce_min_sync(0xffffffffu, s_first[lane][w]);
  if (lane == 0 && blockIdx.x * 32 + w < a.batch) rows[blockIdx.x * 32 + w] = make_int2(last, first);
}

}  // namespace

int launch_attention_mask_rows(cudaStream_t stream, const AttnParams& a, bool transposed_too) {
  LaunchScope scope(stream, "attention_mask_rows");
  return launch_kernel(stream, mask_rows_kernel, dim3(cdiv(a.batch, 32), transposed_too ? 2 : 1), 32 * kMaskWarps, 0, a, a.row_info);
}

template <int R, int kD>
static int launch_rows(cudaStream_t stream, const AttnParams& a) {
  using Cfg = RowsCfg<R, kD>;
  static std::once_flag once[64];
  int dev = 0;
  KFB_CUDA(cudaGetDevice(&dev));
  cudaError_t attr_err = cudaSuccess;
  std::call_once(once[dev & 63], [&] {
    attr_err = cudaFuncSetAttribute(attention_rows_kernel<R, kD>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmem);
  });
  KFB_CUDA(attr_err);
  CUtensorMap tq, tk, tv, tb;
  {
    const uint64_t dims[3] = {(uint64_t)a.ldq, (uint64_t)a.lq, (uint64_t)a.batch};
    const uint64_t str[2] = {(uint64_t)a.ldq * 2, (uint64_t)a.lq * a.ldq * 2};
    const uint32_t box[3] = {kD, kQ, 1};
    KFB_TRY(make_tmap(&tq, a.q, 2, 3, dims, str, box, kD * 2));
  }
  {
    const uint64_t dims[3] = {(uint64_t)a.ldk, (uint64_t)a.lk, (uint64_t)a.batch};
    const uint64_t str[2] = {(uint64_t)a.ldk * 2, (uint64_t)a.lk * a.ldk * 2};
    const uint32_t box[3] = {kD, kT, 1};
    KFB_TRY(make_tmap(&tk, a.k, 2, 3, dims, str, box, kD * 2));
  }
  {
    const uint64_t dims[3] = {(uint64_t)a.lk, (uint64_t)a.heads * kD, (uint64_t)a.batch};
    const uint64_t str[2] = {(uint64_t)a.ldv * 2, (uint64_t)a.heads * kD * a.ldv * 2};
    const uint32_t box[3] = {kT, kD, 1};
    KFB_TRY(make_tmap(&tv, a.vt, 2, 3, dims, str, box, 128));
  }
  const int groups = cdiv(a.batch, a.bias_div);
  {
    const int planes = (a.bias_head_major > 0 ? a.bias_head_major : groups) * a.heads;
    const uint64_t dims[3] = {(uint64_t)a.lk, (uint64_t)a.lq, (uint64_t)planes};
    const uint64_t str[2] = {(uint64_t)a.ldb * 2, (uint64_t)(a.bias_hs > 0 ? a.bias_hs : a.lq * a.ldb) * 2};
    const uint32_t box[3] = {kT, kQ, 1};
    KFB_TRY(make_tmap(&tb, a.bias, 2, 3, dims, str, box, 128));
  }
  RowsParams p;
  p.a = a;
  p.rows = a.row_info;
  p.sets_per_bias = cdiv(a.bias_div, R);
  p.q_blocks = cdiv(a.lq, kQ);
  p.items = p.q_blocks * a.heads * p.sets_per_bias * groups;
  if (!a.row_info_ready) KFB_TRY(launch_attention_mask_rows(stream, a));
  {
    LaunchScope scope(stream, a.tag ? a.tag : "attention_rows");
    KFB_TRY(launch_kernel(stream, attention_rows_kernel<R, kD>, p.items < sm_count() ? p.items : sm_count(), Cfg::kThreads, Cfg::kSmem, tq, tk,
                          tv, tb, p));
  }
  return KFB_OK;
}

int launch_attention_rows(cudaStream_t stream, const AttnParams& a) {
  if (a.dpad == 64) return launch_rows<2, 64>(stream, a);   // (shared memory has room for two groups)
  // A CTA of three row groups takes 5/4 of the time of two (N = 1024) for 3/2 of the work (more warps to fill each other's waits; one
  // more group would leave a single S buffer each, which measured slower); two leave fewer SMs idle in the last wave of few items.
  auto waves = [&](int r) {
    return cdiv(static_cast<long long>(cdiv(a.lq, kQ)) * a.heads * cdiv(a.bias_div, r) * cdiv(a.batch, a.bias_div), (long long)sm_count());
  };
  return waves(3) * 5 <= waves(2) * 4 ? launch_rows<3, 32>(stream, a) : launch_rows<2, 32>(stream, a);
}

}  // namespace kfb
