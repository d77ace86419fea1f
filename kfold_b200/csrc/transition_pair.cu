// The pair track's transition in one kernel: LayerNorm, both gated projections, SwiGLU, output projection, residual.  bf16 rows of 128
// or 256 channels.
//
// What bounds it.  As three launches (LayerNorm, SwiGLU GEMM, output GEMM) it moved the normalised rows and four times as many hidden
// activations through HBM: 1.5 GB for 768 x 768 rows of 128 channels, where reading and writing z is 0.3.  Here the hidden activations
// never leave the SM, and the time is the tensor core's: 6 144 cycles per 128 rows of 128 channels, 24 576 of 256.
//
// Split.  A CTA pair (cta_group::2) takes 256 rows, 128 in each CTA, and walks the hidden channels in chunks of 64:
//   S = LN(z) . [W_a; W_b]^T     256 x 128 (CTA 0 loads the chunk's 64 value rows, CTA 1 its 64 gate rows), K = C
//   h = silu(S_a) S_b            softmax-style in place: a thread owns a row, h goes over S in tensor memory as bf16
//   O += h . W_out^T             A from tensor memory, 256 x C, K = 64
// With single CTAs each would load all of the weights: operand traffic, 128 bytes a cycle through a shared memory, is what the products
// compete with (a chunk of 128 channels reads 56 KB of operands and is filled with 24 KB in 768 cycles of products; h in shared memory
// would add 32).
//   * S has three buffers of 128 columns (C = 128) or two (C = 256), which with O fill the tensor memory.  S and O have a thread each that
//     issues them.  A buffer's next S waits until the product that reads its h is done: tcgen05.mma promises an order only to products of the
//     same accumulator and shape, which these two have not.
//   * Two groups of four SwiGLU warps take the chunks in turn.  (All eight on one chunk: the special-function unit, 512 cycles a chunk, then
//     waits out every chunk's latencies: 6 us more.)
//   * Eight more warps normalise the next tile's rows in place in shared memory while this one is multiplied, and turn the finished tile
//     around: the residual comes back (from L2) into the tile's own buffer, which the products have left, is added, and the buffer leaves
//     as it is.  A thread of its own sees to what a buffer receives and sends.
// The arithmetic and its order are those of layernorm_c128_bf16_kernel / layernorm_c256_bf16_kernel and of the GEMMs this replaces: the
// same bits.
//
// Measured (graph replays, three launches -> this): 589 824 rows of 128 channels 380 -> 191 us (its products: 141 at the measured burst rate; the
// chain S - h - O through three S buffers is the rest), of 256 channels 976 -> 800 (at the power limit); 63 001 rows: 51 -> 28 and 111 -> 84.
// With the next S behind the issue of the product before it they were 187, 749, 28 and 79.
#include <cuda_bf16.h>

#include <mutex>

#include "gemm.cuh"   // glu_half, pack_bf16x2
#include "pair_rows.cuh"
#include "ptx.cuh"
#include "transition_pair.cuh"

namespace kfb {
namespace {

constexpr int kRows = kRowTile;            // rows of a CTA
constexpr int kChunk = 64;                 // hidden channels of a chunk
constexpr int kBox = kRowBox;              // [128 rows][64 bf16], 128-byte swizzle
constexpr int kSlot = 16384;               // unit of the ring of S's weights: 128 columns of K of a CTA's 64 rows
constexpr int kRowWarp = 4, kRowWarps = 8, kGluWarp = kRowWarp + kRowWarps;
constexpr int kThreads = 32 * (kGluWarp + 8);   // weights, S, rows in and out, O, 8 rows, 2 x 4 SwiGLU (a warp reads the tensor-memory lanes warp % 4)

template <int C>
struct Cfg {
  static constexpr int kABytes = (C / 64) * kBox;
  static constexpr int kA = C == 128 ? 3 : 2;         // tiles of rows: multiplied and finished, normalised, on their way
  static constexpr int kSlots = C == 128 ? 6 : 4;
  static constexpr int kS = C == 128 ? 3 : 2;         // S buffers
  static constexpr int kUnits = C / 128;              // ring units of a chunk's S
  static constexpr int kOutUnit = (C / 2) * 128;      // bytes of a chunk's W_out in a CTA; as many of them as S buffers
  static constexpr int kSmem = kA * kABytes + kSlots * kSlot + kS * kOutUnit + 512 + 1024;
  static_assert(kSmem <= 232448, "shared memory");
};

struct PairTransParams {
  const float *ln_w, *ln_b;
  int rows, tiles, chunks, has_resid, w_static;
  float eps;
};

template <int C>
__global__ void __launch_bounds__(kThreads, 1)
transition_pair_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_w1, const __grid_constant__ CUtensorMap tm_w2,
                       const __grid_constant__ CUtensorMap tm_r, const __grid_constant__ CUtensorMap tm_out, const PairTransParams p) {
  using K = Cfg<C>;
  constexpr int kLag = K::kS - 1;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* s_a = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));   // [kA][C / 64] boxes
  uint8_t* s_w = s_a + K::kA * K::kABytes;
  uint8_t* s_v = s_w + K::kSlots * kSlot;    // [kS] W_out
  uint64_t* bars = reinterpret_cast<uint64_t*>(s_v + K::kS * K::kOutUnit);
  uint64_t* full = bars;                     // [slots], in the leader: both CTAs' copies
  uint64_t* empty = full + K::kSlots;        // [slots]
  uint64_t* v_full = empty + K::kSlots;      // [kS], in the leader
  uint64_t* v_free = v_full + K::kS;         // [kS] the product has read it, and the h of the S buffer of the same number
  uint64_t* s_full = v_free + K::kS;         // [kS]
  uint64_t* h_ready = s_full + K::kS;        // [kS], in the leader: 4 warps of each CTA
  uint64_t* rows_in = h_ready + K::kS;       // [kA] a tile's rows have arrived
  uint64_t* resid_in = rows_in + K::kA;      // [kA] a tile's residual has, in their place
  uint64_t* a_norm = resid_in + K::kA;       // [kA] this CTA's rows are normalised: the row warps
  uint64_t* a_peer = a_norm + K::kA;         // [kA], in the leader: and the other CTA's
  uint64_t* a_done = a_peer + K::kA;         // [kA] every S of the tile
  uint64_t* out_done = a_done + K::kA;       // [kA] the row warps have written the output tile
  uint64_t* o_full = out_done + K::kA;
  uint64_t* o_empty = o_full + 1;            // in the leader: the row warps of both CTAs
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_empty + 1);
  static_assert((2 * 6 + 4 * 3 + 6 * 3 + 2) * 8 + 4 <= 512, "barriers");

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = static_cast<int>(ptx::cluster_ctarank());
  const int tile0 = blockIdx.x >> 1, tile_step = gridDim.x >> 1;
  const int my_tiles = (p.tiles - tile0 + tile_step - 1) / tile_step;      // (the grid has no pair without a tile)
  const int total = my_tiles * p.chunks;

  if (threadIdx.x == 0) {
    ptx::prefetch_tmap(&tm_x);
    ptx::prefetch_tmap(&tm_w1);
    ptx::prefetch_tmap(&tm_w2);
    ptx::prefetch_tmap(&tm_out);
    for (int i = 0; i < K::kSlots; ++i) {
      ptx::mbar_init(&full[i], 1);
      ptx::mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < K::kS; ++i) {
      ptx::mbar_init(&v_full[i], 1);
      ptx::mbar_init(&v_free[i], 1);
      ptx::mbar_init(&s_full[i], 1);
      ptx::mbar_init(&h_ready[i], 8);
    }
    for (int i = 0; i < K::kA; ++i) {
      ptx::mbar_init(&rows_in[i], 1);
      ptx::mbar_init(&resid_in[i], 1);
      ptx::mbar_init(&a_norm[i], kRowWarps);
      ptx::mbar_init(&a_peer[i], 1);
      ptx::mbar_init(&a_done[i], 1);
      ptx::mbar_init(&out_done[i], kRowWarps);
    }
    ptx::mbar_init(o_full, 1);
    ptx::mbar_init(o_empty, 2 * kRowWarps);
    ptx::fence_barrier_init();
  }
  if (warp == 1) {
    ptx::tmem_alloc_pair(tmem_slot, 512);
    ptx::tmem_relinquish_pair();
  }
  ptx::tc_fence_before_sync();
  __syncwarp();
  ptx::cluster_sync();
  ptx::tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_s = tmem_base + C;      // O lies before the S buffers

  if (warp == 0) {
    // ---------------------------------------------------------------- weights, in the order of the products.  Where they were written
    // before the launch before this one, the first of them come while that one drains.
    if (ptx::elect_one()) {
      if (!p.w_static) grid_dependency_wait();
      const int last = max((my_tiles - 1) * p.chunks, 2);      // the last tile, and a few chunks on their way
      int slot = 0, v = 0;
      uint32_t par = 0, v_par = 0;
      bool ok = true;
      int c1 = 0, c2 = 0;                     // chunk of the next S and of the next product with h
      for (int i = 0; ok && i < total + kLag; ++i) {
        if (i == last) {
          grid_dependency_wait();             // (a kernel lets the next one start after its own wait)
          grid_dependency_launch();
        }
        if (i < total) {
          const int row = (c1 >> 1) * 256 + 128 * rank + (c1 & 1) * kChunk;
          for (int u = 0; u < K::kUnits; ++u) {
            ok = ptx::mbar_wait(&empty[slot], par ^ 1, 401);
            if (!ok) break;
            if (rank == 0) ptx::mbar_expect_tx(&full[slot], 2 * kSlot);
            const uint32_t bar = ptx::leader_addr(&full[slot]);
#pragma unroll
            for (int k = 0; k < 2; ++k) ptx::tma_load_4d_pair(s_w + slot * kSlot + k * (kSlot / 2), &tm_w1, bar, u * 128 + 64 * k, row, 0, 0);
            if (++slot == K::kSlots) { slot = 0; par ^= 1u; }
          }
          if (++c1 == p.chunks) c1 = 0;
        }
        if (ok && i >= kLag) {
          ok = ptx::mbar_wait(&v_free[v], v_par ^ 1, 415);
          if (!ok) break;
          if (rank == 0) ptx::mbar_expect_tx(&v_full[v], 2 * K::kOutUnit);
          ptx::tma_load_4d_pair(s_v + v * K::kOutUnit, &tm_w2, ptx::leader_addr(&v_full[v]), c2 * kChunk, rank * (C / 2), 0, 0);
          if (++v == K::kS) { v = 0; v_par ^= 1u; }
          if (++c2 == p.chunks) c2 = 0;
        }
      }
      // the last products' arrivals at this CTA's barriers, before it may exit
      for (int i = 0; ok && i < K::kSlots; ++i) {
        ok = ptx::mbar_wait(&empty[slot], par ^ 1, 402);
        if (++slot == K::kSlots) { slot = 0; par ^= 1u; }
      }
      for (int i = 0; ok && i < K::kS; ++i) {
        ok = ptx::mbar_wait(&v_free[v], v_par ^ 1, 416);
        if (++v == K::kS) { v = 0; v_par ^= 1u; }
      }
    }
  } else if (warp == 1) {
    if (rank == 1) {
      // -------------------------------------------------------------- word to the leader that this CTA's rows are normalised (a thread of its
      // own: the release to the other CTA costs the thread that gives it some 1 500 cycles)
      if (ptx::elect_one()) {
        int ab = 0;
        uint32_t a_par = 0;
        for (int it = 0; it < my_tiles; ++it) {
          if (!ptx::mbar_wait(&a_norm[ab], a_par, 412)) break;
          ptx::mbar_arrive_cluster_release(ptx::leader_addr(&a_peer[ab]));
          if (++ab == K::kA) { ab = 0; a_par ^= 1u; }
        }
      }
      // -------------------------------------------------------------- S
    } else if (ptx::elect_one()) {
      constexpr uint32_t idesc = ptx::make_idesc(2 * kRows, 2 * kChunk, 1);
      const uint64_t a_desc = ptx::make_kmajor_desc<128>(ptx::smem_u32(s_a));
      const uint64_t w_desc = ptx::make_kmajor_desc<128>(ptx::smem_u32(s_w));
      int slot = 0, s1 = 0, ab = 0;
      uint32_t par = 0, s_par = 1, a_par = 0;      // s_par: phase of v_free that the buffer's next S waits for (the first kS: none)
      bool ok = true;
      for (int it = 0; ok && it < my_tiles; ++it) {
        ok = ptx::mbar_wait(&a_norm[ab], a_par, 404) && ptx::mbar_wait_cluster(&a_peer[ab], a_par, 413);
        const uint64_t ad = a_desc + ab * (K::kABytes >> 4);
        for (int c = 0; ok && c < p.chunks; ++c) {
          ok = ptx::mbar_wait(&v_free[s1], s_par, 417);
          if (!ok) break;
          ptx::tc_fence_after_sync();
          const uint32_t d = tmem_s + s1 * 128;
#pragma unroll
          for (int u = 0; u < K::kUnits; ++u) {
            ok = ptx::mbar_wait(&full[slot], par, 403);
            if (!ok) break;
            ptx::tc_fence_after_sync();
            const uint64_t wd = w_desc + static_cast<uint64_t>(slot * (kSlot >> 4));
#pragma unroll
            for (int k = 0; k < 8; ++k)
              ptx::mma_f16_ss_pair(d, ad + (2 * u + k / 4) * (kBox >> 4) + (k & 3) * 2, wd + (k / 4) * (kSlot >> 5) + (k & 3) * 2, idesc,
                                   (u > 0 || k > 0) ? 1u : 0u);
            ptx::tc_commit_pair(&empty[slot]);
            if (++slot == K::kSlots) { slot = 0; par ^= 1u; }
          }
          if (!ok) break;
          ptx::tc_commit_pair(&s_full[s1]);
          if (++s1 == K::kS) { s1 = 0; s_par ^= 1u; }
        }
        if (ok) ptx::tc_commit_pair(&a_done[ab]);
        if (++ab == K::kA) { ab = 0; a_par ^= 1u; }
      }
    }
  } else if (warp == 3) {
    // ---------------------------------------------------------------- O.  (By a thread of its own: one for both products took 1 370 cycles a
    // chunk for its waits and commits, of which the products are 768 at 128 channels.)
    if (rank == 0 && ptx::elect_one()) {
      constexpr uint32_t idesc = ptx::make_idesc(2 * kRows, C, 1);
      const uint64_t v_desc = ptx::make_kmajor_desc<128>(ptx::smem_u32(s_v));
      int s2 = 0;
      uint32_t par = 0;
      bool ok = true;
      for (int it = 0; ok && it < my_tiles; ++it) {
        ok = ptx::mbar_wait(o_empty, (it & 1) ^ 1, 405);
        for (int c = 0; ok && c < p.chunks; ++c) {
          ok = ptx::mbar_wait(&v_full[s2], par, 418) && ptx::mbar_wait(&h_ready[s2], par, 406);
          if (!ok) break;
          ptx::tc_fence_after_sync();
#pragma unroll
          for (int k = 0; k < kChunk / 16; ++k)
            ptx::mma_f16_ts_pair(tmem_base, tmem_s + s2 * 128 + k * 8, v_desc + static_cast<uint64_t>(s2 * (K::kOutUnit >> 4)) + k * 2, idesc,
                                 (c > 0 || k > 0) ? 1u : 0u);
          ptx::tc_commit_pair(&v_free[s2]);
          if (++s2 == K::kS) { s2 = 0; par ^= 1u; }
        }
        if (ok) ptx::tc_commit_pair(o_full);
      }
    }
  } else if (warp >= kGluWarp) {
    // ---------------------------------------------------------------- SwiGLU: chunks of one parity (a tile has an even number of them)
    const int group = (warp - kGluWarp) >> 2, quad = warp & 3;
    const uint32_t t_row = tmem_s + (static_cast<uint32_t>(quad * 32) << 16);
    int s = group;
    uint32_t par = 0;
    for (int i = group; i < total; i += 2) {
      const uint32_t t = t_row + s * 128;
      if (!__all_sync(0xffffffffu, ptx::mbar_wait(&s_full[s], par, 407))) break;
      ptx::tc_fence_after_sync();
      // pieces of 16 channels; the next one's trip under the arithmetic of this one.  h (8 columns a piece) goes over values that have
      // been read
      uint32_t va[16], ga[16], vb[16], gb[16];
      auto load = [&](int c, uint32_t (&v)[16], uint32_t (&g)[16]) {
        ptx::tmem_ld_32x32b_x16(t + c, v);
        ptx::tmem_ld_32x32b_x16(t + kChunk + c, g);
      };
      auto finish = [&](int c, const uint32_t (&v)[16], const uint32_t (&g)[16]) {
        uint32_t w[8];
#pragma unroll
        for (int j = 0; j < 16; j += 2) {
          w[j >> 1] = pack_bf16x2(ptx::mul2(glu_half2(v[j], v[j + 1], v[j], v[j + 1]), ptx::pack2(g[j], g[j + 1])));
        }
        ptx::tmem_st_32x32b_x8(t + c / 2, w);
      };
      load(0, va, ga);
      ptx::tmem_ld_wait();
      load(16, vb, gb);
      finish(0, va, ga);
      ptx::tmem_ld_wait();
      load(32, va, ga);
      finish(16, vb, gb);
      ptx::tmem_ld_wait();
      load(48, vb, gb);
      finish(32, va, ga);
      ptx::tmem_ld_wait();
      finish(48, vb, gb);
      ptx::tmem_st_wait();
      ptx::tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive_cluster(ptx::leader_addr(&h_ready[s]));
      s += 2;
      if (s >= K::kS) { s -= K::kS; par ^= 1u; }
    }
  } else if (warp >= kRowWarp) {
    // ---------------------------------------------------------------- rows: LayerNorm of the next tile, residual and output of the last
    const int part = warp - kRowWarp, quad = warp & 3;
    constexpr int kHalf = C / 2;                 // output columns of a warp: two warps share a quadrant's rows
    const int col0 = part / 4 * kHalf;
    const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + col0;
    grid_dependency_wait();
    uint64_t lw[4], lb[4];
    rows_affine<C>(p.ln_w, p.ln_b, lane, lw, lb);
    bool ok = true;
    int ab = 0, ob = 0;                          // buffers of the next tile and of the last, and their phases
    uint32_t a_par = 0, o_par = 0;
    for (int it = 0; it <= my_tiles; ++it) {
      if (it < my_tiles) {
        ok = __all_sync(0xffffffffu, ptx::mbar_wait(&rows_in[ab], a_par, 408)) != 0;
        if (!ok) break;
        rows_layernorm<C>(s_a + ab * K::kABytes, part * (kRows / kRowWarps), kRows / kRowWarps, lane, lw, lb, p.eps);
        ptx::fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&a_norm[ab]);
        if (++ab == K::kA) { ab = 0; a_par ^= 1u; }
      }
      if (it == 0) continue;
      // output of the tile before, over its rows (every S has read them) and, where there is one, the residual that has come in their place
      uint8_t* a = s_a + ob * K::kABytes;
      ok = __all_sync(0xffffffffu, ptx::mbar_wait(p.has_resid ? &resid_in[ob] : &a_done[ob], o_par, 409)) != 0;
      if (!ok) break;
      ok = __all_sync(0xffffffffu, ptx::mbar_wait(o_full, (it - 1) & 1, 410)) != 0;
      if (!ok) break;
      ptx::tc_fence_after_sync();
      const int r = quad * 32 + lane;
#pragma unroll 1
      for (int c = 0; c < kHalf; c += 64) {
        uint32_t x[2][32];
        ptx::tmem_ld_32x32b_x32(t_row + c, x[0]);
        ptx::tmem_ld_32x32b_x32(t_row + c + 32, x[1]);
        ptx::tmem_ld_wait();
        if (c + 64 == kHalf) {
          ptx::tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive_cluster(ptx::leader_addr(o_empty));
        }
        uint8_t* row = a + (col0 + c) / 64 * kBox + r * 128;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          uint4* cell = reinterpret_cast<uint4*>(row + ((i ^ (r & 7)) << 4));
          const uint4 u = p.has_resid ? *cell : make_uint4(0, 0, 0, 0);
          const uint32_t rw[4] = {u.x, u.y, u.z, u.w};
          uint32_t w[4];
#pragma unroll
          for (int j = 0; j < 4; ++j)
            w[j] = pack_bf16x2(__uint_as_float(x[i >> 2][8 * (i & 3) + 2 * j]) + __uint_as_float(rw[j] << 16),
                               __uint_as_float(x[i >> 2][8 * (i & 3) + 2 * j + 1]) + __uint_as_float(rw[j] & 0xffff0000u));
          *cell = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
      ptx::fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&out_done[ob]);
      if (++ob == K::kA) { ob = 0; o_par ^= 1u; }
    }
  } else if (warp == 2) {
    // ---------------------------------------------------------------- a buffer's course: rows in, residual in once every S has read them, output out
    if (ptx::elect_one()) {
      grid_dependency_wait();
      auto row0_of = [&](int it) { return (2 * (tile0 + it * tile_step) + rank) * kRows; };
      auto fetch = [&](const CUtensorMap* map, uint64_t* bar, int it, int b) {
        ptx::mbar_expect_tx(bar, K::kABytes);
#pragma unroll
        for (int kb = 0; kb < C / 64; ++kb) ptx::tma_load_4d(s_a + b * K::kABytes + kb * kBox, map, bar, kb * 64, row0_of(it), 0, 0);
      };
      for (int it = 0; it < K::kA && it < my_tiles; ++it) fetch(&tm_x, &rows_in[it], it, it);
      int b = 0;
      uint32_t b_par = 0;
      for (int it = 0; it < my_tiles; ++it) {
        if (!ptx::mbar_wait(&a_done[b], b_par, 414)) break;
        if (p.has_resid) fetch(&tm_r, &resid_in[b], it, b);
        if (!ptx::mbar_wait(&out_done[b], b_par, 411)) break;
        if (row0_of(it) < p.rows) {
#pragma unroll
          for (int kb = 0; kb < C / 64; ++kb) ptx::tma_store_4d(&tm_out, s_a + b * K::kABytes + kb * kBox, kb * 64, row0_of(it), 0, 0);
          ptx::tma_store_commit();
        }
        if (it + K::kA < my_tiles) {
          ptx::tma_store_wait_read();
          fetch(&tm_x, &rows_in[b], it + K::kA, b);
        }
        if (++b == K::kA) { b = 0; b_par ^= 1u; }
      }
      ptx::tma_store_wait_all();
    }
  }

  ptx::tc_fence_before_sync();
  __syncwarp();
  ptx::cluster_sync();      // neither CTA leaves while the other may still read its operands or reach its barriers
  if (warp == 1) {
    ptx::tc_fence_after_sync();
    ptx::tmem_dealloc_pair(tmem_base, 512);
  }
}

// Pairs of CTAs that the current device holds at once (0: none), asked once per device.
template <int C>
int pairs_held() {
  static std::once_flag once[64];
  static int held[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  std::call_once(once[dev & 63], [&] { held[dev & 63] = clusters_held(transition_pair_kernel<C>, 2, kThreads, Cfg<C>::kSmem); });
  return held[dev & 63];
}
int pairs_held(int c) { return c == 128 ? pairs_held<128>() : pairs_held<256>(); }

template <int C>
int launch(cudaStream_t stream, const void* x, const float* ln_w, const float* ln_b, const void* w_swiglu, const void* w_out, void* out,
           const void* resid, long long rows, int hidden, float eps, int w_static) {
  auto rows_map = [&](CUtensorMap* m, const void* ptr, long long n, int c, uint32_t box_rows) {
    const uint64_t dims[4] = {(uint64_t)c, (uint64_t)n, 1, 1};
    const uint64_t str[3] = {(uint64_t)c * 2, (uint64_t)c * 2 * n, (uint64_t)c * 2 * n};
    const uint32_t box[4] = {64, box_rows, 1, 1};
    return make_tmap(m, ptr, 2, 4, dims, str, box, 128);
  };
  CUtensorMap tx, t1, t2, tr, to;
  KFB_TRY(rows_map(&tx, x, rows, C, kRows));
  KFB_TRY(rows_map(&t1, w_swiglu, 2ll * hidden, C, kChunk));
  KFB_TRY(rows_map(&t2, w_out, C, hidden, C / 2));
  KFB_TRY(rows_map(&tr, resid != nullptr ? resid : x, rows, C, kRows));
  KFB_TRY(rows_map(&to, out, rows, C, kRows));
  const int held = pairs_held<C>();
  KFB_CHECK_ARG(held > 0, "transition: the device holds no pair of this kernel");
  PairTransParams p;
  p.ln_w = ln_w;
  p.ln_b = ln_b;
  p.rows = static_cast<int>(rows);
  p.tiles = static_cast<int>((rows + 2 * kRows - 1) / (2 * kRows));
  p.chunks = hidden / kChunk;
  p.has_resid = resid != nullptr;
  p.w_static = w_static;
  p.eps = eps;
  LaunchScope scope(stream, "transition_pair");
  return launch_kernel_clustered(stream, transition_pair_kernel<C>, 2, 2 * (p.tiles < held ? p.tiles : held), kThreads, Cfg<C>::kSmem, tx, t1, t2,
                                 tr, to, p);
}

}  // namespace

bool transition_pair_ok(const void* x, const void* w_swiglu, const void* w_out, const void* out, const void* resid, long long rows, int c,
                        int hidden, int dtype) {
  const uintptr_t all = reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w_swiglu) | reinterpret_cast<uintptr_t>(w_out) |
                        reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(resid);
  if (dtype != KFB_BF16 || (c != 128 && c != 256) || hidden % 128 != 0 || (all & 15) != 0 || rows > (1ll << 30)) return false;
  return pairs_held(c) > 0;
}

// Few rows: a pair walks all hidden channels of its 256 rows, 1.0 us a chunk at 256 channels and 0.52 at 128, however few tiles there are,
// where the three launches (the same bits) spread the hidden channels over the chip.  us for either, fitted to graph replays of 1 to 40 000
// rows with 128 to 2 048 hidden channels.  Three launches / this, 256 channels and 1 024 hidden: 4 096 rows 19.9 / 25.4, 6 400 23.8 / 25.6,
// 9 216 25.6 / 25.8, 10 500 30.8 / 27.1; 512 hidden: 4 096 16.6 / 17.6, 5 000 17.8 / 17.5; 128 channels and 512 hidden: 256 rows 12.2 / 10.7.
// (Beyond 64 rows for each multiprocessor the three launches take a second round: a fifth more.)
bool transition_pair_is_faster(long long rows, int c, int hidden) {
  const int held = pairs_held(c);
  if (held < 1) return false;
  const double chunks = hidden / kChunk;
  const long long tiles = (rows + 2 * kRows - 1) / (2 * kRows), rounds = (tiles + held - 1) / held;
  const double pair = c == 128 ? 6.9 + 0.52 * chunks * rounds : 9.2 + chunks * rounds;
  const double three = (c == 128 ? 10.3 + 0.22 * chunks : 11.3 + 0.24 * chunks) + 1e-3 * rows * (0.4 + 0.05 * chunks);
  return pair <= (rows > 64ll * sm_count() ? 1.2 : 1.0) * three;
}

int launch_transition_pair(cudaStream_t stream, const void* x, const float* ln_w, const float* ln_b, const void* w_swiglu, const void* w_out,
                           void* out, const void* resid, long long rows, int c, int hidden, float eps, int w_static) {
  return c == 128 ? launch<128>(stream, x, ln_w, ln_b, w_swiglu, w_out, out, resid, rows, hidden, eps, w_static)
                  : launch<256>(stream, x, ln_w, ln_b, w_swiglu, w_out, out, resid, rows, hidden, eps, w_static);
}

}  // namespace kfb
