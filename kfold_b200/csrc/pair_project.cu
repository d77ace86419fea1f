// The pair track's input projections in one kernel: LayerNorm, and everything that is multiplied from the normalised rows.
//   triangle multiplication (128 or 256 channels)  gated and masked operands, channel-major, and the output gate's logits, row-major
//   triangle attention (128 channels)              q, k, g row-major, V^T and the triangle bias channel-major
//
// What bounds it.  HBM: a row of 128 channels is 256 bytes in and 768 (1 032) out.  As a LayerNorm and one or two GEMMs the normalised rows
// went out and came back once more, and each 128 rows were multiplied by one column tile at a time: 96 KB into shared memory and 128 KB
// out of it for a gated tile, at 128 bytes a cycle more than the tile's share of HBM.
//
// Split.  A CTA pair (cta_group::2) takes 256 rows, 128 in each CTA: four runs of up to 64 consecutive positions of one pair row each, so
// that a channel-major output leaves as whole 128-byte lines and a row count like 333 or 400 wastes a tenth of the tiles.  The rows are
// normalised in place in shared memory and stay there while every column of the weights goes by, in units of 256 columns (each CTA loads
// 128) into one of two tensor-memory accumulators: M = 256, N = 256, K = C.
//   * Two teams of four epilogue warps take a unit's halves: 128 accumulator columns, 64 or 128 outputs.
//   * Channel-major outputs are transposed on the way out: tensor memory is read as 8 x 8 fragments, which stmatrix writes transposed.
//     The other way to have channels in the lanes, weights as the M operand, needs both accumulators for one unit of a pair.
//   * Eight warps normalise the next rows meanwhile.  (With four this was the longest chain of all: 8 500 cycles a tile of 128 channels,
//     18 400 of 256, clock stamps.)
// Few rows: with fewer tiles than pairs / units, a pair takes one unit of a tile (and normalises the rows for it alone).
// The arithmetic is that of the LayerNorm kernels and of the GEMMs: the same bits.
//
// Measured (events inside the operators, LayerNorm and projections as two or three launches -> this): 768 x 768 rows, triangle multiplication
// of 128 channels 206 -> 139 us (604 MB: 4.4 TB/s), of 256 544 -> 331, triangle attention's 224 -> 151; 251 x 251: 41 -> 30.5, 88 -> 55 and
// 43 -> 31.6; 64 x 64: 21 -> 16.6, 35 -> 25.8 and 21 -> 18.2.
#include <cuda_bf16.h>

#include <mutex>

#include "gemm.cuh"   // glu_half, pack_bf16x2
#include "pair_project.cuh"
#include "pair_rows.cuh"
#include "ptx.cuh"

namespace kfb {
namespace {

constexpr int kRun = 64;                   // positions of a run
constexpr int kUnit = 256;                 // accumulator columns of a unit
constexpr int kSlot = 128 * 128;           // weight ring: a CTA's 128 rows of 64 K
constexpr int kStage = kRowTile * 64 * 2;  // staged output: 128 positions x 64 channels, two boxes of one run each
constexpr int kKeep = 8;                   // tiles whose position masks are kept
constexpr int kTeams = 2;                  // one for each half of a unit
constexpr int kRowWarp = 4, kRowWarps = 8, kTeamWarp = kRowWarp + kRowWarps;
constexpr int kThreads = 32 * (kTeamWarp + 4 * kTeams);        // operands, MMA, a store for each team, 8 rows, 2 x 4 epilogue

template <int C, bool ATT>
struct Cfg {
  static constexpr int kKb = C / 64;
  static constexpr int kABytes = kKb * kRowBox;
  static constexpr int kUnits = ATT ? 3 : 4 * C / kUnit + 1;
  static constexpr int kLastN = ATT ? 32 : C;               // columns of the last unit: triangle bias, gate logits
  static constexpr int kSlots = 4;
  static constexpr int kA = C == 128 ? 3 : 2;               // tiles of rows: multiplied, normalised, on their way
  static constexpr int kStages = C == 128 ? 2 : 1;          // staged outputs of a team (in half the size they took longer: a store costs the
                                                            // same 1 000 cycles from its last byte staged to the stage's release)
  static constexpr int kSmem = kA * kABytes + kSlots * kSlot + kTeams * kStages * kStage + kKeep * kRowTile + 512 + 1024;
  static_assert(kSmem <= 232448, "shared memory");
};

struct ProjectParams {
  const float *ln_w, *ln_b;
  const unsigned char* mask;
  long long m_n, m_o, m_b;
  int n, runs_per_row, o_extent, batch;
  unsigned long long inv_runs, inv_o, inv_groups;   // of runs_per_row, o_extent and groups, see div_by
  int items, groups;                             // items = tiles x groups; groups: 1, or the units of a tile one by one
  int w_static;
  float eps, bias_scale;
  LnFold fold;                                   // (n == 0: none)
};

struct Run {
  int n0, o, b;
};

// i / d by the reciprocal floor(2^64 / d) + 1: exact for every 32-bit i >= 0, d > 1 (an integer division is a chain of some 200 cycles)
__host__ inline unsigned long long reciprocal(int d) { return d > 1 ? ~0ull / static_cast<unsigned>(d) + 1 : 0; }
__device__ __forceinline__ int div_by(int i, int d, unsigned long long inv) {
  return d > 1 ? static_cast<int>(__umul64hi(static_cast<unsigned>(i), inv)) : i;
}

template <int C, bool ATT>
__global__ void __launch_bounds__(kThreads, 1)
pair_project_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_last,
                    const __grid_constant__ CUtensorMap tm_rows, const __grid_constant__ CUtensorMap tm_chan,
                    const __grid_constant__ CUtensorMap tm_bias, const ProjectParams p) {
  using K = Cfg<C, ATT>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* s_a = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));   // [kA][C / 64] boxes
  uint8_t* s_w = s_a + K::kA * K::kABytes;
  uint8_t* s_out = s_w + K::kSlots * kSlot;  // [team][stage]
  uint8_t* s_keep = s_out + kTeams * K::kStages * kStage;    // [kKeep][128]
  uint64_t* bars = reinterpret_cast<uint64_t*>(s_keep + kKeep * kRowTile);
  uint64_t* full = bars;                     // [slots], in the leader: both CTAs' copies
  uint64_t* empty = full + K::kSlots;        // [slots]
  uint64_t* d_full = empty + K::kSlots;      // [2] a unit's products
  uint64_t* d_empty = d_full + 2;            // [2], in the leader: 2 teams x 4 warps of each CTA
  uint64_t* rows_in = d_empty + 2;           // [kA]
  uint64_t* a_norm = rows_in + K::kA;        // [kA] this CTA's rows are normalised: the row warps
  uint64_t* a_peer = a_norm + K::kA;         // [kA], in the leader: and the other CTA's
  uint64_t* a_done = a_peer + K::kA;         // [kA] every product of the tile
  uint64_t* keep_in = a_done + K::kA;        // [kKeep] a tile's masks: the row warps
  uint64_t* st_full = keep_in + kKeep;       // [team][stage] 4 warps
  uint64_t* st_free = st_full + kTeams * 2;  // [team][stage]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(st_free + kTeams * 2);
  static_assert((2 * 4 + 4 + 4 * 3 + kKeep + 4 * kTeams) * 8 + 4 <= 512, "barriers");

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = static_cast<int>(ptx::cluster_ctarank());
  const int item0 = blockIdx.x >> 1, item_step = gridDim.x >> 1;
  const int my_items = (p.items - item0 + item_step - 1) / item_step;      // (the grid has no pair without an item)
  // an item's tile and units
  auto item_of = [&](int it, int& tile, int& u0, int& u1) {
    const int item = item0 + it * item_step;
    tile = div_by(item, p.groups, p.inv_groups);
    u0 = p.groups == 1 ? 0 : item - tile * p.groups;
    u1 = p.groups == 1 ? K::kUnits : u0 + 1;
  };
  // this CTA's run h of a tile; past the last one: outside the tensors (b = batch)
  auto run_of = [&](int tile, int h) -> Run {
    const int i = 4 * tile + 2 * rank + h;
    const int row = div_by(i, p.runs_per_row, p.inv_runs);
    Run r;
    r.n0 = (i - row * p.runs_per_row) * kRun;
    r.b = div_by(row, p.o_extent, p.inv_o);
    r.o = row - r.b * p.o_extent;
    return r;
  };

  if (threadIdx.x == 0) {
    ptx::prefetch_tmap(&tm_x);
    ptx::prefetch_tmap(&tm_w);
    ptx::prefetch_tmap(&tm_last);
    ptx::prefetch_tmap(&tm_rows);
    ptx::prefetch_tmap(&tm_chan);
    for (int i = 0; i < K::kSlots; ++i) {
      ptx::mbar_init(&full[i], 1);
      ptx::mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      ptx::mbar_init(&d_full[i], 1);
      ptx::mbar_init(&d_empty[i], 2 * 4 * kTeams);
    }
    for (int i = 0; i < K::kA; ++i) {
      ptx::mbar_init(&rows_in[i], 1);
      ptx::mbar_init(&a_norm[i], kRowWarps);
      ptx::mbar_init(&a_peer[i], 1);
      ptx::mbar_init(&a_done[i], 1);
    }
    for (int i = 0; i < kKeep; ++i) ptx::mbar_init(&keep_in[i], kRowWarps);
    for (int i = 0; i < kTeams * 2; ++i) {
      ptx::mbar_init(&st_full[i], 4);
      ptx::mbar_init(&st_free[i], 1);
    }
    ptx::fence_barrier_init();
  }
  if (warp == 1) {
    ptx::tmem_alloc_pair(tmem_slot, 2 * kUnit);
    ptx::tmem_relinquish_pair();
  }
  ptx::tc_fence_before_sync();
  __syncwarp();
  ptx::cluster_sync();
  ptx::tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ---------------------------------------------------------------- operands: weights in the order of the products (the first of them while
    // the launch before this one drains, where they were written before it), rows as soon as their buffer is multiplied
    if (ptx::elect_one()) {
      int slot = 0, w_it = 0, w_tile = 0, w_u = 0, w_u1 = 0, w_kb = 0;     // weights: the next unit's place and K block
      uint32_t par = 0;
      item_of(0, w_tile, w_u, w_u1);
      auto next_weights = [&]() {
        const bool last = w_u == K::kUnits - 1;
        const int rows = last ? K::kLastN / 2 : kUnit / 2;
        if (rank == 0) ptx::mbar_expect_tx(&full[slot], 2 * rows * 128);
        ptx::tma_load_4d_pair(s_w + slot * kSlot, last ? &tm_last : &tm_w, ptx::leader_addr(&full[slot]), w_kb * 64,
                              (last ? 0 : w_u * kUnit) + rank * rows, 0, 0);
        if (++slot == K::kSlots) { slot = 0; par ^= 1u; }
        if (++w_kb < K::kKb) return;
        w_kb = 0;
        if (++w_u < w_u1) return;
        if (++w_it < my_items) item_of(w_it, w_tile, w_u, w_u1);
      };
      int r_it = 0, ab = 0;                   // rows: the next tile and its buffer
      uint32_t a_par = 1;                     // (phase of a_done that the buffer's last tile completes; the first kA tiles wait for none)
      auto next_rows = [&]() {
        int tile, u0, u1;
        item_of(r_it, tile, u0, u1);
        ptx::mbar_expect_tx(&rows_in[ab], K::kABytes);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const Run r = run_of(tile, h);
#pragma unroll
          for (int kb = 0; kb < K::kKb; ++kb)
            ptx::tma_load_4d(s_a + ab * K::kABytes + kb * kRowBox + h * (kRowBox / 2), &tm_x, &rows_in[ab], kb * 64, r.n0, r.o, r.b);
        }
        ++r_it;
        if (++ab == K::kA) { ab = 0; a_par ^= 1u; }
      };
      if (p.w_static)
        for (int i = 0; i < K::kSlots && w_it < my_items; ++i) next_weights();
      grid_dependency_wait();
      bool ok = true;
      uint32_t spins = 0;
      unsigned long long t0 = 0;
      while (ok && (w_it < my_items || r_it < my_items)) {
        bool idle = true;
        if (r_it < my_items && ptx::mbar_test(&a_done[ab], a_par)) {
          next_rows();
          idle = false;
        }
        if (w_it < my_items && ptx::mbar_test(&empty[slot], par ^ 1)) {
          next_weights();
          idle = false;
        }
        if (idle) {
          ok = ptx::spin_on(spins, t0, 501);
        } else {
          spins = 0;
          t0 = 0;
        }
      }
      grid_dependency_launch();
      // the last products' arrivals at this CTA's barriers, before it may exit
      for (int i = 0; ok && i < K::kSlots; ++i) {
        ok = ptx::mbar_wait(&empty[slot], par ^ 1, 502);
        if (++slot == K::kSlots) { slot = 0; par ^= 1u; }
      }
      for (int i = 0; ok && i < K::kA; ++i) {
        ok = ptx::mbar_wait(&a_done[ab], a_par, 507);
        if (++ab == K::kA) { ab = 0; a_par ^= 1u; }
      }
    }
  } else if (warp == 1) {
    if (rank == 1) {
      // -------------------------------------------------------------- word to the leader that this CTA's rows are normalised.  (A thread of
      // its own: the release to the other CTA costs the thread that gives it some 1 500 cycles, a third of a row warp's tile.)
      if (ptx::elect_one()) {
        int ab = 0;
        uint32_t a_par = 0;
        for (int it = 0; it < my_items; ++it) {
          if (!ptx::mbar_wait(&a_norm[ab], a_par, 512)) break;
          ptx::mbar_arrive_cluster_release(ptx::leader_addr(&a_peer[ab]));
          if (++ab == K::kA) { ab = 0; a_par ^= 1u; }
        }
      }
      // -------------------------------------------------------------- MMA issue
    } else if (ptx::elect_one()) {
      constexpr uint32_t idesc_unit = ptx::make_idesc(2 * kRowTile, kUnit, 1);
      constexpr uint32_t idesc_last = ptx::make_idesc(2 * kRowTile, K::kLastN, 1);
      const uint64_t a_desc = ptx::make_kmajor_desc<128>(ptx::smem_u32(s_a));
      const uint64_t w_desc = ptx::make_kmajor_desc<128>(ptx::smem_u32(s_w));
      int slot = 0;
      uint32_t par = 0, unit = 0;
      int ab = 0;
      uint32_t a_par = 0;
      bool ok = true;
      for (int it = 0; ok && it < my_items; ++it) {
        int tile, u0, u1;
        item_of(it, tile, u0, u1);
        ok = ptx::mbar_wait(&a_norm[ab], a_par, 503) && ptx::mbar_wait_cluster(&a_peer[ab], a_par, 504);
        if (!ok) break;
        const uint64_t ad = a_desc + ab * (K::kABytes >> 4);
        for (int u = u0; u < u1; ++u, ++unit) {
          ok = ptx::mbar_wait(&d_empty[unit & 1], ((unit >> 1) & 1) ^ 1, 513);
          if (!ok) break;
          ptx::tc_fence_after_sync();
          const uint32_t d = tmem_base + (unit & 1) * kUnit, idesc = u == K::kUnits - 1 ? idesc_last : idesc_unit;
#pragma unroll
          for (int kb = 0; kb < K::kKb; ++kb) {
            ok = ptx::mbar_wait(&full[slot], par, 505);
            if (!ok) break;
            ptx::tc_fence_after_sync();
            const uint64_t wd = w_desc + static_cast<uint64_t>(slot * (kSlot >> 4));
#pragma unroll
            for (int k = 0; k < 4; ++k)
              ptx::mma_f16_ss_pair(d, ad + kb * (kRowBox >> 4) + k * 2, wd + k * 2, idesc, (kb > 0 || k > 0) ? 1u : 0u);
            ptx::tc_commit_pair(&empty[slot]);
            if (++slot == K::kSlots) { slot = 0; par ^= 1u; }
          }
          if (!ok) break;
          ptx::tc_commit_pair(&d_full[unit & 1]);
        }
        if (ok) ptx::tc_commit_pair(&a_done[ab]);
        if (++ab == K::kA) { ab = 0; a_par ^= 1u; }
      }
    }
  } else if (warp >= kRowWarp && warp < kTeamWarp) {
    // ---------------------------------------------------------------- rows: normalised in place
    const int part = warp - kRowWarp;
    grid_dependency_wait();
    uint64_t lw[4], lb[4];
    rows_affine<C>(p.ln_w, p.ln_b, lane, lw, lb);
    int ab = 0;
    uint32_t a_par = 0;
    for (int it = 0; it < my_items; ++it) {
      if (!__all_sync(0xffffffffu, ptx::mbar_wait(&rows_in[ab], a_par, 506))) break;
      // what of each of the warp's positions is kept: nothing past the row, nothing masked (volatile: asked for here, used behind the rows)
      uint32_t keep = 0;
      if (lane < kRowTile / kRowWarps) {
        int tile, u0, u1;
        item_of(it, tile, u0, u1);
        const Run r = run_of(tile, part / (kRowWarps / 2));
        const int n = r.n0 + part % (kRowWarps / 2) * (kRowTile / kRowWarps) + lane;
        keep = n < p.n && r.b < p.batch;
        if (!ATT && keep)
          asm volatile("ld.global.u8 %0, [%1];" : "=r"(keep) : "l"(p.mask + static_cast<long long>(r.b) * p.m_b + static_cast<long long>(r.o) * p.m_o +
                                                                     static_cast<long long>(n) * p.m_n));
      }
      rows_layernorm<C>(s_a + ab * K::kABytes, part * (kRowTile / kRowWarps), kRowTile / kRowWarps, lane, lw, lb, p.eps);
      if (lane < kRowTile / kRowWarps) s_keep[(it % kKeep) * kRowTile + part * (kRowTile / kRowWarps) + lane] = keep != 0;
      ptx::fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        ptx::mbar_arrive(&a_norm[ab]);
        ptx::mbar_arrive(&keep_in[it % kKeep]);
      }
      if (++ab == K::kA) { ab = 0; a_par ^= 1u; }
    }
  } else if (warp >= kTeamWarp) {
    // ---------------------------------------------------------------- epilogue
    const int team = (warp - kTeamWarp) >> 2, quad = warp & 3;
    const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
    uint8_t* const my_out = s_out + team * (K::kStages * kStage);
    const int s = team;                        // half of every unit
    uint32_t use = 0, unit = 0;
    uint8_t* box = nullptr;
    auto stage_begin = [&]() -> bool {
      const uint32_t round = use / K::kStages, st = use % K::kStages;
      box = my_out + st * kStage;
      return round == 0 || __all_sync(0xffffffffu, ptx::mbar_wait(&st_free[team * 2 + st], (round - 1) & 1, 509)) != 0;
    };
    auto stage_end = [&]() {
      ptx::fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&st_full[team * 2 + use % K::kStages]);
      ++use;
    };
    // Transposed boxes [64 channels][64 positions]: lane l writes the 16 bytes of channel l % 8 of a block, which are the positions of its
    // fragment's lanes.  Blocks of a store: channels 0..7 of positions 0..7, of 8..15, channels 8..15 of either.
    const uint32_t cell = (quad >> 1) * (kStage / 2) + ((lane >> 4) * 8 + (lane & 7)) * 128 +
                          ((((quad & 1) * 4 + ((lane >> 3) & 1)) ^ (lane & 7)) << 4);      // (16 positions on: ^ 32)
    float keep[4];            // of this lane's positions lane / 4 + 8 i of the quadrant
    bool ok = true;
    for (int it = 0; ok && it < my_items; ++it) {
      int tile, u0, u1;
      item_of(it, tile, u0, u1);
      ok = __all_sync(0xffffffffu, ptx::mbar_wait(&keep_in[it % kKeep], (it / kKeep) & 1, 514)) != 0;
      if (!ok) break;
#pragma unroll
      for (int i = 0; i < 4; ++i) keep[i] = s_keep[(it % kKeep) * kRowTile + quad * 32 + (lane >> 2) + 8 * i] ? 1.0f : 0.0f;
      for (int u = u0; u < u1; ++u, ++unit) {
        const bool last = u == K::kUnits - 1;
        ok = __all_sync(0xffffffffu, ptx::mbar_wait(&d_full[unit & 1], (unit >> 1) & 1, 510)) != 0;
        if (!ok) break;
        ptx::tc_fence_after_sync();
        const uint32_t t = t_row + (unit & 1) * kUnit;
        auto release = [&]() {
          ptx::tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive_cluster(ptx::leader_addr(&d_empty[unit & 1]));
        };
        // piece i of a stage: 16 of its channels x 16 of the quadrant's 32 positions
        auto put = [&](int i, const uint32_t (&w)[4]) {
          ptx::stmatrix_x4_trans(ptx::smem_u32(box) + (cell ^ ((i & 1) * 32)) + (i >> 1) * (16 * 128), w[0], w[1], w[2], w[3]);
        };
        if (!ATT && !last) {
          // gated: 64 values and their gates, in pieces of 16 positions x 16 channels, the next one's trip under the arithmetic of this
          uint32_t va[8], ga[8], vb[8], gb[8];
          auto load = [&](int i, uint32_t (&v)[8], uint32_t (&g)[8]) {
            const uint32_t at = t + (static_cast<uint32_t>((i & 1) * 16) << 16) + 64 * s + (i >> 1) * 16;
            ptx::tmem_ld_16x256b_x2(at, v);
            ptx::tmem_ld_16x256b_x2(at + 128, g);
          };
          auto finish = [&](int i, const uint32_t (&v)[8], const uint32_t (&g)[8]) {
            uint32_t w[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const float m = keep[(i & 1) * 2 + (j & 1)];
              w[j] = pack_bf16x2(ptx::mul2(glu_half2(v[2 * j], v[2 * j + 1], g[2 * j], g[2 * j + 1]), ptx::pack2(m, m)));
            }
            put(i, w);
          };
          load(0, va, ga);
          ok = stage_begin();
          if (!ok) break;
#pragma unroll
          for (int i = 0; i < 8; i += 2) {
            ptx::tmem_ld_wait();
            load(i + 1, vb, gb);
            finish(i, va, ga);
            ptx::tmem_ld_wait();
            if (i < 6)
              load(i + 2, va, ga);
            else
              release();
            finish(i + 1, vb, gb);
          }
          stage_end();
        } else if (ATT && last) {
          // bias: at most eight heads, all 128 positions, by the first half's team
          if (s == 0) {
            uint32_t a[4], b[4];
            ptx::tmem_ld_16x256b_x1(t, a);
            ptx::tmem_ld_16x256b_x1(t + (16u << 16), b);
            ok = stage_begin();
            if (!ok) break;
            ptx::tmem_ld_wait();
            release();
            auto two = [&](uint32_t x, uint32_t y, float m) { return pack_bf16x2(__uint_as_float(x) * m, __uint_as_float(y) * m); };
            const float sc = p.bias_scale;
            const uint32_t at = ptx::smem_u32(box) + (quad >> 1) * (kStage / 2) + (lane & 7) * 128 + ((((quad & 1) * 4 + (lane >> 3)) ^ (lane & 7)) << 4);
            ptx::stmatrix_x4_trans(at, two(a[0], a[1], sc * keep[0]), two(a[2], a[3], sc * keep[1]), two(b[0], b[1], sc * keep[2]),
                                   two(b[2], b[3], sc * keep[3]));
            stage_end();
          } else {
            release();
          }
        } else if (ATT && u == 1 && s == 1) {
          // V^T
#pragma unroll 1
          for (int k = 0; k < 4; ++k) {        // 32 channels at a time, 64 in a stage
            uint32_t v[4][8];
#pragma unroll
            for (int i = 0; i < 4; ++i)
              ptx::tmem_ld_16x256b_x2(t + (static_cast<uint32_t>((i & 1) * 16) << 16) + 128 + 32 * k + (i >> 1) * 16, v[i]);
            if ((k & 1) == 0) {
              ok = stage_begin();
              if (!ok) break;
            }
            ptx::tmem_ld_wait();
            if (k == 3) release();
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              uint32_t w[4];
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const float m = keep[(i & 1) * 2 + (j & 1)];
                w[j] = pack_bf16x2(__uint_as_float(v[i][2 * j]) * m, __uint_as_float(v[i][2 * j + 1]) * m);
              }
              put((k & 1) * 4 + i, w);
            }
            if (k & 1) stage_end();
          }
          if (!ok) break;
        } else {
          // row-major: a lane's position, 64 columns at a time
          const int width = last ? K::kLastN / 2 : kUnit / 2;
          const int r = quad * 32 + lane;
#pragma unroll 1
          for (int c = 0; c < width; c += 64) {
            uint32_t x[4][16];      // 16 columns at a time, the next ones on their way
            ptx::tmem_ld_32x32b_x16(t + s * width + c, x[0]);
            ok = stage_begin();
            if (!ok) break;
            uint8_t* row = box + r * 128;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              ptx::tmem_ld_wait();
              if (q < 3)
                ptx::tmem_ld_32x32b_x16(t + s * width + c + 16 * (q + 1), x[q + 1]);
              else if (c + 64 >= width)
                release();
#pragma unroll
              for (int i = 0; i < 2; ++i) {
                uint32_t w[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) w[j] = pack_bf16x2(__uint_as_float(x[q][8 * i + 2 * j]), __uint_as_float(x[q][8 * i + 2 * j + 1]));
                *reinterpret_cast<uint4*>(row + (((2 * q + i) ^ (r & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
              }
            }
            stage_end();
          }
          if (!ok) break;
        }
      }
    }
  } else {
    // ---------------------------------------------------------------- a team's stores; before them, a share of the folded weights
    const int s = warp - 2;
    grid_dependency_wait();
    for (int row = blockIdx.x * kTeams + s; row < p.fold.n; row += gridDim.x * kTeams) {
      // ln_fold_weights_kernel's sums in its order: four warps' partial sums
      const LnFold& f = p.fold;
      float a1[4] = {}, a0[4] = {};
      for (int i0 = 0; i0 < f.k; i0 += 128) {
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          const int i = i0 + w * 32 + lane;
          const long long at = static_cast<long long>(row) * f.k + i;
          const float wv = __bfloat162float(f.w[at]);
          const __nv_bfloat16 wr = __float2bfloat16_rn(wv * (f.gamma != nullptr ? f.gamma[i] : 1.0f));
          f.wf[at] = wr;
          a1[w] += __bfloat162float(wr);
          a0[w] += (f.beta != nullptr ? f.beta[i] : 0.0f) * wv;
        }
      }
#pragma unroll
      for (int m = 16; m > 0; m >>= 1)
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          a1[w] += __shfl_xor_sync(0xffffffffu, a1[w], m);
          a0[w] += __shfl_xor_sync(0xffffffffu, a0[w], m);
        }
      if (lane == 0) {
        f.s1[row] = (a1[0] + a1[1]) + (a1[2] + a1[3]);
        f.s0[row] = (a0[0] + a0[1]) + (a0[2] + a0[3]);
      }
    }
    __syncwarp();
    if (ptx::elect_one()) {
      const uint8_t* my_out = s_out + s * (K::kStages * kStage);
      uint32_t use = 0;
      uint64_t* reading = nullptr;       // stage that the last store reads: free once it has, or once the next one has been issued
      bool ok = true;
      for (int it = 0; ok && it < my_items; ++it) {
        int tile, u0, u1;
        item_of(it, tile, u0, u1);
        const Run run[2] = {run_of(tile, 0), run_of(tile, 1)};
        for (int u = u0; ok && u < u1; ++u) {
          const bool last = u == K::kUnits - 1, bias = ATT && last, gated = !ATT && !last, chan = bias || gated || (ATT && u == 1 && s == 1);
          const int width = last ? K::kLastN / 2 : kUnit / 2;        // columns of a half
          const int stages = bias ? 1 - s : gated ? 1 : width / 64;
          for (int k = 0; k < stages; ++k, ++use) {
            const int st = use % K::kStages;
            const uint32_t st_par = (use / K::kStages) & 1;
            if (reading != nullptr && (K::kStages == 1 || !ptx::mbar_test(&st_full[s * 2 + st], st_par))) {
              ptx::tma_store_wait_read();
              ptx::mbar_arrive(reading);
              reading = nullptr;
            }
            ok = ptx::mbar_wait(&st_full[s * 2 + st], st_par, 511);
            if (!ok) break;
            const uint8_t* src = my_out + st * kStage;
            const int ch = bias ? 0 : gated ? u * 128 + s * 64 : k * 64;
            const int col = (last ? 0 : u * kUnit) + s * width + k * 64;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              if (run[h].b >= p.batch) continue;
              if (chan)
                ptx::tma_store_4d(bias ? &tm_bias : &tm_chan, src + h * (kStage / 2), run[h].n0, run[h].o, ch, run[h].b);
              else
                ptx::tma_store_4d(&tm_rows, src + h * (kStage / 2), col, run[h].n0, run[h].o, run[h].b);
            }
            ptx::tma_store_commit();
            if (reading != nullptr) {
              ptx::tma_store_wait_read_le<1>();
              ptx::mbar_arrive(reading);
            }
            reading = &st_free[s * 2 + st];
          }
        }
      }
      ptx::tma_store_wait_all();
    }
  }

  ptx::tc_fence_before_sync();
  __syncwarp();
  ptx::cluster_sync();      // neither CTA leaves while the other may still read its operands or reach its barriers
  if (warp == 1) {
    ptx::tc_fence_after_sync();
    ptx::tmem_dealloc_pair(tmem_base, 2 * kUnit);
  }
}

// Pairs of CTAs that the current device holds at once (0: none), asked once per device.
template <int C, bool ATT>
int pairs_held() {
  static std::once_flag once[64];
  static int held[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  std::call_once(once[dev & 63], [&] { held[dev & 63] = clusters_held(pair_project_kernel<C, ATT>, 2, kThreads, Cfg<C, ATT>::kSmem); });
  return held[dev & 63];
}

bool rows_ok(const PairRows& r, int dtype) {
  const long long runs = static_cast<long long>(r.batch) * r.n * cdiv(r.n, kRun);
  return dtype == KFB_BF16 && (reinterpret_cast<uintptr_t>(r.x) & 15) == 0 && runs < (1ll << 28);
}

// Tiles of four runs (rows_ok: they fit).
int row_tiles(const PairRows& r) { return cdiv(r.batch * r.n * cdiv(r.n, kRun), 4); }

// Bytes of a tensor map's strides from elements.
int map4(CUtensorMap* m, const void* ptr, uint64_t d0, uint64_t d1, uint64_t d2, uint64_t d3, long long s1, long long s2, long long s3, uint32_t b0,
         uint32_t b1, uint32_t b2) {
  const uint64_t dims[4] = {d0, d1, d2, d3};
  const uint64_t str[3] = {static_cast<uint64_t>(s1) * 2, static_cast<uint64_t>(s2) * 2, static_cast<uint64_t>(s3) * 2};
  const uint32_t box[4] = {b0, b1, b2, 1};
  return make_tmap(m, ptr, 2, 4, dims, str, box, 128);
}

template <int C, bool ATT>
int launch(cudaStream_t stream, const PairRows& r, const void* w, const void* w_last, const CUtensorMap& t_rows, const CUtensorMap& t_chan,
           const CUtensorMap& t_bias, ProjectParams p, const char* tag) {
  using K = Cfg<C, ATT>;
  CUtensorMap tx, tw, tl;
  KFB_TRY(map4(&tx, r.x, C, r.n, r.n, r.batch, r.s_n, r.s_o, r.s_b, 64, kRun, 1));
  const long long w_rows = (K::kUnits - 1) * kUnit;
  KFB_TRY(map4(&tw, w, C, w_rows, 1, 1, C, C * w_rows, C * w_rows, 64, kUnit / 2, 1));
  KFB_TRY(map4(&tl, w_last, C, K::kLastN, 1, 1, C, C * K::kLastN, C * K::kLastN, 64, K::kLastN / 2, 1));
  const int held = pairs_held<C, ATT>();
  KFB_CHECK_ARG(held > 0, "%s: the device holds no pair of this kernel", tag);
  p.ln_w = r.ln_w;
  p.ln_b = r.ln_b;
  p.eps = r.eps;
  p.n = r.n;
  p.runs_per_row = cdiv(r.n, kRun);
  p.o_extent = r.n;
  p.batch = r.batch;
  p.w_static = r.w_static;
  const int tiles = row_tiles(r);
  p.groups = tiles * K::kUnits <= held ? K::kUnits : 1;
  p.items = tiles * p.groups;
  p.inv_runs = reciprocal(p.runs_per_row);
  p.inv_o = reciprocal(p.o_extent);
  p.inv_groups = reciprocal(p.groups);
  LaunchScope scope(stream, tag);
  return launch_kernel_clustered(stream, pair_project_kernel<C, ATT>, 2, 2 * (p.items < held ? p.items : held), kThreads, K::kSmem, tx, tw, tl,
                                 t_rows, t_chan, t_bias, p);
}

}  // namespace

bool trimul_pair_project_ok(const PairRows& r, const void* w_in, const void* w_gout, const void* ab, const void* gl, int dtype) {
  const uintptr_t all = reinterpret_cast<uintptr_t>(w_in) | reinterpret_cast<uintptr_t>(w_gout) | reinterpret_cast<uintptr_t>(ab) |
                        reinterpret_cast<uintptr_t>(gl);
  return (all & 15) == 0 && rows_ok(r, dtype) && (r.c == 128 ? pairs_held<128, false>() > 0 : r.c == 256 && pairs_held<256, false>() > 0);
}

int launch_trimul_pair_project(cudaStream_t stream, const PairRows& r, const void* w_in, const void* w_gout, __nv_bfloat16* ab, int pitch,
                               __nv_bfloat16* gl, const unsigned char* mask, long long m_n, long long m_o, long long m_b, const LnFold* fold) {
  CUtensorMap tr, tc;
  const long long plane = static_cast<long long>(pitch) * r.n;
  KFB_TRY(map4(&tr, gl, r.c, r.n, r.n, r.batch, r.s_n, r.s_o, r.s_b, 64, kRun, 1));
  KFB_TRY(map4(&tc, ab, r.n, r.n, 2 * r.c, r.batch, pitch, plane * r.batch, plane, kRun, 1, 64));
  ProjectParams p = {};
  p.mask = mask;
  p.m_n = m_n;
  p.m_o = m_o;
  p.m_b = m_b;
  if (fold != nullptr) p.fold = *fold;
  return r.c == 128 ? launch<128, false>(stream, r, w_in, w_gout, tr, tc, tc, p, "trimul_project")
                    : launch<256, false>(stream, r, w_in, w_gout, tr, tc, tc, p, "trimul_project");
}

// (Fewer than 16 tiles: most pairs have nothing to do, and a chain of LayerNorm and one unit in each is longer than two launches.  The operator,
// replayed, two launches / one: 24 tokens 17.3 / 18.4 us, 48 19.4 / 20.0, 64 (16 tiles) 21.8 / 21.6, 96 25.3 / 24.8, 251 83.5 / 73.0.)
bool triatt_pair_project_ok(const PairRows& r, const void* w, int heads, int hdp, const void* qkg, const void* vt, const void* bias, int dtype) {
  const uintptr_t all = reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(qkg) | reinterpret_cast<uintptr_t>(vt) |
                        reinterpret_cast<uintptr_t>(bias);
  return r.c == 128 && hdp == 128 && heads <= 8 && (all & 15) == 0 && rows_ok(r, dtype) && row_tiles(r) >= 16 && pairs_held<128, true>() > 0;
}

int launch_triatt_pair_project(cudaStream_t stream, const PairRows& r, const void* w, int heads, __nv_bfloat16* qkg, __nv_bfloat16* vt,
                               __nv_bfloat16* bias, int pitch, float bias_scale) {
  CUtensorMap tr, tc, tb;
  const long long n = r.n, np = pitch;
  KFB_TRY(map4(&tr, qkg, 384, n, n, r.batch, 384, n * 384, n * n * 384, 64, kRun, 1));
  KFB_TRY(map4(&tc, vt, np, n, 128, r.batch, 128 * np, np, 128 * np * n, kRun, 1, 64));
  KFB_TRY(map4(&tb, bias, np, n, heads, r.batch, np, np * n, heads * np * n, kRun, 1, 8));
  ProjectParams p = {};
  p.bias_scale = bias_scale;
  return launch<128, true>(stream, r, w, static_cast<const __nv_bfloat16*>(w) + 512ll * 128, tr, tc, tb, p, "triatt_project");
}

}  // namespace kfb
