// GEMMs onto the float32 residual stream of the samplers:  out = resid + sigmoid(gate) (A . B^T + bias), one tile for each pair of CTAs.
//
// What bounds them.  Five samples of 768 tokens are 3 840 rows of 768 columns: 180 tiles of 128 x 128 on 148 SMs, two rounds of K blocks and
// of an epilogue that fetches gate and residual a chunk at a time (6 800 to 8 900 cycles a tile): 20 us for 9 GFLOP and 30 MB, of which
// either takes 6.
//
// Split.  One round: a CTA pair (cta_group::2) takes 256 rows, four runs of up to 64 consecutive rows (so that a sample of 301 tokens wastes
// 6 % of its tiles and not 22), and as many columns as make one wave of pairs; a pair loads A once for all of them and each half of B once
// for both CTAs.  Residual and gate do not wait for the products: the tile's residual is on its way to shared memory and its gates to the
// registers of the epilogue warps while K goes by.  What is left for the end is one multiply-add per value in place, and every warp sends its
// own 32 x 32 pieces.
// Between events (4 us of them the events'), K = 2 x width: 5 x 768 rows of 768 24.9 -> 18.8 us, of 1 024 30.9 -> 24.9; 5 x 384 rows 17.2 ->
// 15.8 and 20.8 -> 17.1; 2 x 301 of 1 024 16.7 -> 14.7.  Where a cluster shares K (gemm_split.cu) it is left out.
#include <mutex>

#include "common.cuh"
#include "gemm.cuh"

namespace kfb {
namespace {

constexpr int kRun = 64;
constexpr int kThreads = 64 + 32 * kEpiWarps;

template <int BN>
struct Cfg {
  static constexpr int kAStage = 128 * kBK * 2, kBStage = BN / 2 * kBK * 2, kStageBytes = kAStage + kBStage;
  static constexpr int kResid = 128 * BN * 4;
  static constexpr int kFit = (232448 - 1024 - 256 - kResid) / kStageBytes;
  static constexpr int kStages = kFit < 8 ? kFit : 8;
  static constexpr int kSmem = 1024 + kStages * kStageBytes + kResid + 256;
  static constexpr int kChunks = BN / 32, kMine = (kChunks + 1) / 2;     // 32-column chunks: of the tile, of a warp (every other one)
  static constexpr uint32_t kTmemCols = BN <= 64 ? 64 : BN <= 128 ? 128 : 256;
  static_assert(kStages >= 3, "operand ring");
};

struct ResidParams {
  const __nv_bfloat16* gate;
  const float* bias;
  long long g_n, g_o, g_b;
  int n, o_extent, batch, runs_per_row, n_tiles, num_k, has_resid, b_static;
};

template <int BN>
__global__ void __launch_bounds__(kThreads, 1)
gemm_resid_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b, const __grid_constant__ CUtensorMap tm_r,
                  const __grid_constant__ CUtensorMap tm_out, const ResidParams p) {
  using K = Cfg<BN>;
  constexpr int kStages = K::kStages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* s_a = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* s_b = s_a + kStages * K::kAStage;
  uint8_t* s_r = s_b + kStages * K::kBStage;          // [chunk][128 rows][32 columns], 128-byte swizzle
  uint64_t* full = reinterpret_cast<uint64_t*>(s_r + K::kResid);      // [stages], in the leader: both CTAs' copies
  uint64_t* empty = full + kStages;
  uint64_t* resid_in = empty + kStages;
  uint64_t* acc_full = resid_in + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 1);
  static_assert((2 * kStages + 2) * 8 + 4 <= 256, "barriers");

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = static_cast<int>(ptx::cluster_ctarank());
  const int m_tile = static_cast<int>(blockIdx.x >> 1) / p.n_tiles, n_tile = static_cast<int>(blockIdx.x >> 1) - m_tile * p.n_tiles;
  // this CTA's two runs; past the last one: outside the tensors (b = batch)
  int n0[2], o[2], b[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int i = 4 * m_tile + 2 * rank + h, row = i / p.runs_per_row;
    n0[h] = (i - row * p.runs_per_row) * kRun;
    b[h] = row / p.o_extent;
    o[h] = row - b[h] * p.o_extent;
  }

  if (threadIdx.x == 0) {
    ptx::prefetch_tmap(&tm_a);
    ptx::prefetch_tmap(&tm_b);
    ptx::prefetch_tmap(&tm_r);
    ptx::prefetch_tmap(&tm_out);
    for (int i = 0; i < kStages; ++i) {
      ptx::mbar_init(&full[i], 1);
      ptx::mbar_init(&empty[i], 1);
    }
    ptx::mbar_init(resid_in, 1);
    ptx::mbar_init(acc_full, 1);
    ptx::fence_barrier_init();
  }
  if (warp == 1) {
    ptx::tmem_alloc_pair(tmem_slot, K::kTmemCols);
    ptx::tmem_relinquish_pair();
  }
  ptx::tc_fence_before_sync();
  __syncwarp();
  ptx::cluster_sync();
  ptx::tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    // ---------------------------------------------------------------- operands, then (the ring is full) the residual
    if (ptx::elect_one()) {
      const int ahead = p.num_k < kStages ? p.num_k : kStages;
      auto load_b = [&](int st, int kb) {
        if (rank == 0) ptx::mbar_expect_tx(&full[st], 2 * K::kStageBytes);
        ptx::tma_load_4d_pair(s_b + st * K::kBStage, &tm_b, ptx::leader_addr(&full[st]), kb * kBK, n_tile * BN + rank * (BN / 2), 0, 0);
      };
      auto load_a = [&](int st, int kb) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
          ptx::tma_load_4d_pair(s_a + st * K::kAStage + h * (K::kAStage / 2), &tm_a, ptx::leader_addr(&full[st]), kb * kBK, n0[h], o[h], b[h]);
      };
      if (p.b_static)
        for (int i = 0; i < ahead; ++i) load_b(i, i);
      grid_dependency_wait();
      for (int i = 0; i < ahead; ++i) {
        if (!p.b_static) load_b(i, i);
        load_a(i, i);
      }
      if (p.has_resid) {
        ptx::mbar_expect_tx(resid_in, K::kResid);
#pragma unroll 1
        for (int c = 0; c < K::kChunks; ++c)
#pragma unroll
          for (int h = 0; h < 2; ++h)
            ptx::tma_load_4d(s_r + c * 16384 + h * 8192, &tm_r, resid_in, n_tile * BN + c * 32, n0[h], o[h], b[h]);
      }
      grid_dependency_launch();
      int st = 0;
      uint32_t par = 0;
      bool ok = true;
      for (int kb = ahead; kb < p.num_k; ++kb) {
        ok = ptx::mbar_wait(&empty[st], par, 601);
        if (!ok) break;
        load_b(st, kb);
        load_a(st, kb);
        if (++st == kStages) { st = 0; par ^= 1u; }
      }
      // the last products' arrivals at this CTA's barriers, before it may exit
      for (int i = 0; ok && i < ahead; ++i) {
        ok = ptx::mbar_wait(&empty[st], par, 602);
        if (++st == kStages) { st = 0; par ^= 1u; }
      }
    }
  } else if (warp == 1) {
    if (rank == 0 && ptx::elect_one()) {
      constexpr uint32_t idesc = ptx::make_idesc(256, BN, 1);
      const uint64_t a_desc = ptx::make_kmajor_desc<128>(ptx::smem_u32(s_a)), b_desc = ptx::make_kmajor_desc<128>(ptx::smem_u32(s_b));
      int st = 0;
      uint32_t par = 0;
      bool ok = true;
      for (int kb = 0; kb < p.num_k; ++kb) {
        ok = ptx::mbar_wait(&full[st], par, 603);
        if (!ok) break;
        ptx::tc_fence_after_sync();
        const uint64_t ad = a_desc + static_cast<uint64_t>(st * (K::kAStage >> 4)), bd = b_desc + static_cast<uint64_t>(st * (K::kBStage >> 4));
#pragma unroll
        for (int k = 0; k < kBK / 16; ++k) ptx::mma_f16_ss_pair(tmem, ad + k * 2, bd + k * 2, idesc, (kb > 0 || k > 0) ? 1u : 0u);
        ptx::tc_commit_pair(&empty[st]);
        if (++st == kStages) { st = 0; par ^= 1u; }
      }
      if (ok) ptx::tc_commit_pair(acc_full);
    }
  } else {
    // ---------------------------------------------------------------- epilogue: a row per lane, every other 32 columns
    const int quad = warp & 3, share = (warp - 2) >> 2;
    const int h = quad >> 1, r = quad * 32 + lane, n = (h == 0 ? n0[0] : n0[1]) + (quad & 1) * 32 + lane;
    const int oo = h == 0 ? o[0] : o[1], bb = h == 0 ? b[0] : b[1];
    const bool live = n < p.n && bb < p.batch;
    grid_dependency_wait();
    uint4 g[K::kMine][4];
    if (p.gate != nullptr && live) {
      const __nv_bfloat16* row = p.gate + static_cast<long long>(bb) * p.g_b + static_cast<long long>(oo) * p.g_o + static_cast<long long>(n) * p.g_n +
                                 n_tile * BN + share * 32;
#pragma unroll
      for (int c = 0; c < K::kMine; ++c)
#pragma unroll
        for (int i = 0; i < 4; ++i) g[c][i] = 2 * c + share < K::kChunks ? *reinterpret_cast<const uint4*>(row + c * 64 + i * 8) : make_uint4(0, 0, 0, 0);
    } else {
#pragma unroll
      for (int c = 0; c < K::kMine; ++c)
#pragma unroll
        for (int i = 0; i < 4; ++i) g[c][i] = make_uint4(0, 0, 0, 0);
    }
    bool ok = !p.has_resid || __all_sync(0xffffffffu, ptx::mbar_wait(resid_in, 0, 604)) != 0;
    ok = ok && __all_sync(0xffffffffu, ptx::mbar_wait(acc_full, 0, 605)) != 0;
    if (ok) {
      ptx::tc_fence_after_sync();
      const uint32_t t_row = tmem + (static_cast<uint32_t>(quad * 32) << 16) + share * 32;
#pragma unroll
      for (int c = 0; c < K::kMine; ++c) {
        const int chunk = 2 * c + share;
        if (chunk >= K::kChunks) break;
        uint32_t x[32];
        ptx::tmem_ld_32x32b_x32(t_row + c * 64, x);
        ptx::tmem_ld_wait();
        float v[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(x[i]);
        if (p.bias != nullptr) {
          const float4* bias = reinterpret_cast<const float4*>(p.bias + n_tile * BN + chunk * 32);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float4 u = bias[i];
            v[4 * i] += u.x; v[4 * i + 1] += u.y; v[4 * i + 2] += u.z; v[4 * i + 3] += u.w;
          }
        }
        if (p.gate != nullptr) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint32_t w[4] = {g[c][i].x, g[c][i].y, g[c][i].z, g[c][i].w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              v[8 * i + 2 * j] *= sigmoidf_fast(__uint_as_float(w[j] << 16));
              v[8 * i + 2 * j + 1] *= sigmoidf_fast(__uint_as_float(w[j] & 0xffff0000u));
            }
          }
        }
        uint8_t* row = s_r + chunk * 16384 + r * 128;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          float4* cell = reinterpret_cast<float4*>(row + ((i ^ (r & 7)) << 4));
          const float4 u = p.has_resid ? *cell : make_float4(0.f, 0.f, 0.f, 0.f);
          *cell = make_float4(v[4 * i] + u.x, v[4 * i + 1] + u.y, v[4 * i + 2] + u.z, v[4 * i + 3] + u.w);
        }
        ptx::fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0 && n < p.n && bb < p.batch) {       // (lane 0 has the piece's first row)
          ptx::tma_store_4d(&tm_out, s_r + chunk * 16384 + quad * 4096, n_tile * BN + chunk * 32, n, oo, bb);
          ptx::tma_store_commit();
        }
      }
      if (lane == 0) ptx::tma_store_wait_all();
      __syncwarp();
    }
  }

  ptx::tc_fence_before_sync();
  __syncwarp();
  ptx::cluster_sync();      // neither CTA leaves while the other may still read its operands or reach its barriers
  if (warp == 1) {
    ptx::tc_fence_after_sync();
    ptx::tmem_dealloc_pair(tmem, K::kTmemCols);
  }
}

constexpr int kWidths[] = {64, 96, 128, 192, 256};
constexpr int kNumWidths = sizeof(kWidths) / sizeof(kWidths[0]);

// Pairs of CTAs of each width that the current device holds at once (0: none), asked once per device; null without a device.
const int* pairs_held() {
  static std::once_flag once[64];
  static int held[64][kNumWidths];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  int* const of = held[dev & 63];
  std::call_once(once[dev & 63], [&] {
    of[0] = clusters_held(gemm_resid_kernel<64>, 2, kThreads, Cfg<64>::kSmem);
    of[1] = clusters_held(gemm_resid_kernel<96>, 2, kThreads, Cfg<96>::kSmem);
    of[2] = clusters_held(gemm_resid_kernel<128>, 2, kThreads, Cfg<128>::kSmem);
    of[3] = clusters_held(gemm_resid_kernel<192>, 2, kThreads, Cfg<192>::kSmem);
    of[4] = clusters_held(gemm_resid_kernel<256>, 2, kThreads, Cfg<256>::kSmem);
  });
  return of;
}

int row_tiles(const GemmParams& p) { return cdiv(p.batch * p.o_extent * cdiv(p.n_extent, kRun), 4); }

template <int BN>
int launch(cudaStream_t stream, const GemmOperandA& a, const GemmOperandB& b, const GemmParams& p, const char* tag) {
  const EpiSeg& sg = p.seg[0];
  CUtensorMap ta, tb, tr, to;
  {
    const uint64_t dims[4] = {(uint64_t)p.k_extent, (uint64_t)p.n_extent, (uint64_t)p.o_extent, (uint64_t)p.batch};
    const uint64_t str[3] = {(uint64_t)a.s_n * 2, (uint64_t)a.s_o * 2, (uint64_t)a.s_b * 2};
    const uint32_t box[4] = {kBK, kRun, 1, 1};
    KFB_TRY(make_tmap(&ta, a.ptr, 2, 4, dims, str, box, 128));
  }
  {
    const uint64_t dims[4] = {(uint64_t)p.k_extent, (uint64_t)p.n_cols, 1, 1};
    const uint64_t str[3] = {(uint64_t)b.s_col * 2, (uint64_t)b.s_col * p.n_cols * 2, (uint64_t)b.s_col * p.n_cols * 2};
    const uint32_t box[4] = {kBK, BN / 2, 1, 1};
    KFB_TRY(make_tmap(&tb, b.ptr, 2, 4, dims, str, box, 128));
  }
  {
    const uint64_t dims[4] = {(uint64_t)p.n_cols, (uint64_t)p.n_extent, (uint64_t)p.o_extent, (uint64_t)p.batch};
    const uint64_t str[3] = {(uint64_t)sg.s_n * 4, (uint64_t)sg.s_o * 4, (uint64_t)sg.s_b * 4};
    const uint32_t box_r[4] = {32, kRun, 1, 1}, box_o[4] = {32, 32, 1, 1};
    KFB_TRY(make_tmap(&tr, p.resid != nullptr ? p.resid : sg.dst, 4, 4, dims, str, box_r, 128));
    KFB_TRY(make_tmap(&to, sg.dst, 4, 4, dims, str, box_o, 128));
  }
  ResidParams q;
  q.gate = p.gate;
  q.bias = p.col_bias;
  q.g_n = p.g_n;
  q.g_o = p.g_o;
  q.g_b = p.g_b;
  q.n = p.n_extent;
  q.o_extent = p.o_extent;
  q.batch = p.batch;
  q.runs_per_row = cdiv(p.n_extent, kRun);
  q.n_tiles = p.n_cols / BN;
  q.num_k = cdiv(p.k_extent, kBK);
  q.has_resid = p.resid != nullptr;
  q.b_static = p.b_static;
  LaunchScope scope(stream, tag);
  return launch_kernel_clustered(stream, gemm_resid_kernel<BN>, 2, 2 * row_tiles(p) * q.n_tiles, kThreads, Cfg<BN>::kSmem, ta, tb, tr, to, q);
}

}  // namespace

// One wave only: with more, the persistent kernel's epilogues run under the next tile's products.  Of one wave it is the faster of the two
// everywhere (graph replays of SwiGLU and this, K = one and two widths, us, plain tiles / this; the same bits): 128 columns, 64 rows
// 7.6 / 6.5, 3 008 9.3 / 7.6, 15 040 13.5 / 11.3; 768 columns, 1 row 12.5 / 10.5, 129 12.6 / 11.4, 385 13.5 / 11.7, 1 024 14.3 / 13.4,
// 3 840 25.1 / 20.7; K = 1 536 385 16.3 / 13.8, 768 17.6 / 15.1; 1 024 columns, 301 15.3 / 13.5, 3 840 30.0 / 27.5.
int resid_tile(const GemmParams& p, const GemmOperandA& a, const GemmOperandB& b) {
  int best = 0;
  double least = 0.0;
  const EpiSeg& sg = p.seg[0];
  auto extent_ok = [](long long stride, int extent, int unit) { return stride % unit == 0 && (stride != 0 || extent == 1); };
  const bool ok =
      !p.precise && !p.glu && p.nseg == 1 && sg.out_fp32 && sg.s_col == 1 && sg.col_begin == 0 && sg.ncols == p.n_cols && !sg.split && sg.scale == 0.f &&
      (p.gate != nullptr || p.resid != nullptr) && p.resid_scale == nullptr && p.row_stats == nullptr && !(p.rowmask != nullptr && (p.mask_segs & 1)) &&
      !p.b_batched && a.s_k == 0 && a.k_inner == 0 && b.col_inner == 0 && p.n_cols % 64 == 0 && p.k_extent % 8 == 0 && extent_ok(sg.s_n, p.n_extent, 4) &&
      extent_ok(sg.s_o, p.o_extent, 4) && extent_ok(sg.s_b, p.batch, 4) && a.s_n % 8 == 0 && a.s_o % 8 == 0 && a.s_b % 8 == 0 && b.s_col % 8 == 0 &&
      ((reinterpret_cast<uintptr_t>(sg.dst) | reinterpret_cast<uintptr_t>(p.resid) | reinterpret_cast<uintptr_t>(p.gate) |
        reinterpret_cast<uintptr_t>(p.col_bias) | reinterpret_cast<uintptr_t>(a.ptr) | reinterpret_cast<uintptr_t>(b.ptr)) & 15) == 0 &&
      (p.gate == nullptr || (p.g_col == 1 && p.g_n % 8 == 0 && p.g_o % 8 == 0 && p.g_b % 8 == 0)) &&
      static_cast<long long>(p.batch) * p.o_extent * cdiv(p.n_extent, kRun) <= 4096;
  if (!ok) return best;
  const int* const held = pairs_held();
  if (held == nullptr) return best;
  const int blocks = cdiv(p.k_extent, kBK), tiles = row_tiles(p);
  for (int i = 0; i < kNumWidths; ++i) {
    const int bn = kWidths[i];
    if (p.n_cols % bn != 0) continue;
    // a K block: its copies at 64 B per cycle, its products, the issuing thread's turn; beside it launch, fill and the epilogue
    double turn = 256.0 + bn;
    if (turn < 2.0 * bn) turn = 2.0 * bn;
    if (turn < 400.0) turn = 400.0;
    const double t = blocks * turn + 2500.0 + 6.0 * bn;
    if ((best == 0 || t < least) && tiles * (p.n_cols / bn) <= held[i]) {
      best = bn;
      least = t;
    }
  }
  return best;
}

int launch_gemm_resid(cudaStream_t stream, const GemmOperandA& a, const GemmOperandB& b, const GemmParams& p, int bn, const char* tag) {
  switch (bn) {
    case 64: return launch<64>(stream, a, b, p, tag);
    case 96: return launch<96>(stream, a, b, p, tag);
    case 128: return launch<128>(stream, a, b, p, tag);
    case 192: return launch<192>(stream, a, b, p, tag);
    default: return launch<256>(stream, a, b, p, tag);
  }
}

}  // namespace kfb
