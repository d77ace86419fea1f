// GEMMs of few rows, K shared by a cluster of CTAs:  D[row, col] = epilogue(sum_k A[row, k] * B[col, k])
//
// What bounds them.  The output projections of a sampler step of 96 tokens (one row block, 768 columns) are 24 tiles of 32 columns on
// 148 SMs, and a tile's time is its K blocks one after the other: a K block takes the producing and the multiplying thread about 400
// cycles whatever its width (float32-accurate: 1 430, six products of three pairs of parts), 24 of them for the transition.  Here
// `split` CTAs of a cluster take a contiguous share of the K blocks each, of a wider tile; every CTA leaves its float32 partial tile in
// its own shared memory, and after one cluster barrier the CTAs share the tile's elements: each sums the partial tiles of all
// (distributed shared memory, in the order of K) and applies the epilogue.  The partial tile lies in shared memory, so a warp takes it in
// whichever order suits global memory: 4 rows x 128 bytes per access to residual, gate and output.
// Between CUDA events (4 us of them the events'), one sample: 96 tokens of 768 channels, bf16 operands, attention output projection 12.5 ->
// 10.6 us, transition's 13.9 -> 11.6 (mean with the atoms'); 301 tokens of 1 024, float32-accurate, 26.1 -> 18.8 and 31.6 -> 21.2.
// The sums lose less: of the tensor core's truncated accumulation steps each CTA makes its share only (K = 2 048, 301 rows, against 64
// bits: relative error 2.1e-6 -> 4.7e-7).
//
//   warp 0      TMA producer          warp 1   MMA issuer
//   warps 2..9  partial tile from tensor memory to shared memory, then the sum and the epilogue; what that needs from global memory
//               is fetched while the tensor core works.
#include <mutex>

#include "common.cuh"
#include "gemm.cuh"

namespace kfb {
namespace {

__device__ __forceinline__ uint32_t cluster_addr(const void* p, uint32_t rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(ptx::smem_u32(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ float4 ld_cluster(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}

constexpr int kSplitThreads = 64 + 32 * kEpiWarps;
constexpr int kMaxSplit = 8;

template <int BN>
struct SplitCfg {
  using G = GemmCfg<BN>;
  static constexpr int kPartialBytes = kBM * BN * 4;
  static constexpr int kFit = (G::kSmemBytes - 1024 - kPartialBytes - G::kBarrierBytes) / G::kStageBytes;
  static constexpr int kStages = kFit < G::kMaxStages ? kFit : G::kMaxStages;
  static constexpr int kSmem = 1024 + kStages * G::kStageBytes + kPartialBytes + G::kBarrierBytes;
};

// Offset of 16 bytes (four columns) of the partial tile: 128-byte rows per chunk of 32 columns, pieces rotated by the row so that both the
// writers (a row per lane) and the readers (four rows per warp) spread over the banks.
template <int BN>
__device__ __forceinline__ int partial_offset(int row, int chunk, int piece) {
  return row * (BN * 4) + chunk * 128 + ((piece ^ (row & 7)) << 4);
}

template <int BN, bool PRECISE>
__global__ void __launch_bounds__(kSplitThreads, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b, const GemmParams p, int split) {
  using Cfg = SplitCfg<BN>;
  using G = GemmCfg<BN>;
  constexpr int kStages = Cfg::kStages, kChunks = BN / 32;
  constexpr int kTmemCols = PRECISE ? 2 * BN : BN;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* s_a = smem;
  uint8_t* s_b = s_a + kStages * G::kAStage;
  uint8_t* s_part = s_b + kStages * G::kBStage;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(s_part + Cfg::kPartialBytes);
  uint64_t* empty_bar = full_bar + kStages;
  uint64_t* tmem_full = empty_bar + kStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_full + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    ptx::prefetch_tmap(&tm_a);
    ptx::prefetch_tmap(&tm_b);
    for (int s = 0; s < kStages; ++s) {
      ptx::mbar_init(&full_bar[s], 1);
      ptx::mbar_init(&empty_bar[s], 1);
    }
    ptx::mbar_init(tmem_full, 1);
    ptx::fence_barrier_init();
  }
  if (warp == 1) {
    ptx::tmem_alloc(tmem_slot, kTmemCols);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;

  // the cluster's tile, and this CTA's share of its K blocks
  const int rank = blockIdx.x % split, tile = blockIdx.x / split;
  const int n_tile = tile % p.num_n_tiles, m_tile = tile / p.num_n_tiles;
  const int nb = m_tile % p.n_blocks, rest = m_tile / p.n_blocks;
  const int o = rest % p.o_extent, b = rest / p.o_extent;
  const int blocks = PRECISE ? (p.k_extent / 6 + kBK - 1) / kBK : (p.k_extent + kBK - 1) / kBK;
  const int kb0 = blocks * rank / split, kb1 = blocks * (rank + 1) / split;
  const int loads = (PRECISE ? 3 : 1) * (kb1 - kb0);       // ring stages: of a K block three, (x0, w0), (x1, w1), (x2, w2)

  auto load_a = [&](int i) {
    const int st = i % kStages;
    if constexpr (PRECISE)
      ptx::tma_load_5d(s_a + st * G::kAStage, &tm_a, &full_bar[st], (kb0 + i / 3) * kBK, nb * kBM, o, part_a(i % 3), b);
    else
      ptx::tma_load_4d(s_a + st * G::kAStage, &tm_a, &full_bar[st], (kb0 + i) * kBK, nb * kBM, o, b);
  };
  auto load_b = [&](int i) {
    const int st = i % kStages;
    if constexpr (PRECISE)
      ptx::tma_load_5d(s_b + st * G::kBStage, &tm_b, &full_bar[st], (kb0 + i / 3) * kBK, n_tile * BN, 0, part_b(i % 3), 0);
    else
      ptx::tma_load_4d(s_b + st * G::kBStage, &tm_b, &full_bar[st], (kb0 + i) * kBK, n_tile * BN, 0, 0);
  };
  // weights that are not the previous launch's are fetched under its tail (see gemm.cuh)
  int ahead = 0;
  if (warp == 0 && p.b_static && ptx::elect_one()) {
    ahead = loads < kStages ? loads : kStages;
    for (int i = 0; i < ahead; ++i) {
      ptx::mbar_expect_tx(&full_bar[i], G::kStageBytes);
      load_b(i);
    }
  }
  grid_dependency_wait();

  const EpiSeg& sg = p.seg[0];
  // element groups of the tile: 4 rows x 32 columns, dealt out to the CTAs and their epilogue warps
  const int epi = warp - 2;
  struct Item {
    int row, col;             // of this lane: row of the tile, first of four columns of the output
    int off;                  // in the partial tile
    bool live;
    long long at, gate_at;
  };
  auto item_of = [&](int j) {
    Item it;
    const int idx = rank + split * (epi + kEpiWarps * j);
    const int chunk = idx % kChunks, group = idx / kChunks, piece = lane & 7;
    it.row = group * 4 + (lane >> 3);
    it.col = n_tile * BN + chunk * 32 + piece * 4;
    const int n = nb * kBM + it.row;
    it.live = group < kBM / 4 && n < p.n_extent && it.col < sg.ncols;
    it.off = partial_offset<BN>(it.row & (kBM - 1), chunk, piece);
    it.at = static_cast<long long>(b) * sg.s_b + static_cast<long long>(o) * sg.s_o + static_cast<long long>(n) * sg.s_n + it.col;
    it.gate_at = static_cast<long long>(b) * p.g_b + static_cast<long long>(o) * p.g_o + static_cast<long long>(n) * p.g_n + it.col;
    return it;
  };
  struct Extra {
    float4 resid;
    float4 gate;     // the factor's logits
  };
  auto fetch = [&](const Item& it) {
    Extra e = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
    if (!it.live) return e;
    if (p.resid != nullptr) e.resid = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p.resid) + it.at);
    if (p.gate != nullptr) {
      if constexpr (PRECISE) {
        e.gate = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p.gate) + it.gate_at);
      } else {
        const uint2 u = *reinterpret_cast<const uint2*>(p.gate + it.gate_at);
        e.gate = make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
      }
    }
    return e;
  };
  constexpr int kPre = 2;          // groups per warp whose residual and gate are fetched before the sums exist
  Extra pre[kPre];

  if (warp == 0) {
    if (ptx::elect_one()) {
      grid_dependency_launch();
      for (int i = 0; i < loads; ++i) {
        const int st = i % kStages;
        if (i >= ahead) {
          if (!ptx::mbar_wait(&empty_bar[st], ((i / kStages) & 1) ^ 1, 501)) break;
          ptx::mbar_expect_tx(&full_bar[st], G::kStageBytes);
          load_b(i);
        }
        load_a(i);
      }
    }
  } else if (warp == 1) {
    if (ptx::elect_one()) {
      constexpr uint32_t idesc = ptx::make_idesc(kBM, BN, 1);
      bool ok = true;
      uint64_t ad[3], bd[3];
      auto product = [&](uint64_t x, uint64_t w, uint32_t d, bool first) {
#pragma unroll
        for (int k = 0; k < kBK / 16; ++k) ptx::mma_f16_ss(d, x + k * 2, w + k * 2, idesc, (first && k == 0) ? 0u : 1u);
      };
      for (int i = 0; ok && i < loads; i += PRECISE ? 3 : 1) {
#pragma unroll
        for (int j = 0; j < (PRECISE ? 3 : 1); ++j) {
          const int st = (i + j) % kStages;
          ok = ok && ptx::mbar_wait(&full_bar[st], ((i + j) / kStages) & 1, 502);
          if (!ok) break;
          ptx::tc_fence_after_sync();
          ad[j] = ptx::make_kmajor_desc<128>(ptx::smem_u32(s_a + st * G::kAStage));
          bd[j] = ptx::make_kmajor_desc<128>(ptx::smem_u32(s_b + st * G::kBStage));
          // (float32-accurate: the small products in an accumulator of their own, as in gemm.cuh)
          if (j == 0) {
            product(ad[0], bd[0], tmem, i == 0);
          } else {
            product(ad[0], bd[j], tmem + BN, i == 0 && j == 1);
            product(ad[j], bd[0], tmem + BN, false);
            if (j == 1) product(ad[1], bd[1], tmem + BN, false);
          }
        }
        if (!ok) break;
#pragma unroll
        for (int j = 0; j < (PRECISE ? 3 : 1); ++j) ptx::tc_commit(&empty_bar[(i + j) % kStages]);
      }
      if (ok) ptx::tc_commit(tmem_full);
    }
  } else {
#pragma unroll
    for (int j = 0; j < kPre; ++j) pre[j] = fetch(item_of(j));
    const int quad = warp & 3, r = quad * 32 + lane;
    if (__all_sync(0xffffffffu, ptx::mbar_wait(tmem_full, 0, 503))) {
      ptx::tc_fence_after_sync();
      const uint32_t t_row = tmem + (static_cast<uint32_t>(quad * 32) << 16);
#pragma unroll 1
      for (int chunk = epi >> 2; chunk < kChunks; chunk += kEpiWarps / 4) {
        uint32_t x[32];
        ptx::tmem_ld_32x32b_x32(t_row + chunk * 32, x);
        ptx::tmem_ld_wait();
        if constexpr (PRECISE) {
          uint32_t y[32];
          ptx::tmem_ld_32x32b_x32(t_row + BN + chunk * 32, y);
          ptx::tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) x[i] = __float_as_uint(__uint_as_float(x[i]) + __uint_as_float(y[i]));
        }
#pragma unroll
        for (int q = 0; q < 8; ++q)
          *reinterpret_cast<uint4*>(s_part + partial_offset<BN>(r, chunk, q)) = make_uint4(x[4 * q], x[4 * q + 1], x[4 * q + 2], x[4 * q + 3]);
      }
    }
  }
  ptx::tc_fence_before_sync();
  __syncwarp();
  ptx::cluster_sync();
  if (warp == 1) {
    ptx::tc_fence_after_sync();
    ptx::tmem_dealloc(tmem, kTmemCols);
  }
  if (warp >= 2) {
    const int per_cta = (kBM / 4 * kChunks - rank + split - 1) / split;        // element groups of this CTA
    for (int j = 0; epi + kEpiWarps * j < per_cta; ++j) {
      const Item it = item_of(j);
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
      for (int s = 0; s < split; ++s) {
        const float4 v = ld_cluster(cluster_addr(s_part + it.off, s));
        acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
      }
      if (!it.live) continue;
      Extra e;
      if (j == 0) e = pre[0];
      else if (j == 1) e = pre[1];
      else e = fetch(it);
      if (p.col_bias != nullptr) {
        acc.x += p.col_bias[it.col]; acc.y += p.col_bias[it.col + 1];
        acc.z += p.col_bias[it.col + 2]; acc.w += p.col_bias[it.col + 3];
      }
      if (p.gate != nullptr) {
        acc.x *= PRECISE ? sigmoidf_exact(e.gate.x) : sigmoidf_fast(e.gate.x);
        acc.y *= PRECISE ? sigmoidf_exact(e.gate.y) : sigmoidf_fast(e.gate.y);
        acc.z *= PRECISE ? sigmoidf_exact(e.gate.z) : sigmoidf_fast(e.gate.z);
        acc.w *= PRECISE ? sigmoidf_exact(e.gate.w) : sigmoidf_fast(e.gate.w);
      }
      if (p.resid != nullptr) { acc.x += e.resid.x; acc.y += e.resid.y; acc.z += e.resid.z; acc.w += e.resid.w; }
      *reinterpret_cast<float4*>(reinterpret_cast<float*>(sg.dst) + it.at) = acc;
    }
  }
  __syncwarp();
  ptx::cluster_sync();     // nobody leaves while a partial tile is still being read
}

template <int BN, bool PRECISE>
struct SplitLauncher {
  // clusters of `split` CTAs that the device holds at once (0: the size cannot be launched)
  static int resident(int dev, int split) {
    static std::once_flag once[64];
    static int held[64][kMaxSplit + 1];
    std::call_once(once[dev & 63], [&] {
      for (int s = 2; s <= kMaxSplit; ++s) held[dev & 63][s] = clusters_held(gemm_split_kernel<BN, PRECISE>, s, kSplitThreads, SplitCfg<BN>::kSmem);
    });
    return split <= kMaxSplit ? held[dev & 63][split] : 0;
  }
  static int launch(cudaStream_t stream, const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p, int split, const char* tag) {
    LaunchScope scope(stream, tag);
    return launch_kernel_clustered(stream, gemm_split_kernel<BN, PRECISE>, split, p.num_m_tiles * p.num_n_tiles * split, kSplitThreads,
                                   SplitCfg<BN>::kSmem, ta, tb, p, split);
  }
};

template <bool PRECISE>
int resident(int dev, int bn, int split) {
  return bn == 32 ? SplitLauncher<32, PRECISE>::resident(dev, split) : bn == 64 ? SplitLauncher<64, PRECISE>::resident(dev, split)
                                                                                  : SplitLauncher<128, PRECISE>::resident(dev, split);
}

}  // namespace

// float32 results only: a bf16 residual stream turns a last bit that depends on the number of rows into 0.5 % of the result after four
// blocks, and its output projections (shorter epilogues, K of the pair track's width) gained 1 to 2 us of 11 to 14.
SplitPlan split_plan(const GemmParams& p, bool plain_operands, double other_cycles) {
  SplitPlan best = {0, 0};
  const EpiSeg& sg = p.seg[0];
  const bool ok = plain_operands && sg.out_fp32 && !p.glu && !p.b_batched && p.nseg == 1 && sg.col_begin == 0 && sg.s_col == 1 && sg.ncols == p.n_cols && !sg.split &&
                  sg.scale == 0.f && p.row_stats == nullptr && p.resid_scale == nullptr && !(p.rowmask != nullptr && (p.mask_segs & 1)) &&
                  p.n_cols % 4 == 0 && sg.s_n % 4 == 0 && sg.s_o % 4 == 0 && sg.s_b % 4 == 0 &&
                  ((reinterpret_cast<uintptr_t>(sg.dst) | reinterpret_cast<uintptr_t>(p.resid)) & 15) == 0 &&
                  (p.gate == nullptr || (p.g_col == 1 && p.g_n % 4 == 0 && p.g_o % 4 == 0 && p.g_b % 4 == 0 &&
                                         (reinterpret_cast<uintptr_t>(p.gate) & (p.precise ? 15 : 7)) == 0));
  if (!ok) return best;
  const int blocks = cdiv(p.precise ? p.k_extent / 6 : p.k_extent, kBK), sms = sm_count();
  double least = 0.8 * other_cycles;
  // (cheapest first: the two K blocks of a least share and what comes beside them do not fit)
  if (blocks < 2 || least < split_cycles(p.precise, 32, 1) + 2500.0) return best;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return best;
  for (int bn = 32; bn <= 128; bn *= 2) {
    const int tiles = p.num_m_tiles * cdiv(p.n_cols, bn);
    for (int s : {2, 3, 4, 6, 8}) {
      if (s > blocks || static_cast<long long>(tiles) * s > sms) break;
      // beside the main loop: barriers and launch, element groups one after the other, partial tiles of the others at 16 B per cycle
      const double t = split_cycles(p.precise, bn, cdiv(blocks, s)) + 2000.0 + 500.0 * cdiv(bn, 8 * s) + 32.0 * bn * (s - 1) / s;
      // (a cluster's CTAs share a GPC: 24 clusters of six need not all fit, though 144 CTAs do)
      if (t < least && tiles <= (p.precise ? resident<true>(dev, bn, s) : resident<false>(dev, bn, s))) {
        least = t;
        best = {bn, s};
      }
    }
  }
  return best;
}

int launch_gemm_split(cudaStream_t stream, const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p, const SplitPlan& plan, const char* tag) {
  if (p.precise) {
    switch (plan.bn) {
      case 32: return SplitLauncher<32, true>::launch(stream, ta, tb, p, plan.split, tag);
      case 64: return SplitLauncher<64, true>::launch(stream, ta, tb, p, plan.split, tag);
      default: return SplitLauncher<128, true>::launch(stream, ta, tb, p, plan.split, tag);
    }
  }
  switch (plan.bn) {
    case 32: return SplitLauncher<32, false>::launch(stream, ta, tb, p, plan.split, tag);
    case 64: return SplitLauncher<64, false>::launch(stream, ta, tb, p, plan.split, tag);
    default: return SplitLauncher<128, false>::launch(stream, ta, tb, p, plan.split, tag);
  }
}

}  // namespace kfb
