// Host launcher of the persistent tcgen05 GEMM (see gemm.cuh for the kernel).
#include <limits.h>
#include <stdio.h>
#include <string.h>

#include <mutex>

#include "common.cuh"
#include "gemm.cuh"
#include "layernorm.cuh"

namespace kfb {

// Tiles in flight: CTAs, or pairs of them, that the current device holds at once (0: it holds no pair).  Once per device and kernel, whose
// shared memory it also allows.
template <int BN, bool GLU, bool AUX, bool PRECISE, bool SWAP, bool STATS, bool PAIR, bool TWIN>
static int tiles_held(int* held) {
  constexpr auto kernel = gemm_bf16_kernel<BN, GLU, AUX, PRECISE, SWAP, STATS, PAIR, TWIN>;
  static std::once_flag once[64];
  static int resident[64];
  int dev = 0;
  KFB_CUDA(cudaGetDevice(&dev));
  cudaError_t attr_err = cudaSuccess;
  std::call_once(once[dev & 63], [&] {
    if (PAIR) {     // (a multiprocessor without a neighbour to pair with stays idle)
      resident[dev & 63] = clusters_held(kernel, 2, gemm_threads<AUX, STATS, TWIN>(), GemmCfg<BN, PAIR>::kSmemBytes);
      return;
    }
    attr_err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, GemmCfg<BN, PAIR>::kSmemBytes);
    resident[dev & 63] = attr_err == cudaSuccess ? sm_count() : 0;
  });
  KFB_CUDA(attr_err);
  *held = resident[dev & 63];
  return KFB_OK;
}

template <int BN, bool GLU, bool AUX, bool PRECISE, bool SWAP = false, bool STATS = false, bool PAIR = false, bool TWIN = false>
static int launch_variant(cudaStream_t stream, const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap* tout,
                          const GemmParams& p, const char* tag) {
  using Cfg = GemmCfg<BN, PAIR>;
  constexpr auto kernel = gemm_bf16_kernel<BN, GLU, AUX, PRECISE, SWAP, STATS, PAIR, TWIN>;
  constexpr int threads = gemm_threads<AUX, STATS, TWIN>();
  int held = 0;
  KFB_TRY((tiles_held<BN, GLU, AUX, PRECISE, SWAP, STATS, PAIR, TWIN>(&held)));
  KFB_CHECK_ARG(held > 0, "GEMM: the device holds no tile of this kernel");
  const int total = p.num_m_tiles * p.num_n_tiles;
  const int grid = total < held ? total : held;     // (pairs count as one)
  GemmParams q = p;
  {
    // the persistent loops step by the grid size: its digits in the (n tile, row block, outer, batch) index
    if (q.rows_first) {
      q.step_n_tile = grid / q.n_blocks;
      q.step_nb = grid - q.step_n_tile * q.n_blocks;
    } else {
      const int m_step = grid / q.num_n_tiles;
      q.step_n_tile = grid - m_step * q.num_n_tiles;
      q.step_nb = m_step % q.n_blocks;
      const int rest = m_step / q.n_blocks;
      q.step_o = rest % q.o_extent;
      q.step_b = rest / q.o_extent;
    }
  }
  {
    LaunchScope scope(stream, tag);
    KFB_TRY(launch_kernel_clustered(stream, kernel, PAIR ? 2 : 1, PAIR ? 2 * grid : grid, threads, Cfg::kSmemBytes, ta, tb, tout[0], tout[1],
                                    tout[2], q));
  }
  return KFB_OK;
}

static int launch_pair(cudaStream_t stream, const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap* tout, GemmParams p, const char* tag) {
  using Cfg = GemmCfg<256, true>;
  p.stages = Cfg::stages_for(p.aux ? p.aux_bufs * (p.aux_gate + p.aux_resid) * Cfg::kAuxTileBytes : p.glu ? Cfg::kGluStagingBytes : Cfg::kStagingBytes);
  if (p.twin)
    return p.glu ? launch_variant<256, true, false, false, false, false, true, true>(stream, ta, tb, tout, p, tag)
                 : launch_variant<256, false, false, false, false, false, true, true>(stream, ta, tb, tout, p, tag);
  if (p.glu) return launch_variant<256, true, false, false, false, false, true>(stream, ta, tb, tout, p, tag);
  if (p.aux) return launch_variant<256, false, true, false, false, false, true>(stream, ta, tb, tout, p, tag);
  return launch_variant<256, false, false, false, false, false, true>(stream, ta, tb, tout, p, tag);
}

template <int BN>
static int launch_bn(cudaStream_t stream, const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap* tout,
                     GemmParams p, const char* tag) {
  using Cfg = GemmCfg<BN>;
  p.stages = Cfg::stages_for(p.aux ? p.aux_bufs * (p.aux_gate + p.aux_resid) * Cfg::kAuxTileBytes + (p.stats_in_kernel ? kStatsBytes : 0)
                                   : p.xpose ? Cfg::kXposeStagingBytes : Cfg::kStagingBytes);
  if constexpr (BN == 32) {
    KFB_CHECK_ARG(!p.glu && !p.aux, "32-column tiles exist for the plain kernels only");
    if (p.precise) return launch_variant<32, false, false, true>(stream, ta, tb, tout, p, tag);
    return launch_variant<32, false, false, false>(stream, ta, tb, tout, p, tag);
  } else {
  if constexpr (BN <= 128) {
    if (p.precise) {
      if (p.glu) return launch_variant<BN, true, false, true>(stream, ta, tb, tout, p, tag);
      return launch_variant<BN, false, false, true>(stream, ta, tb, tout, p, tag);
    }
  }
  if constexpr (BN == 256) {
    if (p.glu && p.swap) {
      p.stages = Cfg::stages_for(Cfg::kSwapStagingBytes);
      if (p.twin) return launch_variant<BN, true, false, false, true, false, false, true>(stream, ta, tb, tout, p, tag);
      return launch_variant<BN, true, false, false, true>(stream, ta, tb, tout, p, tag);
    }
  }
  if (p.glu) {
    p.stages = Cfg::stages_for(Cfg::kGluStagingBytes);
    if constexpr (BN == 256) {
      if (p.twin) return launch_variant<BN, true, false, false, false, false, false, true>(stream, ta, tb, tout, p, tag);
    }
    return launch_variant<BN, true, false, false>(stream, ta, tb, tout, p, tag);
  }
  if constexpr (BN == 64 || BN == 128) {
    if (p.stats_in_kernel) return launch_variant<BN, false, true, false, false, true>(stream, ta, tb, tout, p, tag);
  }
  if constexpr (BN >= 64) {
    if (p.aux) return launch_variant<BN, false, true, false>(stream, ta, tb, tout, p, tag);
  }
  if constexpr (BN == 128) {
    if (p.twin) return launch_variant<BN, false, false, false, false, false, false, true>(stream, ta, tb, tout, p, tag);
  }
  return launch_variant<BN, false, false, false>(stream, ta, tb, tout, p, tag);
  }
}

// Narrower tiles for GEMMs of few rows: with the default width a sampler step's projections of 96 tokens fill 6 to 32 of the 148
// SMs, and a tile's time is the trip of its operands through one SM.  Modelled time of a width: waves x (K blocks x bytes of a
// stage / 64 B per cycle + epilogue); it is only taken where the default leaves SMs idle, so that large GEMMs keep their tiles.
// (The GLU kernels pair value and gate columns inside 128-channel blocks: 64 columns are their narrowest tile.)
static int narrow_tile(const GemmParams& p, int bn) {
  const long long sms = sm_count();
  if (static_cast<long long>(p.num_m_tiles) * cdiv(p.n_cols, bn) >= sms) return bn;
  const int num_k = p.precise ? 3 * cdiv(p.k_extent / 6, kBK) : cdiv(p.k_extent, kBK);
  const int lo = p.glu ? 64 : 32;
  double best = 1e30;
  int pick = bn;
  for (int w = bn; w >= lo; w /= 2) {
    const long long tiles = static_cast<long long>(p.num_m_tiles) * cdiv(p.n_cols, w);
    const double waves = static_cast<double>((tiles + sms - 1) / sms);
    const double t = waves * (num_k * (16384.0 + 128.0 * w) / 64.0 + 600.0 + 12.0 * w);
    if (t < best) { best = t; pick = w; }
  }
  return pick;
}

// CTA pairs (PAIR in gemm.cuh) pay where the main loop is long enough to hide the epilogue of a tile twice as wide and the tiles are at
// least a wave of pairs.  Measured, one CTA -> pair: triangle contraction at 768 tokens 108 -> 99 us (128 channels), 201 -> 180 (256);
// at 400 tokens (seven K blocks) 71 -> 62; SwiGLU of 256 channels at 768 x 768 rows 585 -> 472, its output projection (K = 1 024) 362 ->
// 318; token transformer, 5 x 768 rows of 768: projection 35 -> 29, SwiGLU 24.5 -> 22.5; conditioning tables of those rows (six, staged)
// 415 -> 390.  The other side of the lines: SwiGLU of 128 channels (two K blocks) 106 -> 107; gate projection of 256 (four, plain) 105 -> 109;
// contraction at 333 tokens (three row blocks, a quarter of the pairs' work padding) 49.7 -> 51.6; float32 output projections with gate and
// residual 22.4 -> 23.5.
static bool pair_tile(const GemmParams& p, int bn) {
  if (p.precise || bn < 128 || p.n_cols < 256 || p.glu == GLU_SIGMOID) return false;
  const int num_k = cdiv(p.k_extent, kBK), pairs = cdiv(p.n_blocks, 2);
  if (num_k < (p.glu ? 4 : 6) || (2 * pairs - p.n_blocks) * 8 > p.n_blocks) return false;
  if (2ll * pairs * p.o_extent * p.batch * cdiv(p.n_cols, 256) < sm_count()) return false;
  for (int i = 0; i < p.nseg; ++i) {
    const EpiSeg& sg = p.seg[i];
    const bool channel_major = sg.s_n == 1 && sg.s_col != 1;      // whole swapped tiles, behind the row-major segments
    if (sg.col_begin % 256 != 0 || sg.out_fp32) return false;
    if (channel_major && (p.glu || ((p.mask_segs >> i) & 1) || (i == 0 && (p.gate != nullptr || p.resid != nullptr)))) return false;
    if (!channel_major && (sg.s_col != 1 || (i > 0 && p.seg[i - 1].s_n == 1 && p.seg[i - 1].s_col != 1))) return false;
  }
  // (a device, or the part of one that this process may use, without two free multiprocessors in a cluster's reach; every pair kernel
  // takes a multiprocessor's whole shared memory, so that one of them answers for all)
  int held = 0;
  const bool known = tiles_held<256, true, false, false, false, false, true, true>(&held) == KFB_OK;
  if (!known) cudaGetLastError();
  return known && held > 0;
}

static long long* g_trace_buf = nullptr;
static char g_trace_tag[64] = "";
void set_gemm_trace(long long* device_buffer, const char* tag) {
  g_trace_buf = device_buffer;
  snprintf(g_trace_tag, sizeof(g_trace_tag), "%s", tag ? tag : "");
}

int launch_gemm_bf16(cudaStream_t stream, const GemmOperandA& a, const GemmOperandB& b, GemmParams p, int force_bn,
                     const char* tag, GemmExtra* extra) {
  if (extra != nullptr) extra->taken = false;
  KFB_CHECK_ARG(p.n_extent > 0 && p.o_extent > 0 && p.batch > 0 && p.n_cols > 0 && p.k_extent > 0, "empty GEMM");
  KFB_CHECK_ARG(p.nseg >= 1 && p.nseg <= 3, "GEMM needs 1..3 output segments");
  p.n_blocks = cdiv(p.n_extent, kBM);
  p.num_m_tiles = p.n_blocks * p.o_extent * p.batch;
  int bn = force_bn;
  if (bn == 0) bn = p.n_cols >= 256 ? 256 : (p.n_cols > 64 ? 128 : 64);
  if (p.precise && bn > 128) bn = 128;  // the fp32-accurate variant keeps four accumulators in tensor memory
  if (a.s_k == 0 && a.k_inner == 0 && b.col_inner == 0 && (p.precise ? !p.glu : p.glu != GLU_SIGMOID)) bn = narrow_tile(p, bn);
  // K shared by a cluster where rows are few (the gate / residual epilogue of 128 float32 columns takes the other kernel 8 000 cycles)
  const bool plain_operands = a.s_k == 0 && a.k_inner == 0 && b.col_inner == 0;
  SplitPlan plan = {0, 0};
  if (force_bn == 0 && static_cast<long long>(p.num_m_tiles) * cdiv(p.n_cols, bn) <= sm_count())
    plan = split_plan(p, plain_operands, split_cycles(p.precise, bn, cdiv(p.precise ? p.k_extent / 6 : p.k_extent, kBK)) +
                                             ((p.gate != nullptr || p.resid != nullptr) && !p.precise ? 50.0 : 12.0) * bn);
  // One wave of pairs onto a residual stream otherwise: the bits of the plain tiles.  (It has no say in whether K is shared, which they and
  // the sum's order hang on.)
  if (plan.bn == 0 && force_bn == 0) {
    const int onto = resid_tile(p, a, b);
    if (onto != 0) return launch_gemm_resid(stream, a, b, p, onto, tag);
  }
  if (plan.bn != 0) bn = plan.bn;
  p.pair = plan.bn == 0 && pair_tile(p, bn) && a.s_k == 0 && a.k_inner == 0 && b.col_inner == 0;
  if (p.pair) bn = 256;
  // One row-major float32 segment with a gate and / or a residual (the output projections of the sampler's float32 activation
  // stream): 128-column tiles whose epilogue moves gate, residual and output through per-warp shared-memory tiles.
  p.xpose = 0;
  if (plan.bn == 0 && !p.precise && !p.glu && force_bn == 0 && p.nseg == 1 && a.s_k == 0 && a.k_inner == 0 && b.col_inner == 0 &&
      (p.gate != nullptr || p.resid != nullptr) && p.resid_scale == nullptr) {
    const EpiSeg& sg = p.seg[0];
    const bool seg_ok = sg.out_fp32 && sg.vec && sg.s_col == 1 && sg.col_begin == 0 && !sg.split && sg.ncols % 32 == 0 &&
                        sg.s_n % 4 == 0 && sg.s_o % 4 == 0 && sg.s_b % 4 == 0 &&
                        (p.resid == nullptr || (reinterpret_cast<uintptr_t>(p.resid) & 15) == 0);
    const bool gate_ok = p.gate == nullptr ||
                         (p.g_col == 1 && (reinterpret_cast<uintptr_t>(p.gate) & 15) == 0 && p.g_n % 8 == 0 && p.g_o % 8 == 0 &&
                          p.g_b % 8 == 0);
    if (seg_ok && gate_ok) {
      p.xpose = 1;
      if (bn > 128) bn = 128;
    }
  }
  if (p.xpose) p.pair = 0;
  // Gate / residual prefetch and staged output: one row-major bf16 segment of whole 32-column chunks, aligned strides.  Two buffers
  // of 128-column tiles (each set is loaded while the one before is in the epilogue); with a long K and the residual only, one
  // buffer of 256-column tiles: its load hides behind the K loop, and A is read once.
  p.aux = p.aux_gate = p.aux_resid = 0;
  p.aux_bufs = 2;
  if (plan.bn == 0 && !p.precise && !p.xpose && !p.glu && p.nseg == 1 && p.seg[0].vec && !p.seg[0].out_fp32 && p.seg[0].s_col == 1 &&
      p.seg[0].col_begin == 0 && p.seg[0].ncols == p.n_cols && (p.gate != nullptr || p.resid != nullptr) && bn >= 64 && p.n_cols % 32 == 0) {
    const EpiSeg& sg = p.seg[0];
    const bool ok_o = (reinterpret_cast<uintptr_t>(sg.dst) & 15) == 0 && sg.s_n % 8 == 0 && sg.s_o % 8 == 0 && (sg.s_o != 0 || p.o_extent == 1) &&
                      sg.s_b % 8 == 0 && (sg.s_b != 0 || p.batch == 1);
    const bool ok_g = p.gate == nullptr || (p.g_col == 1 && (reinterpret_cast<uintptr_t>(p.gate) & 15) == 0 && p.g_n % 8 == 0 && p.g_n != 0 &&
                                            p.g_o % 8 == 0 && (p.g_o != 0 || p.o_extent == 1) && p.g_b % 8 == 0 && (p.g_b != 0 || p.batch == 1));
    const bool ok_r = p.resid == nullptr || (reinterpret_cast<uintptr_t>(p.resid) & 15) == 0;
    if (ok_o && ok_g && ok_r) {
      p.aux = 1;
      p.aux_gate = p.gate != nullptr;
      p.aux_resid = p.resid != nullptr;
      if (bn == 256) {
        if (p.k_extent >= 512 && p.aux_gate + p.aux_resid == 1)
          p.aux_bufs = 1;
        else
          bn = 128;
      }
    }
  }
  if (bn != 256) p.pair = 0;
  // few rows with statistics to take: twice the tiles, half the epilogue (pair block of 64 tokens, two of them: 142.5 -> 138.9 us;
  // 251 tokens, which have the tiles: as they were)
  if (p.aux && bn == 128 && a.s_k != 0 && p.row_stats != nullptr && static_cast<long long>(p.num_m_tiles) * cdiv(p.n_cols, 64) <= sm_count()) bn = 64;
  KFB_CHECK_ARG(bn == 32 || bn == 64 || bn == 128 || bn == 256, "unsupported BN %d", bn);
  // LayerNorm statistics of K-outer rows: taken by the kernel itself where it has the warps for it, by a pass before it otherwise.  The
  // statistics hold a stage of the ring a little longer, which costs little where a tile is few stages or comes from L2 (768 x 768 rows
  // of 128 channels: pass + kernel 33 + 110 us, kernel alone 124; 400 x 400 of 256, 82 MB: 34 + 67, 87), and more than the pass where
  // rows of four stages, read once for each of two column tiles, come from HBM (768 x 768 of 256, 302 MB: 58 + 215, 294).
  p.stats_in_kernel = p.aux && bn <= 128 && a.s_k != 0 && p.row_stats != nullptr &&
                      (p.k_extent <= 128 || static_cast<long long>(a.s_k) * p.k_extent * 2 <= (96ll << 20));
  if (a.s_k != 0 && p.row_stats != nullptr && !p.stats_in_kernel)
    KFB_TRY(launch_cm_stats(stream, static_cast<const __nv_bfloat16*>(a.ptr), p.row_stats, a.s_k, p.k_extent, a.s_k,
                            p.stats_eps));
  if (p.precise) KFB_CHECK_ARG(p.k_extent % 48 == 0, "precise GEMM: K=%d is not six equal parts of whole 16-byte pieces", p.k_extent);
  if (p.glu) KFB_CHECK_ARG(p.n_cols % bn == 0, "GLU GEMM needs n_cols (%d) to be a multiple of the N tile (%d)", p.n_cols, bn);
  for (int i = 0; i < p.nseg; ++i) KFB_CHECK_ARG(p.seg[i].col_begin % 32 == 0, "segment start must be a multiple of 32");
  p.trace = (g_trace_buf != nullptr && strcmp(g_trace_tag, tag) == 0) ? g_trace_buf : nullptr;
  p.num_n_tiles = cdiv(p.n_cols, bn);
  if (p.pair) {
    p.n_blocks = cdiv(p.n_blocks, 2);
    p.num_m_tiles = p.n_blocks * p.o_extent * p.batch;
  }

  CUtensorMap ta, tb;
  p.a_mn_major = a.s_k != 0 ? 1 : 0;
  p.k_inner = a.k_inner;
  KFB_CHECK_ARG(a.k_inner == b.k_inner, "split K: both operands must be split alike (%d, %d)", a.k_inner, b.k_inner);
  if (p.precise) {
    // the parts are a dimension of their own: a K block never runs into the next part, whatever K is
    const int k = p.k_extent / 6;
    KFB_CHECK_ARG(!p.a_mn_major && !p.k_inner, "precise GEMM: plain K-major operands only");
    const uint64_t dims[5] = {(uint64_t)k, (uint64_t)p.n_extent, (uint64_t)p.o_extent, 6, (uint64_t)p.batch};
    const uint64_t str[4] = {(uint64_t)a.s_n * 2, (uint64_t)a.s_o * 2, (uint64_t)k * 2, (uint64_t)a.s_b * 2};
    const uint32_t box[5] = {kBK, kBM, 1, 1, 1};
    KFB_TRY(make_tmap(&ta, a.ptr, 2, 5, dims, str, box, 128));
  } else if (p.k_inner) {
    KFB_CHECK_ARG(!p.a_mn_major && !p.precise && p.k_inner % kBK == 0 && p.k_extent % p.k_inner == 0,
                  "split K: pieces of %d elements (multiple of %d) in K=%d, plain bf16 GEMM", p.k_inner, kBK, p.k_extent);
    const uint64_t dims[5] = {(uint64_t)p.k_inner, (uint64_t)p.n_extent, (uint64_t)p.o_extent, (uint64_t)(p.k_extent / p.k_inner),
                              (uint64_t)p.batch};
    const uint64_t str[4] = {(uint64_t)a.s_n * 2, (uint64_t)a.s_o * 2, (uint64_t)a.s_k_hi * 2, (uint64_t)a.s_b * 2};
    const uint32_t box[5] = {kBK, kBM, 1, 1, 1};
    KFB_TRY(make_tmap(&ta, a.ptr, 2, 5, dims, str, box, 128));
  } else if (p.a_mn_major) {
    KFB_CHECK_ARG(a.s_n == 1 && p.k_extent % kBK == 0 && !p.precise && !p.glu, "K-outer A operand: rows must be contiguous, K a "
                  "multiple of %d, plain bf16 GEMM", kBK);
    const uint64_t dims[4] = {(uint64_t)p.n_extent, (uint64_t)p.k_extent, (uint64_t)p.o_extent, (uint64_t)p.batch};
    const uint64_t str[3] = {(uint64_t)a.s_k * 2, (uint64_t)a.s_o * 2, (uint64_t)a.s_b * 2};
    const uint32_t box[4] = {64, kBK, 1, 1};
    KFB_TRY(make_tmap(&ta, a.ptr, 2, 4, dims, str, box, 128));
  } else {
    const uint64_t dims[4] = {(uint64_t)p.k_extent, (uint64_t)p.n_extent, (uint64_t)p.o_extent, (uint64_t)p.batch};
    const uint64_t str[3] = {(uint64_t)a.s_n * 2, (uint64_t)a.s_o * 2, (uint64_t)a.s_b * 2};
    const uint32_t box[4] = {kBK, kBM, 1, 1};
    KFB_TRY(make_tmap(&ta, a.ptr, 2, 4, dims, str, box, 128));
  }
  {
    const int inner = b.col_inner > 0 ? b.col_inner : p.n_cols;
    if (b.col_inner > 0)
      KFB_CHECK_ARG(p.n_cols % inner == 0 && inner % bn == 0, "split B operand: %d columns in pieces of %d, tile %d", p.n_cols,
                    inner, bn);
    p.b_col_inner = inner;
    if (p.precise) {
      const int k = p.k_extent / 6;
      const uint64_t dims[5] = {(uint64_t)k, (uint64_t)inner, (uint64_t)(p.n_cols / inner), 6, (uint64_t)(p.b_batched ? p.batch : 1)};
      const uint64_t str[4] = {(uint64_t)b.s_col * 2, (uint64_t)b.s_col_hi * 2, (uint64_t)k * 2, (uint64_t)b.s_b * 2};
      const uint32_t box[5] = {kBK, (uint32_t)bn, 1, 1, 1};
      KFB_TRY(make_tmap(&tb, b.ptr, 2, 5, dims, str, box, 128));
    } else if (p.k_inner) {
      const uint64_t dims[5] = {(uint64_t)p.k_inner, (uint64_t)inner, (uint64_t)(p.n_cols / inner),
                                (uint64_t)(p.k_extent / p.k_inner), (uint64_t)(p.b_batched ? p.batch : 1)};
      const uint64_t str[4] = {(uint64_t)b.s_col * 2, (uint64_t)b.s_col_hi * 2, (uint64_t)b.s_k_hi * 2, (uint64_t)b.s_b * 2};
      const uint32_t box[5] = {kBK, (uint32_t)bn, 1, 1, 1};
      KFB_TRY(make_tmap(&tb, b.ptr, 2, 5, dims, str, box, 128));
    } else {
    const uint64_t dims[4] = {(uint64_t)p.k_extent, (uint64_t)inner, (uint64_t)(p.n_cols / inner),
                              (uint64_t)(p.b_batched ? p.batch : 1)};
    const uint64_t str[3] = {(uint64_t)b.s_col * 2, (uint64_t)b.s_col_hi * 2, (uint64_t)b.s_b * 2};
    const uint32_t box[4] = {kBK, (uint32_t)(p.pair || (p.glu && bn < 256) ? bn / 2 : bn), 1, 1};
    KFB_TRY(make_tmap(&tb, b.ptr, 2, 4, dims, str, box, 128));
    }
  }
  if (plan.bn != 0) return launch_gemm_split(stream, ta, tb, p, plan, tag);
  // channel-major bf16 segments that satisfy the TMA alignment rules are stored through shared memory
  CUtensorMap tout[3];
  tout[0] = tout[1] = tout[2] = ta;  // placeholders (never dereferenced unless a segment selects them)
  int next_slot = 0;
  // a sigmoid-GLU GEMM whose only output is channel-major bf16 is computed in the swapped orientation
  p.swap = (p.glu == GLU_SIGMOID && bn == 256 && p.nseg == 1 && !p.precise && p.seg[0].s_n == 1 && p.seg[0].s_col != 1 &&
            !p.seg[0].out_fp32 && p.seg[0].col_begin == 0 && p.n_cols % 256 == 0 && p.col_bias == nullptr &&
            p.gate == nullptr && p.resid == nullptr && (p.rowmask == nullptr || (p.mask_segs & 1)))
               ? 1 : 0;
  // ... and, when the destination satisfies the copy engine's alignment rules, stored as whole tiles by TMA
  p.swap_staged = 0;
  if (p.swap) {
    const EpiSeg& sg = p.seg[0];
    const bool aligned = (reinterpret_cast<uintptr_t>(sg.dst) & 15) == 0 && sg.s_col % 8 == 0 &&
                         (sg.s_o % 8 == 0 && (sg.s_o != 0 || p.o_extent == 1)) && (sg.s_b % 8 == 0 && (sg.s_b != 0 || p.batch == 1));
    if (aligned) {
      const uint64_t dims[4] = {(uint64_t)p.n_extent, (uint64_t)p.o_extent, (uint64_t)sg.ncols, (uint64_t)p.batch};
      const uint64_t str[3] = {(uint64_t)sg.s_o * 2, (uint64_t)sg.s_col * 2, (uint64_t)sg.s_b * 2};
      const uint32_t box[4] = {64, 1, kBM, 1};
      KFB_TRY(make_tmap(&tout[0], sg.dst, 2, 4, dims, str, box, 128));
      p.swap_staged = 1;
      next_slot = 1;
    }
  }
  // ... and the same rows' plain columns of a second matrix, as more column tiles of the launch: up to two K blocks, where a tile is
  // mostly output (gate logits of 128 channels, 768 x 768 rows: 110 + 57 us in two launches, 149 in one; 64 x 64: a launch of 4 us
  // less; of 256 channels, four K blocks: 316 + 107, 431)
  p.glu_tiles = p.num_n_tiles;
  if (extra != nullptr && p.swap_staged && p.k_extent <= 128 && extra->cols % 128 == 0 && (reinterpret_cast<uintptr_t>(extra->w) & 15) == 0 && extra->w_ld % 8 == 0 &&
      (reinterpret_cast<uintptr_t>(extra->dst) & 15) == 0 && extra->s_n % 8 == 0 && extra->s_o % 8 == 0 && (extra->s_o != 0 || p.o_extent == 1) &&
      extra->s_b % 8 == 0 && (extra->s_b != 0 || p.batch == 1)) {
    const uint64_t wdims[4] = {(uint64_t)p.k_extent, (uint64_t)extra->cols, 1, 1};
    const uint64_t wstr[3] = {(uint64_t)extra->w_ld * 2, (uint64_t)extra->w_ld * extra->cols * 2, (uint64_t)extra->w_ld * extra->cols * 2};
    const uint32_t wbox[4] = {kBK, 128, 1, 1};
    KFB_TRY(make_tmap(&tout[1], extra->w, 2, 4, wdims, wstr, wbox, 128));
    const uint64_t dims[4] = {(uint64_t)extra->cols, (uint64_t)p.n_extent, (uint64_t)p.o_extent, (uint64_t)p.batch};
    const uint64_t str[3] = {(uint64_t)extra->s_n * 2, (uint64_t)extra->s_o * 2, (uint64_t)extra->s_b * 2};
    const uint32_t box[4] = {64, kBM, 1, 1};
    KFB_TRY(make_tmap(&tout[2], extra->dst, 2, 4, dims, str, box, 128));
    p.num_n_tiles += extra->cols / 128;
    extra->taken = true;
  }
  // trailing channel-major bf16 segments that start on a tile boundary are computed in the swapped orientation as well
  // (plain BN = 128 kernel): the threads then store runs of consecutive positions directly
  p.swap_col_begin = INT_MAX;
  if ((bn == 128 || p.pair) && !p.glu && !p.precise && !p.a_mn_major) {
    for (int i = p.nseg - 1; i >= 0; --i) {
      const EpiSeg& sg = p.seg[i];
      const bool cm = sg.s_n == 1 && sg.s_col != 1 && !sg.out_fp32 && !sg.split && sg.col_begin % bn == 0 &&
                      !((p.mask_segs >> i) & 1) && (i > 0 || (p.gate == nullptr && p.resid == nullptr));
      if (!cm) break;
      p.swap_col_begin = sg.col_begin;
    }
  }
  for (int i = 0; i < p.nseg; ++i) {
    EpiSeg& sg = p.seg[i];
    sg.tma_slot = -1;
    if (p.swap || sg.col_begin >= p.swap_col_begin) continue;
    const bool aligned = (reinterpret_cast<uintptr_t>(sg.dst) & 15) == 0 && sg.s_o % 8 == 0 && sg.s_col % 8 == 0 &&
                         (sg.s_b % 8 == 0 || p.batch == 1) && (sg.s_o != 0 || p.o_extent == 1);
    if (sg.s_n == 1 && sg.s_col != 1 && !sg.out_fp32 && aligned && next_slot < 2 && !p.precise) {
      const uint64_t dims[4] = {(uint64_t)p.n_extent, (uint64_t)p.o_extent, (uint64_t)sg.ncols, (uint64_t)p.batch};
      const uint64_t str[3] = {(uint64_t)sg.s_o * 2, (uint64_t)sg.s_col * 2, (uint64_t)sg.s_b * 2};
      const uint32_t box[4] = {kBM, 1, 32, 1};
      KFB_TRY(make_tmap(&tout[next_slot], sg.dst, 2, 4, dims, str, box, 0));
      sg.tma_slot = next_slot++;
    }
  }
  if (p.aux) {
    KFB_CHECK_ARG(next_slot == 0, "GEMM: gate / residual prefetch beside a staged segment");
    const EpiSeg& sg = p.seg[0];
    const uint32_t box[4] = {64, kBM, 1, 1};
    const uint64_t dims[4] = {(uint64_t)p.n_cols, (uint64_t)p.n_extent, (uint64_t)p.o_extent, (uint64_t)p.batch};
    const uint64_t ostr[3] = {(uint64_t)sg.s_n * 2, (uint64_t)sg.s_o * 2, (uint64_t)sg.s_b * 2};
    const uint64_t gstr[3] = {(uint64_t)p.g_n * 2, (uint64_t)p.g_o * 2, (uint64_t)p.g_b * 2};
    if (p.aux_gate) KFB_TRY(make_tmap(&tout[0], p.gate, 2, 4, dims, gstr, box, 128));
    if (p.aux_resid) KFB_TRY(make_tmap(&tout[1], p.resid, 2, 4, dims, ostr, box, 128));
    KFB_TRY(make_tmap(&tout[2], sg.dst, 2, 4, dims, ostr, box, 128));
  }
  // full tiles of one row-major bf16 segment of the plain BN = 128 kernel leave through shared memory and a TMA store
  p.rm_seg = -1;
  p.rm_slot = 0;
  const bool rm_plain = (bn == 128 || p.pair) && !p.glu;
  const bool rm_glu = bn == 256 && p.glu && !p.swap;      // the GLU kernel: 128 output columns per tile
  if ((rm_plain || rm_glu) && !p.precise && !p.aux && !p.a_mn_major && next_slot == 0) {
    for (int i = 0; i < p.nseg; ++i) {
      const EpiSeg& sg = p.seg[i];
      if (rm_glu && (i != 0 || sg.ncols % 128 != 0)) break;   // the GLU route handles segment 0 made of whole tiles only
      const bool ok_seg = sg.s_col == 1 && sg.vec && !sg.out_fp32 && sg.col_begin % 128 == 0 && sg.ncols >= 128 &&
                          sg.col_begin < p.swap_col_begin && (reinterpret_cast<uintptr_t>(sg.dst) & 15) == 0 && sg.s_n % 8 == 0 &&
                          (sg.s_o % 8 == 0 && (sg.s_o != 0 || p.o_extent == 1)) && (sg.s_b % 8 == 0 && (sg.s_b != 0 || p.batch == 1)) &&
                          !((p.mask_segs >> i) & 1) && (i != 0 || (p.gate == nullptr && p.resid == nullptr));
      if (!ok_seg) continue;
      const uint64_t dims[4] = {(uint64_t)sg.ncols, (uint64_t)p.n_extent, (uint64_t)p.o_extent, (uint64_t)p.batch};
      const uint64_t str[3] = {(uint64_t)sg.s_n * 2, (uint64_t)sg.s_o * 2, (uint64_t)sg.s_b * 2};
      const uint32_t box[4] = {64, kBM, 1, 1};
      KFB_TRY(make_tmap(&tout[0], sg.dst, 2, 4, dims, str, box, 128));
      p.rm_seg = i;
      break;
    }
  }
  // two epilogue groups: every tile staged or swapped, nothing else to do to it, and more than one tile for each CTA (with one, the
  // second group has nothing to do)
  p.twin = 0;
  {
    const EpiSeg& s0 = p.seg[0];
    const bool bare = p.gate == nullptr && p.resid == nullptr && p.row_stats == nullptr;
    const bool whole_columns = s0.ncols % (p.glu ? 128 : bn) == 0 || (p.nseg == 1 && p.col_bias == nullptr && !p.glu);
    const long long tiles = static_cast<long long>(p.num_m_tiles) * p.num_n_tiles * (p.pair ? 2 : 1);
    if (bare && !p.precise && !p.aux && !p.a_mn_major && (tiles > sm_count() || p.num_n_tiles != p.glu_tiles)) {
      if (p.swap)
        p.twin = p.swap_staged || p.num_n_tiles != p.glu_tiles;
      else if (p.glu)
        p.twin = p.rm_seg == 0 && p.nseg == 1 && p.col_bias == nullptr && whole_columns && (p.mask_segs & 1) == 0;
      else
        p.twin = p.rm_seg == 0 && whole_columns && s0.col_begin == 0 && s0.scale == 0.f && (reinterpret_cast<uintptr_t>(p.col_bias) & 15) == 0 &&
                 (p.nseg == 1 || p.seg[1].col_begin >= p.swap_col_begin);
    }
  }
  // Weights that the L2 does not keep beside what is written (a stack's conditioning tables: 57 MB and 28) are read once where the row blocks
  // of a column tile follow each other; the rows, which are then read for every column tile, are few.  Both tables of 24 blocks of 768
  // channels, 3 840 rows: 415 -> 380 us; of 16 of 1 024, 301 rows, float32-accurate: 209 -> 184.
  p.rows_first = p.o_extent == 1 && p.batch == 1 && p.n_blocks > 1 && p.num_n_tiles > p.n_blocks && !p.a_mn_major && p.num_n_tiles == p.glu_tiles &&
                 static_cast<long long>(p.n_cols) * p.k_extent * 2 > (16ll << 20);
  if (p.pair) return launch_pair(stream, ta, tb, tout, p, tag);
  switch (bn) {
    case 32: return launch_bn<32>(stream, ta, tb, tout, p, tag);
    case 64: return launch_bn<64>(stream, ta, tb, tout, p, tag);
    case 128: return launch_bn<128>(stream, ta, tb, tout, p, tag);
    default: return launch_bn<256>(stream, ta, tb, tout, p, tag);
  }
}

}  // namespace kfb
