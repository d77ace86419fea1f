// Whole transformer stacks of the diffusion network in one call: the kernel sequences of the single operators, issued from
// native code.  A pass over the 24-block token transformer is about 170 launches; issued one operator at a time through the
// Python layer they took 35 us each on the host (8.7 ms for a 96-token step whose kernels need 2.0 ms), issued here about 3 us.
//
// Both stacks start with the conditioning tables: every AdaLN's gate / shift rows and every output gate of every block depend
// on the conditioning s alone, so one LayerNorm of s and two GEMMs (each AdaLN's scale folded into its weight columns) produce
// two wide tables, and the blocks read their columns in place.
#include "attention.cuh"
#include "ops_common.cuh"

using namespace kfb;

namespace {

struct Tables {
  void *gs, *og;              // [rows][gs_cols], [rows][og_cols]: bf16, or fp32 in the fp32-accurate mode
  long long gs_cols, og_cols;
};

size_t tables_bytes(long long rows, int c_s, long long gs_cols, long long og_cols, int precise) {
  const size_t e = precise ? 4 : 2, parts = precise ? 6 : 1;
  return 2 * align_up(static_cast<size_t>(rows) * c_s * 2 * parts, 256) + align_up(static_cast<size_t>(rows) * gs_cols * e, 256) +
         align_up(static_cast<size_t>(rows) * og_cols * e, 256);
}

// rows x [w (n, k)] -> dst (rows, n) with a column bias; precise: x and w are triple splits, dst is fp32
int table_gemm(cudaStream_t stream, const void* x, const void* w, const float* bias, void* dst, long long rows, long long n, int k,
               int precise, const char* tag) {
  GemmParams p = {};
  p.n_extent = static_cast<int>(rows);
  p.o_extent = 1;
  p.batch = 1;
  p.n_cols = static_cast<int>(n);
  p.k_extent = precise ? 6 * k : k;
  p.precise = precise;
  p.nseg = 1;
  p.seg[0] = row_major_seg(dst, static_cast<int>(n), n, 0, 0, precise);
  p.col_bias = bias;
  p.b_static = 1;
  GemmOperandA a = {x, static_cast<long long>(p.k_extent), 0, 0};
  GemmOperandB b = {w, static_cast<long long>(p.k_extent), 0};
  return launch_gemm_bf16(stream, a, b, p, 0, tag);
}

int build_tables(cudaStream_t stream, Carver& cv, Tables& t, const kfb_conditioning& cond, const void* s, int s_dtype, long long rows,
                 int precise) {
  t.gs_cols = cond.gs_cols;
  t.og_cols = cond.og_cols;
  const size_t parts = precise ? 6 : 1, e = precise ? 4 : 2;
  __nv_bfloat16* sn = cv.take<__nv_bfloat16>(static_cast<size_t>(rows) * cond.c_s * parts);
  __nv_bfloat16* sc = cv.take<__nv_bfloat16>(static_cast<size_t>(rows) * cond.c_s * parts);
  t.gs = cv.take<uint8_t>(static_cast<size_t>(rows) * t.gs_cols * e);
  t.og = cv.take<uint8_t>(static_cast<size_t>(rows) * t.og_cols * e);
  const void* raw = sc;
  if (precise) {
    KFB_TRY(launch_layernorm_split(stream, static_cast<const float*>(s), sn, nullptr, nullptr, rows, cond.c_s, cond.c_s, cond.eps, 1));
    KFB_TRY(launch_layernorm_split(stream, static_cast<const float*>(s), sc, nullptr, nullptr, rows, cond.c_s, cond.c_s, 0.f, 0));
  } else {
    KFB_TRY(launch_layernorm(stream, s, sn, nullptr, nullptr, rows, cond.c_s, cond.c_s, cond.c_s, cond.eps, s_dtype, KFB_BF16));
    if (s_dtype == KFB_BF16)
      raw = s;
    else
      KFB_TRY(launch_to_bf16(stream, static_cast<const float*>(s), sc, rows * cond.c_s));
  }
  KFB_TRY(table_gemm(stream, sn, cond.w_gs, cond.b_gs, t.gs, rows, t.gs_cols, cond.c_s, precise, "conditioning_adaln"));
  return table_gemm(stream, raw, cond.w_og, cond.b_og, t.og, rows, t.og_cols, cond.c_s, precise, "conditioning_gates");
}

const void* column(const void* table, long long col, int precise) {
  return static_cast<const uint8_t*>(table) + col * (precise ? 4 : 2);
}

int check_cond(const char* what, const kfb_conditioning* cond, const void* s, int s_dtype, int precise) {
  KFB_CHECK_ARG(cond && s && cond->w_gs && cond->b_gs && cond->w_og && cond->b_og, "%s: null pointer", what);
  KFB_CHECK_ARG(cond->c_s >= 8 && cond->c_s % 8 == 0 && cond->c_s <= 1024, "%s: conditioning channels %d", what, cond->c_s);
  KFB_CHECK_ARG(s_dtype == KFB_FP32 || (s_dtype == KFB_BF16 && !precise), "%s: conditioning dtype %d", what, s_dtype);
  return KFB_OK;
}

size_t attn_ws(int batch, int l, int c, int heads, int precise) {
  return precise ? kfb_apb_workspace_bytes_precise(batch, l, c) : kfb_apb_workspace_bytes(batch, l, c, heads);
}
// Samples of one complex share their pair bias: with head dims of 33 to 64 their attention goes through the kernel that adds a bias
// tile to two batch entries at once (attention_rows.cu), where the other kernel's CTAs (one for 128 queries of a head and sample)
// are more than one wave: 768 tokens x 5 samples, 16 heads of 48, 54 -> 38 us; 256 x 3, one wave, 10 -> 12 us.
bool attn_shares_bias(int precise, int batch, int samples, int l, int heads, int d) {
  return !precise && samples >= 2 && d > 32 && static_cast<long long>(cdiv(l, 128)) * heads * batch > sm_count();
}
size_t trans_ws(long long rows, int c, int hidden, int precise) {
  return precise ? kfb_cond_transition_workspace_bytes_precise(rows, c, hidden) : kfb_cond_transition_workspace_bytes(rows, hidden);
}

}  // namespace

extern "C" {

KFB_API size_t kfb_token_stack_workspace_bytes(int groups, int samples, int s_samples, int l, int c, int c_s, int heads, int hidden,
                                               long long gs_cols, long long og_cols, int precise) {
  const long long rows = static_cast<long long>(groups) * samples * l;
  const size_t a = attn_ws(groups * samples, l, c, heads, precise), t = trans_ws(rows, c, hidden, precise);
  return tables_bytes(static_cast<long long>(groups) * s_samples * l, c_s, gs_cols, og_cols, precise) +
         align_up(static_cast<size_t>(rows) * c * (precise ? 12 : 2), 256) + align_up(sizeof(int2) * groups * samples, 256) +
         align_up(a > t ? a : t, 256);
}

KFB_API int kfb_token_stack_fwd(const kfb_token_block* blocks, int n_blocks, const kfb_conditioning* cond, const void* a, void* out,
                                int act_dtype, const void* s, int s_dtype, const void* pair_bias, long long bias_block_stride,
                                long long bias_head_stride, long long bias_ld, const unsigned char* mask, void* workspace,
                                size_t workspace_bytes, int groups, int samples, int s_samples, int l, int c, int heads, int hidden,
                                float eps, int precise, void* stream_) {
  KFB_CHECK_ARG(blocks && n_blocks >= 1 && a && out && pair_bias && mask && workspace, "token_stack: null pointer");
  KFB_CHECK_ARG(act_dtype == KFB_FP32 || (act_dtype == KFB_BF16 && !precise), "token_stack: activation dtype %d", act_dtype);
  KFB_TRY(check_cond("token_stack", cond, s, s_dtype, precise));
  KFB_CHECK_ARG(groups >= 1 && samples >= 1 && l >= 1 && (s_samples == 1 || s_samples == samples), "token_stack: groups %d samples %d (%d) l %d",
                groups, samples, s_samples, l);
  KFB_CHECK_ARG(heads >= 1 && c % heads == 0 && c % 8 == 0 && hidden % 128 == 0, "token_stack: c=%d heads=%d hidden=%d", c, heads, hidden);
  KFB_CHECK_ARG(cond->gs_cols == 4ll * c * n_blocks && cond->og_cols == 2ll * c * n_blocks, "token_stack: conditioning tables of %lld / %lld columns",
                cond->gs_cols, cond->og_cols);
  KFB_CHECK_ARG(bias_ld >= l && bias_head_stride >= bias_ld * l && (precise || (bias_ld % 8 == 0 && bias_head_stride % 8 == 0 && bias_block_stride % 8 == 0)),
                "token_stack: bias pitch %lld, head stride %lld", bias_ld, bias_head_stride);
  KFB_CHECK_ARG((reinterpret_cast<uintptr_t>(workspace) & 255) == 0, "token_stack: workspace must be 256-byte aligned");
  const size_t need = kfb_token_stack_workspace_bytes(groups, samples, s_samples, l, c, cond->c_s, heads, hidden, cond->gs_cols,
                                                      cond->og_cols, precise);
  KFB_CHECK_ARG(workspace_bytes >= need, "token_stack: workspace %zu < %zu bytes", workspace_bytes, need);
  cudaStream_t stream = as_stream(stream_);
  const int batch = groups * samples;
  const int share = samples / s_samples;            // consecutive samples that use the same conditioning rows
  const long long rows = static_cast<long long>(batch) * l;
  Carver cv(workspace);
  Tables t;
  KFB_TRY(build_tables(stream, cv, t, *cond, s, s_dtype, static_cast<long long>(groups) * s_samples * l, precise));
  void* an = cv.take<uint8_t>(static_cast<size_t>(rows) * c * (precise ? 12 : 2));   // fp32-accurate: triple-split rows
  int2* mask_rows = cv.take<int2>(batch);
  if (!attn_shares_bias(precise, batch, samples, l, heads, c / heads)) {
    mask_rows = nullptr;
  } else {
    AttnParams m = {};
    m.batch = batch;
    m.lk = l;
    m.mask = mask;
    m.mask_lo_extent = samples;
    m.m_hi = l;
    m.m_k = 1;
    m.row_info = mask_rows;
    KFB_TRY(launch_attention_mask_rows(stream, m));   // once for all blocks
  }
  const size_t ab = attn_ws(batch, l, c, heads, precise), tb = trans_ws(rows, c, hidden, precise);
  const size_t op_bytes = ab > tb ? ab : tb;
  void* op_ws = cv.take<uint8_t>(op_bytes);
  const int ada_dtype = precise ? KFB_FP32_PRECISE : act_dtype, op_dtype = precise ? KFB_FP32_PRECISE : act_dtype;
  const size_t bias_e = precise ? 4 : 2;
  const void* cur = a;
  for (int i = 0; i < n_blocks; ++i) {
    const kfb_token_block& w = blocks[i];
    KFB_TRY(launch_adaln(stream, cur, an, column(t.gs, 4ll * c * i, precise), rows, c, share, l, eps, ada_dtype,
                         precise ? KFB_FP32_PRECISE : KFB_BF16, t.gs_cols, 1));
    ApbArgs r;
    r.x = an;
    r.x_is_split = precise;
    r.w_static = 1;
    r.pair_bias = static_cast<const uint8_t*>(pair_bias) + bias_block_stride * i * bias_e;
    r.ldb = bias_ld; r.bias_hs = bias_head_stride; r.bias_div = samples;
    r.mask = mask; r.mask_share = samples; r.rows = mask_rows;
    r.w_proj = w.w_proj; r.proj_bias = w.proj_bias; r.w_out = w.w_out; r.out_bias = w.out_bias;
    r.out_gate = column(t.og, 2ll * c * i, precise); r.gate_share = share; r.gate_ld = t.og_cols;
    r.out = out; r.resid = cur;
    r.workspace = op_ws; r.workspace_bytes = op_bytes;
    r.batch = batch; r.l = l; r.c = c; r.heads = heads; r.out_dtype = op_dtype;
    KFB_TRY(apb_run(stream, r));
    cur = out;                                      // from here on the stream is updated in place
    KFB_TRY(launch_adaln(stream, cur, an, column(t.gs, 4ll * c * i + 2ll * c, precise), rows, c, share, l, eps, ada_dtype,
                         precise ? KFB_FP32_PRECISE : KFB_BF16, t.gs_cols, 1));
    KFB_TRY(cond_transition_run(stream, an, precise, 1, w.w_swiglu, w.w_tout, column(t.og, 2ll * c * i + c, precise), t.og_cols, out, cur, op_ws,
                                op_bytes, rows, c, hidden, share, l, op_dtype));
  }
  return KFB_OK;
}

KFB_API size_t kfb_atom_stack_workspace_bytes(int groups, int samples, int l, int c, int c_s, int heads, int hidden, long long gs_cols,
                                              long long og_cols) {
  const long long rows = static_cast<long long>(groups) * samples * l;
  const size_t a = kfb_apb_window_workspace_bytes(groups * samples, l, c, heads), t = trans_ws(rows, c, hidden, 0);
  return tables_bytes(static_cast<long long>(groups) * l, c_s, gs_cols, og_cols, 0) + 2 * align_up(static_cast<size_t>(rows) * c * 2, 256) +
         align_up(a > t ? a : t, 256);
}

KFB_API int kfb_atom_stack_fwd(const kfb_atom_block* blocks, int n_blocks, const kfb_conditioning* cond, const void* a, void* out,
                               int act_dtype, const void* s, int s_dtype, const void* window_bias, long long bias_windows,
                               const unsigned char* mask, int mask_share, int bias_share, void* workspace, size_t workspace_bytes,
                               int groups, int samples, int l, int c, int heads, int hidden, float eps, void* stream_) {
  KFB_CHECK_ARG(blocks && n_blocks >= 1 && a && out && window_bias && mask && workspace, "atom_stack: null pointer");
  KFB_CHECK_ARG(act_dtype == KFB_FP32 || act_dtype == KFB_BF16, "atom_stack: activation dtype %d", act_dtype);
  KFB_TRY(check_cond("atom_stack", cond, s, s_dtype, 0));
  KFB_CHECK_ARG(groups >= 1 && samples >= 1 && l >= 32 && l % 32 == 0, "atom_stack: groups %d samples %d atoms %d", groups, samples, l);
  KFB_CHECK_ARG(cond->gs_cols == 6ll * c * n_blocks && cond->og_cols == 2ll * c * n_blocks, "atom_stack: conditioning tables of %lld / %lld columns",
                cond->gs_cols, cond->og_cols);
  KFB_CHECK_ARG((reinterpret_cast<uintptr_t>(workspace) & 255) == 0, "atom_stack: workspace must be 256-byte aligned");
  const size_t need = kfb_atom_stack_workspace_bytes(groups, samples, l, c, cond->c_s, heads, hidden, cond->gs_cols, cond->og_cols);
  KFB_CHECK_ARG(workspace_bytes >= need, "atom_stack: workspace %zu < %zu bytes", workspace_bytes, need);
  cudaStream_t stream = as_stream(stream_);
  const int batch = groups * samples;
  const long long rows = static_cast<long long>(batch) * l, srows = static_cast<long long>(groups) * l;
  Carver cv(workspace);
  Tables t;
  KFB_TRY(build_tables(stream, cv, t, *cond, s, s_dtype, srows, 0));
  __nv_bfloat16* xq = cv.take<__nv_bfloat16>(static_cast<size_t>(rows) * c);
  __nv_bfloat16* xk = cv.take<__nv_bfloat16>(static_cast<size_t>(rows) * c);
  const size_t ab = kfb_apb_window_workspace_bytes(batch, l, c, heads), tb = trans_ws(rows, c, hidden, 0);
  const size_t op_bytes = ab > tb ? ab : tb;
  void* op_ws = cv.take<uint8_t>(op_bytes);
  const void* cur = a;
  for (int i = 0; i < n_blocks; ++i) {
    const kfb_atom_block& w = blocks[i];
    const long long g0 = 6ll * c * i;
    KFB_TRY(launch_adaln_two(stream, cur, xq, xk, column(t.gs, g0, 0), column(t.gs, g0 + 2ll * c, 0), rows, c, samples, l, eps, act_dtype, t.gs_cols, 1));
    // the output gate is shared by the samples: query row r reads gate row r % (l) of its group
    for (int g = 0; g < groups; ++g) {
      const size_t row0 = static_cast<size_t>(g) * samples * l, e = act_dtype == KFB_FP32 ? 4 : 2;
      const size_t nb = static_cast<size_t>(samples) / bias_share * (l / 32);
      KFB_TRY(kfb_apb_window_fwd(xq + row0 * c, xk + row0 * c,
                                 static_cast<const __nv_bfloat16*>(window_bias) + (static_cast<size_t>(i) * heads * bias_windows + g * nb) * 4096,
                                 mask + static_cast<size_t>(g) * (samples / mask_share) * l, w.w_q, w.q_bias, w.w_kv, w.w_out, w.out_bias,
                                 column(t.og, 2ll * c * i + static_cast<long long>(g) * l * t.og_cols, 0), l, t.og_cols,
                                 static_cast<uint8_t*>(out) + row0 * c * e, static_cast<const uint8_t*>(cur) + row0 * c * e, op_ws, op_bytes,
                                 samples, l, c, heads, bias_share, mask_share, static_cast<int>(bias_windows), act_dtype, stream_));
    }
    cur = out;
    KFB_TRY(launch_adaln(stream, cur, xq, column(t.gs, g0 + 4ll * c, 0), rows, c, samples, l, eps, act_dtype, KFB_BF16, t.gs_cols, 1));
    KFB_TRY(cond_transition_run(stream, xq, 0, 1, w.w_swiglu, w.w_tout, column(t.og, 2ll * c * i + c, 0), t.og_cols, out, cur, op_ws, op_bytes,
                                rows, c, hidden, samples, l, act_dtype));
  }
  return KFB_OK;
}

}  // extern "C"
