// A block of the pair stacks as one native call (kfb_pair_block_fwd): the operators' kernel sequences one after the other, the
// pair and single tensors updated in place after the first operator.  The block of a 64-token complex is 22 launches of 3 to
// 8 us; issued operator by operator from Python the host took 0.6 ms for them.
#include "ops_common.cuh"

using namespace kfb;

namespace {

size_t max_of(size_t a, size_t b) { return a > b ? a : b; }

size_t operator_bytes(const kfb_pair_block& k, int batch, int n, int precise) {
  const long long pos = static_cast<long long>(batch) * n * n, rows = static_cast<long long>(batch) * n;
  size_t m = precise ? kfb_trimul_workspace_bytes_precise(batch, n, k.c) : kfb_trimul_workspace_bytes(batch, n, k.c) + trimul_fold_bytes(k.c);
  if (k.has_attention)
    m = max_of(m, precise ? kfb_triatt_workspace_bytes_precise(batch, n, k.c, k.tri_heads) : kfb_triatt_workspace_bytes(batch, n, k.c, k.tri_heads));
  m = max_of(m, precise ? kfb_transition_workspace_bytes_precise(pos, k.c, k.hidden_z) : kfb_transition_workspace_bytes(pos, k.c, k.hidden_z));
  if (k.has_single) {
    m = max_of(m, precise ? kfb_pair_bias_workspace_bytes_precise(batch, n, k.c) : kfb_pair_bias_workspace_bytes(batch, n, k.c));
    m = max_of(m, precise ? kfb_apb_workspace_bytes_precise(batch, n, k.c_s) : kfb_apb_workspace_bytes(batch, n, k.c_s, k.heads));
    m = max_of(m, precise ? kfb_transition_workspace_bytes_precise(rows, k.c_s, k.hidden_s) : kfb_transition_workspace_bytes(rows, k.c_s, k.hidden_s));
  }
  return align_up(m, 256);
}

size_t mask_rows_bytes(const kfb_pair_block& k, int batch, int n) {
  return k.has_attention ? align_up(sizeof(int2) * 2 * batch * n, 256) : 0;
}

int bias_pitch(int n, int precise) { return precise ? n : pitch16(n); }

}  // namespace

extern "C" {

KFB_API size_t kfb_pair_block_workspace_bytes(const kfb_pair_block* blk, int batch, int n, int precise) {
  size_t m = operator_bytes(*blk, batch, n, precise) + mask_rows_bytes(*blk, batch, n);
  if (blk->has_single)
    m += align_up(static_cast<size_t>(batch) * blk->heads * n * bias_pitch(n, precise) * (precise ? 4 : 2), 256) +
         align_up(static_cast<size_t>(batch) * n * blk->c_s * (precise ? 4 : 2), 256);
  return m;
}

KFB_API int kfb_pair_block_fwd(const kfb_pair_block* blk, const void* z, void* z_out, int z_dtype, const void* s, void* s_out, int s_dtype,
                               const unsigned char* pair_mask, const unsigned char* mask, void* workspace, size_t workspace_bytes,
                               int batch, int n, void* stream) {
  KFB_CHECK_ARG(blk && z && z_out && pair_mask && workspace, "pair_block: null pointer");
  const kfb_pair_block& k = *blk;
  const int precise = z_dtype == KFB_FP32_PRECISE;
  KFB_CHECK_ARG(is_dtype(z_dtype), "pair_block: bad dtype %d", z_dtype);
  if (k.has_single) {
    KFB_CHECK_ARG(s && s_out && mask && k.w_bias && k.w_proj && k.w_out, "pair_block: null pointer (single track)");
    KFB_CHECK_ARG(is_dtype(s_dtype) && (s_dtype == KFB_FP32_PRECISE) == (precise != 0), "pair_block: dtypes %d and %d", z_dtype, s_dtype);
  }
  KFB_CHECK_ARG((reinterpret_cast<uintptr_t>(workspace) & 255) == 0, "pair_block: workspace must be 256-byte aligned");
  const size_t need = kfb_pair_block_workspace_bytes(blk, batch, n, precise);
  KFB_CHECK_ARG(workspace_bytes >= need, "pair_block: workspace %zu < %zu bytes", workspace_bytes, need);
  const size_t ob = operator_bytes(k, batch, n, precise);
  const long long pos = static_cast<long long>(batch) * n * n, rows = static_cast<long long>(batch) * n;
  // (inside the operators' scratch, behind what the triangle multiplication takes of it)
  void* fold_room = precise ? nullptr : static_cast<uint8_t*>(workspace) + kfb_trimul_workspace_bytes(batch, n, k.c);
  const void* cur = z;
  for (int dir = 0; dir < 2; ++dir) {
    const kfb_trimul_weights& w = dir ? k.mul_in : k.mul_out;
    KFB_TRY(trimul_run(as_stream(stream), dir, cur, pair_mask, w.ln_in_w, w.ln_in_b, w.w_in, w.w_gout, w.ln_out_w, w.ln_out_b, w.w_pout, z_out,
                       cur, workspace, ob, batch, n, k.c, k.eps, z_dtype, fold_room, dir));
    cur = z_out;
  }
  // the mask scans of both directions in one launch, after the operators' scratch
  int2* scans = nullptr;
  if (k.has_attention && triatt_scans_mask(k.c, k.tri_heads, n, z_dtype)) {
    scans = reinterpret_cast<int2*>(static_cast<uint8_t*>(workspace) + ob);
    KFB_TRY(triatt_mask_rows(as_stream(stream), pair_mask, scans, batch, n));
  }
  for (int dir = 0; k.has_attention && dir < 2; ++dir) {
    const kfb_triatt_weights& w = dir ? k.att_end : k.att_start;
    KFB_TRY(triatt_run(as_stream(stream), dir, cur, pair_mask, w.ln_w, w.ln_b, w.w_proj, w.w_out, z_out, cur, workspace, ob, batch, n, k.c,
                       k.tri_heads, k.eps, z_dtype, scans != nullptr ? scans + static_cast<long long>(dir) * batch * n : nullptr, 1));
  }
  KFB_TRY(transition_run(as_stream(stream), cur, k.trans_z.ln_w, k.trans_z.ln_b, k.trans_z.w_swiglu, k.trans_z.w_out, z_out, cur, workspace, ob,
                         pos, k.c, k.hidden_z, k.eps, z_dtype, 1));
  if (!k.has_single) return KFB_OK;
  // single track: its operands come after the operators' scratch
  uint8_t* extra = static_cast<uint8_t*>(workspace) + ob + mask_rows_bytes(k, batch, n);
  const int pitch = bias_pitch(n, precise);
  void* bias = extra;
  void* an = extra + align_up(static_cast<size_t>(batch) * k.heads * n * pitch * (precise ? 4 : 2), 256);
  if (precise)
    KFB_TRY(kfb_pair_bias_fwd(z_out, k.ln_z_w, k.ln_z_b, k.w_bias, bias, workspace, ob, batch, n, k.c, k.heads, 0, k.eps, z_dtype, stream));
  else
    KFB_TRY(pair_bias_run(z_out, k.ln_z_w, k.ln_z_b, k.w_bias, bias, workspace, batch, n, n, k.c, k.heads, 0, k.eps, z_dtype,
                          as_stream(stream), pitch));
  KFB_TRY(launch_layernorm(as_stream(stream), s, an, k.ln_s_w, k.ln_s_b, rows, k.c_s, k.c_s, k.c_s, k.eps, is_fp32_io(s_dtype) ? KFB_FP32 : KFB_BF16,
                           precise ? KFB_FP32 : KFB_BF16));
  ApbArgs r;
  r.x = an;
  r.w_static = 1;
  r.pair_bias = bias; r.ldb = pitch; r.bias_hs = static_cast<long long>(n) * pitch;
  r.mask = mask;
  r.w_proj = k.w_proj; r.proj_bias = k.proj_bias; r.w_out = k.w_out; r.out_bias = k.out_bias;
  r.out = s_out; r.resid = s;
  r.workspace = workspace; r.workspace_bytes = ob;
  r.batch = batch; r.l = n; r.c = k.c_s; r.heads = k.heads; r.out_dtype = s_dtype;
  KFB_TRY(apb_run(as_stream(stream), r));
  return transition_run(as_stream(stream), s_out, k.trans_s.ln_w, k.trans_s.ln_b, k.trans_s.w_swiglu, k.trans_s.w_out, s_out, s_out, workspace, ob,
                        rows, k.c_s, k.hidden_s, k.eps, s_dtype, 1);
}

}  // extern "C"
