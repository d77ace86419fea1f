// Small helpers shared by the operator entry points.
#pragma once
#include "common.cuh"
#include "gemm.cuh"
#include "layernorm.cuh"

namespace kfb {

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }
inline bool is_dtype(int d) { return d == KFB_BF16 || d == KFB_FP32 || d == KFB_FP32_PRECISE; }
inline bool is_fp32_io(int d) { return d == KFB_FP32 || d == KFB_FP32_PRECISE; }
inline size_t dtype_bytes(int d) { return d == KFB_BF16 ? 2 : 4; }

// Carves 256-byte aligned pieces out of a caller-provided workspace.
struct Carver {
  uint8_t* base;
  size_t off = 0;
  explicit Carver(void* p) : base(static_cast<uint8_t*>(p)) {}
  template <typename T>
  T* take(size_t count) {
    T* r = reinterpret_cast<T*>(base + off);
    off += align_up(count * sizeof(T), 256);
    return r;
  }
};

// Row-major output segment [rows][ld] starting at column 0.
inline EpiSeg row_major_seg(void* dst, int ncols, long long ld, long long s_o, long long s_b, int out_fp32, int col_begin = 0) {
  EpiSeg s = {};
  s.col_begin = col_begin;
  s.ncols = ncols;
  s.out_fp32 = out_fp32;
  s.dst = dst;
  s.s_col = 1;
  s.s_n = ld;
  s.s_o = s_o;
  s.s_b = s_b;
  const int v = out_fp32 ? 4 : 8;
  s.vec = (ld % v == 0) && (s_o % v == 0) && (s_b % v == 0) && ((reinterpret_cast<uintptr_t>(dst) & 15) == 0);
  return s;
}

// Pitch of rows of l positions that TMA maps read or the epilogues store channel-major: whole 32-byte sectors.
inline int pitch16(int l) { return (l + 15) / 16 * 16; }

// Gated pair-bias self-attention on normalised rows (kfb_apb_fwd and the stacks; see include/kfold_b200.h).
struct ApbArgs {
  const void* x = nullptr;            // bf16 (batch, l, c); precise: fp32, or its triple split when x_is_split
  int x_is_split = 0;
  int w_static = 0;                   // a launch of this library lies between the last write of the weights and this call
  const void* pair_bias = nullptr;    // [batch / bias_div][heads][l][ldb], head planes bias_hs elements apart (0: l * ldb)
  long long ldb = 0, bias_hs = 0;
  int bias_div = 1;
  const unsigned char* mask = nullptr;  // [batch / mask_share][l]
  int mask_share = 1;
  int2* rows = nullptr;               // launch_attention_mask_rows' result for the mask: the attention kernel for shared biases
  const void* w_proj = nullptr; const float* proj_bias = nullptr;
  const void* w_out = nullptr; const float* out_bias = nullptr;
  const void* out_gate = nullptr; int gate_share = 1; long long gate_ld = 0;
  void* out = nullptr; const void* resid = nullptr;
  void* workspace = nullptr; size_t workspace_bytes = 0;
  int batch = 0, l = 0, c = 0, heads = 0, out_dtype = 0;
};
int apb_run(cudaStream_t stream, const ApbArgs& r);

// kfb_triatt_fwd; mask_rows: what triatt_mask_rows wrote for this direction, or null (the operator scans the mask itself); w_static as in
// ApbArgs.
int triatt_run(cudaStream_t stream, int ending, const void* x, const unsigned char* mask, const float* ln_w, const float* ln_b,
               const void* w_proj_packed, const void* w_out, void* out, const void* resid, void* workspace, size_t workspace_bytes, int batch,
               int n, int c, int heads, float eps, int dtype, int2* mask_rows, int w_static);
// kfb_trimul_fwd; fold_room: trimul_fold_bytes(c) bytes (256-byte aligned) beside the workspace for the output projection's folded
// weights, which then cost no launch, or null.  (bf16 path; the fp32-accurate one folds nothing.)  w_static as in ApbArgs.
size_t trimul_fold_bytes(int c);
int trimul_run(cudaStream_t stream, int incoming, const void* x, const unsigned char* mask, const float* ln_in_w, const float* ln_in_b,
               const void* w_in_packed, const void* w_gout, const float* ln_out_w, const float* ln_out_b, const void* w_pout, void* out,
               const void* resid, void* workspace, size_t workspace_bytes, int batch, int n, int c, float eps, int dtype, void* fold_room,
               int w_static);
// kfb_transition_fwd; w_static as in ApbArgs.
int transition_run(cudaStream_t stream, const void* x, const float* ln_w, const float* ln_b, const void* w_swiglu_packed, const void* w_out,
                   void* out, const void* resid, void* workspace, size_t workspace_bytes, long long rows, int c, int hidden, float eps, int dtype,
                   int w_static);
// Whether these sizes take the attention kernel that scans the mask, and the scan for both directions in one launch: batch * n entries
// of the starting node, then those of the ending node.
bool triatt_scans_mask(int c, int heads, int n, int dtype);
int triatt_mask_rows(cudaStream_t stream, const unsigned char* mask, int2* rows, int batch, int n);

// bf16 pair bias (kfb_pair_bias_fwd) with bias rows `pitch` elements apart (0: n).
int pair_bias_run(const void* z, const float* ln_w, const float* ln_b, const void* w, void* bias_out, void* workspace, int batch,
                  int rows, int n, int c, int heads, int transposed, float eps, int dtype, cudaStream_t stream, int pitch);

// Conditioned transition on AdaLN-normalised rows (kfb_cond_transition_fwd and the stacks).  x_is_split: precise mode, x is
// already the triple split; w_static as in ApbArgs.
int cond_transition_run(cudaStream_t stream, const void* x_normed, int x_is_split, int w_static, const void* w_swiglu, const void* w_out,
                        const void* out_gate, long long gate_ld, void* out, const void* resid, void* workspace,
                        size_t workspace_bytes, long long rows, int c, int hidden, int samples, int l, int dtype);

}  // namespace kfb
