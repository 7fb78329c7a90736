// Internal interface between the C ABI layer and the kernel files.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "nsa_b200.h"

namespace nsa {

enum { BR_SEL = 0, BR_CMP = 1, BR_SWA = 2 };

// Every pointer (NULL included) on a 16-byte boundary, as the kernels' vector accesses need it
template <typename... P>
inline bool aligned16(const P*... p) { return ((reinterpret_cast<uintptr_t>(p) | ...) & 15u) == 0; }

// Parameters of the generic attention kernels (all three branches).
struct AttnParams {
  const void *q, *k, *v, *dout;
  void* out;
  int64_t q_sb, q_sh, q_sn;
  int64_t k_sb, k_sh, k_sn;
  int64_t v_sb, v_sh, v_sn;
  int64_t o_sb, o_sh, o_sn;
  int64_t do_sb, do_sh, do_sn;
  float* lse;
  float *dq, *dk, *dv;  // contiguous fp32; dk/dv have `key_rows` rows per head
  float* slot_grads;
  int batch, q_heads, kv_heads, groups, seq, d;
  int key_rows;  // rows of k/v per head (seq, or num_mem + ncb)
  float scale;
  // selected branch
  const int64_t* idx;
  const uint8_t* mask;
  int block, nsel, diag;
  // compressed branch
  int num_mem, ncb, stride, causal, imp_heads, round_bf16;
  float sentinel;
  float* importance;
  // sliding branch
  int window;
};

struct SelectParams {
  const float* imp;
  const void* pooled;      // bf16 [rows, seq, cols], instead of imp
  int causal_limit;        // columns at and past i / block are not read: probability 0
  int64_t* idx;
  float* vals;
  uint8_t* mask;           // optional: value above the threshold below which a slot is masked out
  int rows, seq, ncb, cpf, cols, k, block, exclude_own, input_is_prob, round_bf16;
  float neg_max;
};

struct CombineParams {
  const void *o[3], *gates, *dout;
  int64_t o_sb[3], o_sh[3], o_sn[3];
  int64_t g_sb, g_sh, g_sn;
  void* out;
  void* d_o[3];
  float* d_gates;
  float* delta;            // backward, optional: [3][batch * q_heads * seq] gate x d gate
  void* d_logits;          // backward, with `logits`: [batch, seq, 3 q_heads] in the tensors' type, instead of d_gates
  int logits;              // `gates` holds logits: the gate is their sigmoid, rounded as a tensor of it would be
  int batch, q_heads, seq, d;
  float* clear[2];         // backward, optional: fp32 buffers of `clear_pieces` sixteen-byte pieces to zero in the same launch
  int64_t clear_pieces[2];
};

constexpr int kMaxGather = NSA_MAX_GATHER;
struct GatherTargets {
  void* outs[kMaxGather];
  int num_outs, multicast;
  int64_t total_features, feature_offset;
};

struct WindowParams {
  const void *x, *pos, *dout;
  void *out, *dx;
  float* dpos;
  int64_t x_sb, x_sh, x_sn;
  int64_t dx_sb, dx_sh, dx_sn;   // strides of dx
  int batch, heads, seq, d, block, stride, ncb;
};

struct RotaryParams {
  const void* x;
  void* out;
  const float *cos, *sin;
  int64_t x_sb, x_sh, x_sn;
  int64_t o_sb, o_sh, o_sn;   // strides of out
  int batch, heads, seq, d, inverse;
};

struct NormParams {
  const void* x;      // [rows, dim] rows x_stride elements apart
  const void* weight; // [dim] in the dtype of x, or fp32 when weight_f32
  void* y;            // [rows, dim] contiguous (forward)
  float* rstd;        // [rows]: written by the forward, read by the backward
  const void* dy;     // [rows, dim] contiguous (backward)
  void* dx;           // [rows, dim] contiguous (backward)
  float* dweight;     // [dim] fp32 (backward)
  int64_t rows, x_stride;
  int dim, weight_f32;
  int accumulate;     // backward: dweight is added to as it is instead of zeroed first
  float eps;
};

// One decoding step (see nsa_decode.cu): the newest token's queries against the caches.
struct DecodeParams {
  const void *q, *qr;            // [B, Hq, d] contiguous: un-rotated / rotated queries of the token
  const void *keys, *vals;       // [B, Hkv, T, d]: rotated keys and values, the token included
  int64_t k_sb, k_sh, k_sn, v_sb, v_sh, v_sn;
  const void *ck, *cv;           // [B, Hkv, ncb, d]: compressed blocks, without memory slots
  int64_t ck_sb, ck_sh, ck_sn, cv_sb, cv_sh, cv_sn;
  const void *mem_k, *mem_v;     // [Hkv, num_mem, d] contiguous
  const void* gates;             // [B, Hq, 3] contiguous
  void* out;                     // [B, Hq * d]
  int batch, q_heads, kv_heads, d, T, ncb, num_mem, stride, block, nsel, window;
  float scale;
  // instead of q and qr: the token rows of the qkv projection [B, (Hq + 2 Hkv) d]; the key (rotated) and the value are
  // then appended at row `row` of the caches (which `keys` / `vals` look into) and, un-rotated, at row `run_row` of the
  // window that is being filled
  const void* qkv;
  const float* inv_freq;         // [d / 2]
  void *new_keys, *new_vals, *run_k, *run_v;
  int64_t c_sb, c_sh, r_sb, r_sh;
  int row, run_row;
  int chained;                   // the kernel launched before is the projection that writes qkv and gates (launch_project)
};

// Projection of up to 16 rows (see nsa_decode.cu): y = f(x) w^T (+ bias) (ReLU), f = RMS norm, addition of `add`, or
// nothing; for two independent sets at once where `sets` is 2 (keys and values).  Row t of x is at
// x + (t / heads) x_sb + (t % heads) x_sh, of y likewise; `add` has one row per head.  Behind the rows of the first set:
// gates = sigmoid(f(x) gate_w^T + gate_b).
struct ProjectParams {
  const void *x[2], *w[2], *bias[2], *add[2];   // w [features, dim], bias [features] or NULL, add [heads, dim] or NULL
  void* y[2];
  const void *norm_w, *gate_w, *gate_b;         // [dim] or NULL, [gates_n, dim], [gates_n]
  void* gates;                                  // [rows, gates_n]
  int64_t x_sb, x_sh, y_sb, y_sh;
  int rows, heads, sets, dim, features, gates_n, relu;
  int chained;                                  // 1: first, 2: last kernel of a step, see nsa_decode.cu; else 0
  float eps;
};

// The rows of a key and a value cache into larger ones: per head one contiguous run of `pieces` sixteen-byte pieces, the heads
// `src_step` / `dst_step` pieces apart
struct CacheCopy {
  const void* src[2];
  void* dst[2];
  int64_t src_step, dst_step, pieces;
  int heads;
};

// The passes of a layer step between its GEMMs and its attention kernels (see nsa_layer.cu)
struct LayerShape {
  int batch, seq, heads, kv_heads, d, ncb, cbs, stride, num_mem;
};
struct LayerPrep {
  const void *qkv, *pos_k, *pos_v;   // [B, N, (Hq + 2 Hkv) d], [Hkv, cbs, d] twice
  const float* inv_freq;             // [d / 2]
  void *qr, *kr, *v_out;             // [B, Hq, N, d]; [B, Hkv, N, d] with the strides below (v_out may be NULL)
  int64_t c_sb, c_sh;
  void *kw, *vw;                     // [B, Hkv, ncb, cbs, d]
};
struct ColumnSums {
  void* x[2];                        // [rows, cols], masked in place
  const void* act[2];
  float* out[2];                     // added to
  int64_t rows;
  int cols, sets;                    // cols a multiple of 16 bytes
};
struct QkvGrad {
  const void* dq[3];                 // compressed, selected, sliding: [B, Hq, N, d] in the layer's type ...
  const float* dq_f32[3];            // ... or fp32
  const float *dk, *dv;              // [B, Hkv, N, d]
  const void *dkw, *dvw;             // [B, Hkv, ncb, cbs, d] or NULL
  const float* inv_freq;
  void* out;                         // [B, N, (Hq + 2 Hkv) d]
};

// Column sums of the gates' gradient (see nsa_layer.cu)
struct GateSums {
  const void* x;                     // [rows, cols]
  float* out;
  int64_t rows;
  int cols;
  float* partial;                    // gate_sums_partial(cols) floats
  unsigned* arrived;                 // gate_sums_counters(cols), zero
};

// Gradient through the differentiable top-k (see nsa_topk_grad.cu)
struct TopkGrad {
  const float* importance;           // [B, Hs, N, ncb], as the forward left it
  const int64_t* idx;                // [B, Hs, N, k]
  const float* dvals;                // [B, Hs, N, k]
  float* dlog;                       // [B, Hs, N, ncb], scratch
  const void *qkv, *ck;              // [B, N, (Hq + 2 Hkv) d]; [B, Hkv, num_mem + ncb, d]
  float *dq, *dck;                   // [B, Hq, N, d], [B, Hkv, num_mem + ncb, d]: added to
  int batch, seq, heads, kv_heads, sel_heads, d, ncb, num_mem, cpf, k, block, stride, causal;
  float scale;                       // of the logits, over the heads that share a selection
};

// Matrix products that share a launch: C [m, n] = the sum over the two parts of op(A) op(B), row-major, dense rows of C.
// NT: A [m, k], B [n, k];  NN: A [m, k], B [k, n];  TN: A [k, m], B [k, n].  Behind the sum: zero where act [m, n] is not
// positive; the column sums of what is stored are added to `sums`.
enum { kGemmNT = 0, kGemmNN = 1, kGemmTN = 2 };
struct GemmTask {
  const void *a[2], *b[2];
  int64_t lda[2], ldb[2];
  int k[2];                          // k[1] = 0: one part
  const void* act;
  float* sums;
  void* c;
  int m, n, op;
  int first_cta, split, c_vec;       // filled in by launch_gemm
};
struct GemmGroup {
  static constexpr int kMost = 4;
  GemmTask task[kMost];
  int* status;
  int tasks;
  int cols, split;                   // 0, or the columns of a tile (fp32: 64, 128) and the CTAs that share one (1, 2, 4, 8)
};

int fail(int code, const char* msg);

// Every host function that launches kernels of this library reports how many it launched; nsa_launch_count() returns
// the running total (a benchmark reads it before and after its timed region).
void count_launches(int n);

int simt_attend(const AttnParams& P, int branch, int dtype, bool backward, cudaStream_t stream);
int launch_select(const SelectParams& P, cudaStream_t stream);
int launch_combine(const CombineParams& P, int dtype, bool backward, cudaStream_t stream);
int launch_rotary(const RotaryParams& P, int dtype, cudaStream_t stream);
int launch_windows(const WindowParams& P, int dtype, bool backward, cudaStream_t stream);
int launch_rmsnorm(const NormParams& P, int dtype, bool backward, cudaStream_t stream);
int launch_combine_gather(const CombineParams& P, const GatherTargets& Gt, int dtype, cudaStream_t stream);
int launch_layer_prep(const LayerShape& L, const LayerPrep& P, int dtype, cudaStream_t stream);
int launch_join_mem(const LayerShape& L, const void* mem, const void* ck, const void* cv, void* out, int dtype, cudaStream_t stream);
int launch_split_mem(const LayerShape& L, const float* grad, void* dc, float* dmem, float* dbias, int dtype, cudaStream_t stream);
int launch_relu_sums(const ColumnSums& P, int dtype, cudaStream_t stream);
int64_t gate_sums_partial(int cols);    // floats
int gate_sums_counters(int cols);       // zero before the call
int launch_layer_tail(const LayerShape& L, const QkvGrad& P, const GateSums& S, float* dpos, int dtype, cudaStream_t stream);
// fp32: sums of up to 35840 products (70 steps of 64 on each of 8 CTAs), of up to 4480 in a task with column sums (one CTA); a task
// beyond that is not served, nor is any other of its group
bool gemm_serves(const GemmGroup& G, int dtype);
int launch_gemm(GemmGroup& G, int dtype, cudaStream_t stream);
int launch_topk_grad(const TopkGrad& P, int dtype, cudaStream_t stream);
int launch_round(const float* src, void* dst, int64_t n, cudaStream_t stream);
int launch_decode(const DecodeParams& P, int dtype, cudaStream_t stream);
int fill_decode(DecodeParams& P, const nsa_decode_args& a);   // checks the arguments; q and qr may be NULL
int launch_cache_copy(const CacheCopy& P, cudaStream_t stream);
bool project_serves(int batch, int dim, int dtype);
int launch_project(const ProjectParams& P, int dtype, cudaStream_t stream);

// Tensor-core family for the selected-block branch.  Each returns
// NSA_ERR_UNSUPPORTED (without touching the error message state of a later
// successful call) when the shape is outside what it serves.
int64_t sm100_sel_workspace_bytes(const nsa_sel_fwd_args& a, bool backward);
int64_t sm100_sel_index_bytes(const nsa_sel_fwd_args& a);
int64_t sm100_swa_index_bytes(const nsa_swa_fwd_args& a);
int64_t sm100_cmp_index_bytes(const nsa_cmp_fwd_args& a);
int sm100_sel_fwd(const nsa_sel_fwd_args& a, cudaStream_t stream);
// with dkv_out: dk and dv lie one behind the other, are cleared first and rounded into it (bf16) at the end
int sm100_sel_bwd(const nsa_sel_bwd_args& a, void* dkv_out, cudaStream_t stream);
// nsa_sel_bwd of the tensor-core family with dq_out and, in place of cleared dk and dv, dkv_out
int sel_bwd_rounded(const nsa_sel_bwd_args& a, void* dkv_out, cudaStream_t stream);
int sm100_sel_fwd_static(const nsa_sel_fwd_args& a, cudaStream_t stream);
int64_t sm100_swa_workspace_bytes(const nsa_swa_fwd_args& a, bool backward);
int sm100_swa_fwd(const nsa_swa_fwd_args& a, cudaStream_t stream);
int sm100_swa_bwd(const nsa_swa_bwd_args& a, cudaStream_t stream);
int64_t sm100_cmp_workspace_bytes(const nsa_cmp_fwd_args& a, bool backward);
int sm100_cmp_fwd(const nsa_cmp_fwd_args& a, cudaStream_t stream);
bool sm100_cmp_fwd_pools(const nsa_cmp_fwd_args& a);
int sm100_sel_fwd_combine(const nsa_sel_fwd_args& a, const CombineParams& c, const GatherTargets& t, cudaStream_t stream);
int sm100_cmp_bwd(const nsa_cmp_bwd_args& a, cudaStream_t stream);
int64_t sm100_static_scratch_bytes();
int sm100_sel_static_status(int* out, cudaStream_t stream);
int sm100_wait_selftest(int* status_device, int64_t limit_cycles, cudaStream_t stream);
bool sm100_sel_bwd_overwrites_dq(const nsa_sel_fwd_args& a);
bool sm100_swa_bwd_overwrites_dq(const nsa_swa_fwd_args& a);
bool sm100_cmp_bwd_overwrites_dq(const nsa_cmp_fwd_args& a);

}  // namespace nsa
