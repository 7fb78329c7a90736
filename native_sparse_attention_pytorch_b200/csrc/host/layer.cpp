// The whole layer natively: forward and backward of SparseAttention as one autograd node.
//
// Run module by module, a training step of the layer is nine autograd functions, some 140 launches and 3 ms of host
// time whatever the size; most of the launches are small conversions, additions and copies between layouts.  Here the
// layer is 35 to 50 launches: the GEMMs (library in the forward, which decides ReLU units and blocks; in the backward
// nsa_gemm.cu where it is faster), the attention kernels, and one pass for everything between two of them (nsa_layer.cu).

#include <ATen/Context.h>
#include <ATen/cuda/CUDAContext.h>
#include <cublas_v2.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>

#include <climits>
#include <cmath>
#include <limits>
#include <list>
#include <mutex>

#include "nsa_kernels.h"
#include "rooms.h"

namespace nsa_host {

// Sizes and options of a layer call, from Python as one list of integers
struct LayerConfig {
  int64_t heads, kv_heads, d, window, cbs, stride, block, nsel, num_mem, causal, shared, diff_topk;
};

static LayerConfig config_of(const std::vector<int64_t>& c) {
  return {c.at(0), c.at(1), c.at(2), c.at(3), c.at(4), c.at(5), c.at(6), c.at(7), c.at(8), c.at(9), c.at(10), c.at(11)};
}

// The parameters, in the order of the autograd function's arguments
struct LayerWeights {
  Tensor norm, qkv, gate, gate_b, out, mem, pos_k, pos_v, k1, kb1, k2, kb2, v1, vb1, v2, vb2;
};
static LayerWeights weights_of(const std::vector<OptTensor>& w) {
  auto t = [&](size_t i) { return w.at(i).value_or(Tensor()); };
  return {t(0), t(1), t(2), t(3), t(4), t(5), t(6), t(7), t(8), t(9), t(10), t(11), t(12), t(13), t(14), t(15)};
}
constexpr int kWeights = 16;

bool layer_takes(const Tensor& x, const std::vector<OptTensor>& w, int64_t heads, int64_t kv_heads, int64_t d, int64_t cbs, int64_t num_mem) {
  if (x.dim() != 3 || !x.has_storage() || reinterpret_cast<uintptr_t>(x.data_ptr()) % 16 || x.size(2) % 8) return false;
  const int64_t dim = x.size(2);
  if (w.at(0).has_value() && !fits(w[0], x, {dim})) return false;
  if (!fits(w.at(1), x, {(heads + 2 * kv_heads) * d, dim}) || !fits(w.at(2), x, {3 * heads, dim}) || !fits(w.at(3), x, {3 * heads}) ||
      !fits(w.at(4), x, {dim, heads * d}) || !fits(w.at(5), x, {2, kv_heads, num_mem, d}))
    return false;
  if (w.size() == 6) return true;
  if (!w.at(8).has_value() || w[8]->dim() != 2) return false;
  const int64_t hidden = w[8]->size(0);
  for (int s = 0; s < 2; ++s)
    if (!fits(w.at(6 + s), x, {kv_heads, cbs, d}) || !fits(w.at(8 + 4 * s), x, {hidden, cbs * d}) || !fits(w.at(9 + 4 * s), x, {hidden}) ||
        !fits(w.at(10 + 4 * s), x, {d, hidden}) || !fits(w.at(11 + 4 * s), x, {d}))
      return false;
  return hidden % 8 == 0;
}

// Row-major GEMMs, C [M, N] = (beta C +) op(A) op(B), on the library and with the settings at::mm uses, without the
// tensor views and the dispatch around them (8 us of host time per product; a training step has 17).
enum class Op { NT, NN, TN };   // A [M, K], B [N, K];  A [M, K], B [K, N];  A [K, M], B [K, N]
static void gemm(Op op, at::ScalarType type, int64_t M, int64_t N, int64_t K, const void* A, const void* B, void* C, float beta = 0.f) {
  const float alpha = 1.f;
  const cublasOperation_t ta = op == Op::NT ? CUBLAS_OP_T : CUBLAS_OP_N, tb = op == Op::TN ? CUBLAS_OP_T : CUBLAS_OP_N;
  const int lda = (int)(op == Op::NT ? K : N), ldb = (int)(op == Op::TN ? M : K);   // column-major: C^T = op(B)^T op(A)^T
  const cublasHandle_t handle = at::cuda::getCurrentCUDABlasHandle();
  const cublasStatus_t rc =
      type == at::kFloat
          ? cublasSgemm(handle, ta, tb, (int)N, (int)M, (int)K, &alpha, (const float*)B, lda, (const float*)A, ldb, &beta, (float*)C, (int)N)
          : cublasGemmEx(handle, ta, tb, (int)N, (int)M, (int)K, &alpha, B, CUDA_R_16BF, lda, A, CUDA_R_16BF, ldb, &beta, C, CUDA_R_16BF,
                         (int)N, CUBLAS_COMPUTE_32F, CUBLAS_GEMM_DEFAULT_TENSOR_OP);
  if (rc != CUBLAS_STATUS_SUCCESS) throw Error("layer: a library GEMM failed");
}
// The settings above are PyTorch's defaults; where a program changed them its products go through at::mm.
static bool default_blas(at::ScalarType type) {
  auto& ctx = at::globalContext();
  return ctx.blasPreferredBackend() == at::BlasBackend::Cublas &&
         (type == at::kFloat || ctx.allowBF16ReductionCuBLAS() == at::CuBLASReductionOption::AllowReducedPrecisionWithSplitK);
}
static Tensor product(Op op, const Tensor& A, const Tensor& B) {
  if (!default_blas(A.scalar_type())) return op == Op::NT ? at::mm(A, B.t()) : op == Op::NN ? at::mm(A, B) : at::mm(A.t(), B);
  const int64_t M = A.size(op == Op::TN ? 1 : 0), K = A.size(op == Op::TN ? 0 : 1), N = B.size(op == Op::NT ? 0 : 1);
  Tensor C = at::empty({M, N}, A.options());
  gemm(op, A.scalar_type(), M, N, K, A.data_ptr(), B.data_ptr(), C.data_ptr());
  return C;
}

// Products that do not depend on one another: in one launch of nsa_gemm.cu, or one library GEMM each.
//   fp32: in one launch, unless the program allows TF32 (which the library's kernels then use) or changed the settings above.
//   bf16: while the K steps of the tiles come to at most kStepsPerSM per SM.  Beyond that the library's larger tiles, which
//   read the operands a quarter as often, win on the GPU: the last products of a layer's backward, own kernel against library,
//   with 4 steps per SM (1024 rows, dim 256) 16 us against 21, with 7 (512 rows, dim 512) 23 against 17, with 29 (2048 rows)
//   47 against 24; on the host the launch is 4 us, a library product 12 to 17.
class Products {
 public:
  struct Product {
    Op op;
    Tensor A, B, C;         // matrices; C dense
    Tensor A2, B2;          // a second product that is added, or undefined
    Tensor act;             // own kernel only: zero where this is not positive,
    float* sums = nullptr;  // and the column sums of the result are added here
  };
  Products(at::ScalarType type, int32_t* status) : type_(type), status_(status) { items_.reserve(nsa::GemmGroup::kMost); }
  Product& add(Op op, const Tensor& A, const Tensor& B, const Tensor& C) {
    items_.push_back({op, A, B, C});
    return items_.back();
  }
  // False: by the library, which leaves `act` and `sums` to the caller
  bool run(cudaStream_t stream) const {
    nsa::GemmGroup g;
    const bool own = grouped(g);
    if (own) check(nsa::launch_gemm(g, code(), stream));
    else
      for (const Product& p : items_) library(p);
    return own;
  }
  // The products as one launch; false where the library serves better, or has to
  bool grouped(nsa::GemmGroup& g) const {
    g = {};
    g.status = status_;
    int64_t steps = 0, most = 0;
    for (const Product& p : items_) {
      nsa::GemmTask& t = g.task[g.tasks++];
      t.op = p.op == Op::NT ? nsa::kGemmNT : p.op == Op::NN ? nsa::kGemmNN : nsa::kGemmTN;
      t.m = (int)p.C.size(0); t.n = (int)p.C.size(1);
      int64_t deep = 0;
      auto part = [&](int i, const Tensor& A, const Tensor& B) {
        const int64_t K = depth(p, A);
        t.a[i] = A.data_ptr(); t.lda[i] = A.size(1);
        t.b[i] = B.data_ptr(); t.ldb[i] = B.size(1);
        t.k[i] = (int)K;
        deep += (K + 63) / 64;
        most = std::max({most, K, A.size(1), B.size(1)});
      };
      part(0, p.A, p.B);
      if (p.A2.defined()) part(1, p.A2, p.B2);
      t.act = ptr<void>(p.act); t.sums = p.sums; t.c = p.C.data_ptr();
      steps += (p.C.size(0) + 127) / 128 * ((p.C.size(1) + 63) / 64) * deep;
      most = std::max({most, p.C.size(0), p.C.size(1)});
    }
    if (most >= INT_MAX || !default_blas(type_) || !nsa::gemm_serves(g, code())) return false;
    return type_ == at::kFloat ? !at::globalContext().allowTF32CuBLAS() : steps <= 148 * kStepsPerSM;
  }

 private:
  static constexpr int64_t kStepsPerSM = 5;
  std::vector<Product> items_;
  at::ScalarType type_;
  int32_t* status_;

  int code() const { return type_ == at::kFloat ? NSA_F32 : NSA_BF16; }
  static int64_t depth(const Product& p, const Tensor& A) { return A.size(p.op == Op::TN ? 0 : 1); }
  void library(const Product& p) const {
    const Tensor a = p.op == Op::TN ? p.A.t() : p.A, b = p.op == Op::NT ? p.B.t() : p.B;
    Tensor c = p.C;
    auto issue = [&](const Tensor& A, const Tensor& B, float beta) {
      gemm(p.op, type_, c.size(0), c.size(1), depth(p, A), A.data_ptr(), B.data_ptr(), c.data_ptr(), beta);
    };
    if (default_blas(type_)) {
      issue(p.A, p.B, 0.f);
      if (p.A2.defined()) issue(p.A2, p.B2, 1.f);
    } else {
      at::mm_out(c, a, b);
      if (p.A2.defined()) c.addmm_(p.op == Op::TN ? p.A2.t() : p.A2, p.op == Op::NT ? p.B2.t() : p.B2);
    }
  }
};

// A [B, H, N, d] view without a tensor: pointer and strides in elements
static nsa_tensor heads_view(void* p, int64_t sb, int64_t sh, int64_t sn) { return {p, sb, sh, sn}; }

// One allocation cut into 256-byte aligned parts
class Slab {
 public:
  int64_t add(int64_t bytes) {
    const int64_t at = size_;
    size_ += (bytes + 255) / 256 * 256;
    return at;
  }
  void allocate(const Tensor& like) { buf_ = bytes(size_ > 0 ? size_ : 1, like); }
  uint8_t* at(int64_t off) const { return static_cast<uint8_t*>(buf_.data_ptr()) + off; }
  const Tensor& tensor() const { return buf_; }
  Tensor view(int64_t off, at::IntArrayRef sizes, at::ScalarType type) const {
    int64_t n = 1;
    for (const int64_t s : sizes) n *= s;
    const int64_t el = c10::elementSize(type);
    return buf_.narrow(0, off, n * el).view(type).view(sizes);
  }

 private:
  int64_t size_ = 0;
  Tensor buf_;
};

// What both directions know about a call
struct Layer {
  LayerConfig c;
  int64_t B, N, dim, G, ncb, F, el, k_sel, hs;
  int dt;
  at::ScalarType type;
  float scale;
  nsa::LayerShape shape;
  int32_t* status;

  Layer(const LayerConfig& cfg, const Tensor& x, int64_t status_word) : c(cfg) {
    B = x.size(0); N = x.size(1); dim = x.size(2);
    G = c.heads / c.kv_heads; ncb = N / c.stride; F = (c.heads + 2 * c.kv_heads) * c.d;
    el = x.element_size(); dt = dtype_code(x); type = x.scalar_type();
    hs = c.shared ? c.kv_heads : c.heads;
    k_sel = std::min(std::min(c.nsel, ncb), ncb / (c.block / c.stride));
    scale = (float)(1.0 / std::sqrt((double)c.d));
    shape = {(int)B, (int)N, (int)c.heads, (int)c.kv_heads, (int)c.d, (int)ncb, (int)c.cbs, (int)c.stride, (int)c.num_mem};
    status = reinterpret_cast<int32_t*>(status_word);
  }

  int64_t rows(int64_t heads) const { return B * heads * N; }
  // contiguous [B, H, N, d]
  nsa_tensor heads_of(void* p, int64_t H, int64_t n) const { return heads_view(p, H * n * c.d, n * c.d, c.d); }
  // the queries (part 0), keys (1) or values (2) inside the qkv projection's output
  nsa_tensor in_qkv(void* qkv, int part) const {
    const int64_t first = part == 0 ? 0 : part == 1 ? c.heads : c.heads + c.kv_heads;
    return heads_view(static_cast<uint8_t*>(qkv) + first * c.d * el, N * F, c.d, F);
  }
  float sentinel() const {   // (-finfo.max) // 10 in the tensor's type
    if (dt == NSA_F32) return std::floor(-std::numeric_limits<float>::max() / 10.f);
    return (float)c10::BFloat16((float)std::floor(-3.3895313892515355e38 / 10.0));
  }

  nsa_cmp_fwd_args cmp_args(void* qkv, void* ckv, void* out, float* lse) const {
    nsa_cmp_fwd_args a = {};
    const int64_t kv = c.num_mem + ncb;
    a.q = in_qkv(qkv, 0);
    a.ck = heads_of(ckv, c.kv_heads, kv);
    a.cv = heads_of(static_cast<uint8_t*>(ckv) + B * c.kv_heads * kv * c.d * el, c.kv_heads, kv);
    a.out = heads_of(out, c.heads, N);
    a.lse = lse;
    a.batch = B; a.q_heads = c.heads; a.kv_heads = c.kv_heads; a.sel_heads = k_sel > 0 ? hs : c.kv_heads;
    a.seq = N; a.dim_head = c.d; a.num_mem = c.num_mem; a.ncb = ncb; a.stride = c.stride; a.causal = c.causal; a.dtype = dt;
    a.scale = scale; a.sentinel = sentinel(); a.status = status;
    return a;
  }
  nsa_sel_fwd_args sel_args(void* qr, const nsa_tensor& kr, const nsa_tensor& v, void* out, float* lse, const int64_t* idx,
                            const uint8_t* mask) const {
    nsa_sel_fwd_args a = {};
    a.q = heads_of(qr, c.heads, N); a.k = kr; a.v = v; a.out = heads_of(out, c.heads, N);
    a.idx = idx; a.mask = mask; a.lse = lse;
    a.batch = B; a.q_heads = c.heads; a.kv_heads = c.kv_heads; a.sel_heads = k_sel > 0 ? hs : c.kv_heads;
    a.seq = N; a.dim_head = c.d; a.block = c.block; a.nsel = k_sel; a.dtype = dt; a.scale = scale; a.status = status;
    a.diag = k_sel > 0 ? (c.causal ? NSA_DIAG_CAUSAL : NSA_DIAG_NONE) : (c.causal ? NSA_DIAG_CAUSAL : NSA_DIAG_FULL);
    return a;
  }
  nsa_swa_fwd_args swa_args(void* qr, const nsa_tensor& kr, const nsa_tensor& v, void* out, float* lse) const {
    nsa_swa_fwd_args a = {};
    a.q = heads_of(qr, c.heads, N); a.k = kr; a.v = v; a.out = heads_of(out, c.heads, N);
    a.lse = lse;
    a.batch = B; a.q_heads = c.heads; a.kv_heads = c.kv_heads; a.seq = N; a.dim_head = c.d;
    a.window = c.window; a.causal = c.causal; a.dtype = dt; a.scale = scale; a.status = status;
    return a;
  }
  nsa::CombineParams combine_params(void* const (&outs)[3], const void* logits) const {
    nsa::CombineParams p = {};
    for (int s = 0; s < 3; ++s) {
      p.o[s] = outs[s];
      p.o_sb[s] = c.heads * N * c.d; p.o_sh[s] = N * c.d; p.o_sn[s] = c.d;
    }
    p.gates = logits; p.g_sb = N * 3 * c.heads; p.g_sh = 3; p.g_sn = 3 * c.heads;
    p.logits = 1;
    p.batch = B; p.q_heads = c.heads; p.seq = N; p.d = c.d;
    return p;
  }
};

// Scratch of one attention call
template <typename Args, typename Size>
static Tensor scratch(Args& a, Size size, int backward, const Tensor& like) {
  const int64_t need = size(&a, backward);
  if (need < 0) check(need);
  Tensor ws;
  if (need > 0) {
    ws = bytes(need, like);
    a.workspace = ws.data_ptr();
    a.workspace_bytes = need;
  }
  return ws;
}

// -> out; cache (rotated keys, values, ck, cv, window keys, window values) where asked for; what the backward needs where asked for
static std::vector<OptTensor> layer_forward(Tensor x, std::vector<OptTensor> weights, double eps, Tensor inv_freq,
                                            std::vector<int64_t> cfg, int64_t status, bool save, bool want_cache) {
  const c10::cuda::CUDAGuard guard(x.device());
  const LayerWeights w = weights_of(weights);
  x = x.contiguous();
  const Layer L(config_of(cfg), x, status);
  const LayerConfig& c = L.c;
  cudaStream_t st = (cudaStream_t)stream_of(x);
  const int64_t B = L.B, N = L.N, BN = B * N, d = c.d, el = L.el, hkv = c.kv_heads;
  const at::ScalarType type = L.type;

  // norm
  Tensor xn = x.view({BN, L.dim}), rstd;
  if (w.norm.defined()) {
    const Tensor x2 = xn;
    if (L.dim * el / 16 <= 256) {
      xn = at::empty({BN, L.dim}, x.options());
      rstd = empty({BN}, x, at::kFloat);
      nsa::NormParams p = {};
      p.x = x2.data_ptr(); p.weight = w.norm.data_ptr(); p.y = xn.data_ptr(); p.rstd = ptr<float>(rstd);
      p.rows = BN; p.x_stride = L.dim; p.dim = L.dim; p.eps = (float)eps;
      check(nsa::launch_rmsnorm(p, L.dt, false, st));
    } else {
      xn = at::rms_norm(x2, {L.dim}, w.norm, eps);
    }
  }
  // The products in front of the ReLU and the selection stay with the library, as in the layer run module by module: a value
  // that rounds the other way there switches a hidden unit or a block, and the two forms of the layer have to agree.  (The gate
  // projection and the second product of the value network decide neither; they are library calls as well, 12 to 17 us of host
  // time each.)
  const Tensor qkv = product(Op::NT, xn, w.qkv);
  const Tensor logits = at::addmm(w.gate_b, xn, w.gate.t());
  if (!save) xn = Tensor();   // here and below: what nobody needs any more makes room for the partial results

  // kept for the backward (or until the end of this call): rotated q, compressed keys and values, branch outputs, ...
  const int64_t q_bytes = L.rows(c.heads) * d * el, k_bytes = L.rows(hkv) * d * el, kv = c.num_mem + L.ncb;
  Slab keep;
  const int64_t at_qr = keep.add(q_bytes), at_kr = keep.add(k_bytes);
  const int64_t at_win = keep.add(2 * B * hkv * L.ncb * c.cbs * d * el);
  const int64_t at_ckv = keep.add(2 * B * hkv * kv * d * el);
  const int64_t at_o = keep.add((save ? 3 : 2) * q_bytes), at_lse = keep.add(3 * L.rows(c.heads) * 4);
  const int64_t picks = L.rows(L.hs) * L.k_sel;
  const int64_t at_idx = keep.add(picks * 8), at_mask = keep.add(picks);
  keep.allocate(x);
  // branch outputs: compressed, selected, sliding; without a backward the selected one is only needed where the merge does
  // not do the combine
  uint8_t* const o = keep.at(at_o);
  void* outs[3] = {o, save ? o + q_bytes : nullptr, o + (save ? 2 : 1) * q_bytes};
  void* const qr = keep.at(at_qr);
  float* const lse = reinterpret_cast<float*>(keep.at(at_lse));

  nsa::LayerPrep prep = {};
  prep.qkv = qkv.data_ptr(); prep.pos_k = w.pos_k.data_ptr(); prep.pos_v = w.pos_v.data_ptr(); prep.inv_freq = ptr<float>(inv_freq);
  prep.qr = qr;
  const int64_t win_half = B * hkv * L.ncb * c.cbs * d * el;
  prep.kw = keep.at(at_win); prep.vw = keep.at(at_win + win_half);
  nsa_tensor kr = L.heads_of(keep.at(at_kr), hkv, N), v = L.in_qkv(qkv.data_ptr(), 2);
  GrownPair cache;
  if (want_cache) {   // keys and values straight into buffers a following generation can append to
    cache = Rooms::instance().fresh(x, B, hkv, N, std::min<int64_t>(std::max<int64_t>(N / 8, 64), 1024), d);
    prep.kr = cache.k_buf; prep.v_out = cache.v_buf; prep.c_sb = cache.k.stride(0); prep.c_sh = cache.k.stride(1);
    kr = t4(cache.k);
    v = t4(cache.v);
  } else {
    prep.kr = kr.ptr; prep.c_sb = kr.stride_b; prep.c_sh = kr.stride_h;
  }
  check(nsa::launch_layer_prep(L.shape, prep, L.dt, st));

  // compress networks: Linear, ReLU, Linear over each window
  const int64_t wins = B * hkv * L.ncb, width = c.cbs * d;
  const Tensor kw = keep.view(at_win, {wins, width}, type), vw = keep.view(at_win + win_half, {wins, width}, type);
  Tensor hk = at::_addmm_activation(w.kb1, kw, w.k1.t()), hv = at::_addmm_activation(w.vb1, vw, w.v1.t());
  const Tensor ck = at::addmm(w.kb2, hk, w.k2.t()), cv = at::addmm(w.vb2, hv, w.v2.t());
  if (!save) hk = hv = Tensor();
  void* const ckv = keep.at(at_ckv);
  check(nsa::launch_join_mem(L.shape, w.mem.data_ptr(), ck.data_ptr(), cv.data_ptr(), ckv, L.dt, st));

  // compressed branch; its logits rank the blocks
  int64_t* const idx = reinterpret_cast<int64_t*>(keep.at(at_idx));
  uint8_t* const mask = keep.at(at_mask);
  Tensor importance;
  {
    nsa_cmp_fwd_args a = L.cmp_args(qkv.data_ptr(), ckv, outs[0], lse);
    const int64_t cpf = c.block / c.stride;
    bool pooled = false;
    if (L.k_sel > 0) {
      a.pool = cpf;
      pooled = c.causal && !c.diff_topk && L.hs == hkv && nsa_cmp_fwd_pools(&a);
      importance = pooled ? at::empty({B, L.hs, N, L.ncb / cpf}, x.options().dtype(at::kBFloat16))
                          : at::empty({B, L.hs, N, L.ncb}, x.options().dtype(at::kFloat));
      if (pooled) a.pooled = importance.data_ptr();
      else { a.importance = ptr<float>(importance); a.pool = 0; }
    }
    const Tensor ws = scratch(a, nsa_cmp_workspace_bytes, 0, x);
    check(nsa_cmp_fwd(&a, st));
    if (L.k_sel > 0) {
      nsa::SelectParams p = {};
      p.imp = pooled ? nullptr : ptr<float>(importance);
      p.pooled = pooled ? importance.data_ptr() : nullptr;
      p.causal_limit = pooled;
      p.idx = idx; p.mask = mask;
      p.rows = B * L.hs; p.seq = N; p.cpf = pooled ? 1 : cpf; p.ncb = pooled ? L.ncb / cpf : L.ncb; p.cols = p.ncb / p.cpf;
      p.k = L.k_sel; p.block = c.block; p.exclude_own = c.block != c.stride; p.round_bf16 = L.dt == NSA_BF16;
      p.neg_max = L.dt == NSA_BF16 ? -3.3895313892515355e38f : -std::numeric_limits<float>::max();
      check(nsa::launch_select(p, st));
    }
    if (!c.diff_topk) importance = Tensor();
  }
  // sliding branch
  {
    nsa_swa_fwd_args a = L.swa_args(qr, kr, v, outs[2], lse + 2 * L.rows(c.heads));
    const Tensor ws = scratch(a, nsa_swa_workspace_bytes, 0, x);
    check(nsa_swa_fwd(&a, st));
  }
  // selected branch and gated combine: one pass over the partial results where the kernels can (then the branch's own
  // output is stored for the backward only), else one after the other
  Tensor index;
  const Tensor merged = at::empty({BN, c.heads * d}, x.options());
  {
    nsa_sel_fwd_args a = L.sel_args(qr, kr, v, outs[1], lse + L.rows(c.heads), L.k_sel > 0 ? idx : nullptr, L.k_sel > 0 ? mask : nullptr);
    const Tensor ws = scratch(a, nsa_sel_workspace_bytes, 0, x);
    if (save && ws.defined()) {
      index = bytes(nsa_sel_index_bytes(&a), x);
      a.index_out = index.data_ptr();
      a.index_out_bytes = index.numel();
    }
    nsa::CombineParams p = L.combine_params(outs, logits.data_ptr());
    nsa::GatherTargets t = {};
    t.outs[0] = merged.data_ptr(); t.num_outs = 1; t.total_features = c.heads * d;
    nsa_sel_fwd_args fused = a;
    if (!save) fused.out = no_tensor();
    int rc = ws.defined() ? nsa::sm100_sel_fwd_combine(fused, p, t, st) : NSA_ERR_UNSUPPORTED;
    Tensor selected;
    if (rc == NSA_ERR_UNSUPPORTED) {
      if (!save) {
        selected = bytes(q_bytes, x);
        a.out.ptr = selected.data_ptr();
        p.o[1] = a.out.ptr;
      }
      check(nsa_sel_fwd(&a, st));
      rc = nsa::launch_combine_gather(p, t, L.dt, st);
    }
    check(rc);
  }
  // output projection
  const Tensor out = at::empty({B, N, L.dim}, x.options());
  {
    Products p(type, L.status);
    p.add(Op::NT, merged, w.out, out.view({BN, L.dim}));
    p.run(st);
  }

  auto opt = [](const Tensor& t) { return t.defined() ? OptTensor(t) : OptTensor(); };
  std::vector<OptTensor> result = {out};
  if (want_cache) {
    // the un-rotated rows of the window that is being filled (its overlap with the last complete one first, zero where
    // that lies before the sequence)
    const int64_t first = L.ncb * c.stride - (c.cbs - c.stride), len = N - first, pad = std::max<int64_t>(0, -first);
    GrownPair run = Rooms::instance().fresh(x, B, hkv, len, 4 * c.cbs, d);
    const Tensor all = qkv.view({B, N, c.heads + 2 * hkv, d}).permute({0, 2, 1, 3});
    for (int s = 0; s < 2; ++s) {
      const Tensor dst = s == 0 ? run.k : run.v;
      if (pad > 0) dst.narrow(2, 0, pad).zero_();
      dst.narrow(2, pad, len - pad).copy_(all.narrow(1, c.heads + s * hkv, hkv).narrow(2, std::max<int64_t>(0, first), len - pad));
    }
    result.insert(result.end(), {cache.k, cache.v, ck.view({B, hkv, L.ncb, d}), cv.view({B, hkv, L.ncb, d}), run.k, run.v});
  }
  if (save) {
    result.insert(result.end(), {x, xn, opt(rstd), qkv, logits, keep.tensor(), hk, hv, opt(index), merged,
                                 c.diff_topk ? opt(importance) : OptTensor()});
  }
  return result;
}

// -> gradients of x and of the parameters, in the order of the forward's arguments; `needs` says which are wanted.  With
// `keep_built` the indexes of the sliding and the compressed backward that had to be built here follow.
static std::vector<OptTensor> layer_backward(Tensor dout, std::vector<OptTensor> weights, std::vector<OptTensor> saved,
                                             double eps, Tensor inv_freq, std::vector<int64_t> cfg, int64_t status,
                                             std::vector<bool> needs, OptTensor swa_index, OptTensor cmp_index, bool keep_built) {
  const LayerWeights w = weights_of(weights);
  auto sv = [&](size_t i) { return saved.at(i).value_or(Tensor()); };
  const Tensor x = sv(0), xn = sv(1), rstd = sv(2), qkv = sv(3), logits = sv(4), kept = sv(5), hk = sv(6), hv = sv(7), index = sv(8),
               merged = sv(9), importance = sv(10);
  const c10::cuda::CUDAGuard guard(x.device());
  const Layer L(config_of(cfg), x, status);
  const LayerConfig& c = L.c;
  cudaStream_t st = (cudaStream_t)stream_of(x);
  const int64_t B = L.B, N = L.N, BN = B * N, d = c.d, el = L.el, hkv = c.kv_heads, H = c.heads;
  const at::ScalarType type = L.type;
  const int64_t q_elems = L.rows(H) * d, k_elems = L.rows(hkv) * d, q_bytes = q_elems * el, kv = c.num_mem + L.ncb;
  const int64_t c_elems = B * hkv * kv * d;
  // the forward's slab, cut as there
  Slab keep;
  const int64_t at_qr = keep.add(q_bytes), at_kr = keep.add(k_elems * el);
  const int64_t at_win = keep.add(2 * B * hkv * L.ncb * c.cbs * d * el);
  const int64_t at_ckv = keep.add(2 * c_elems * el);
  const int64_t at_o = keep.add(3 * q_bytes), at_lse = keep.add(3 * L.rows(H) * 4);
  const int64_t picks = L.rows(L.hs) * L.k_sel;
  const int64_t at_idx = keep.add(picks * 8), at_mask = keep.add(picks);
  uint8_t* const kp = static_cast<uint8_t*>(kept.data_ptr());
  float* const lse = reinterpret_cast<float*>(kp + at_lse);
  auto kept_view = [&](int64_t off, at::IntArrayRef sizes, at::ScalarType t) {
    int64_t n = 1;
    for (const int64_t s : sizes) n *= s;
    return kept.narrow(0, off, n * (int64_t)c10::elementSize(t)).view(t).view(sizes);
  };

  // fp32 accumulators, cleared together (beside the combine's backward): dk, dv; dck, dcv; (counters); then the small gradients that end up in the layer's type.  An
  // fp32 layer returns the small ones as they are: there they have memory of their own, a gradient that a program keeps
  // must not keep the scratch of dk and dv with it.
  const int64_t pos = hkv * c.cbs * d, mems = hkv * c.num_mem * d, hid = w.k1.size(0);
  auto even = [](int64_t n) { return (n + 7) / 8 * 8; };
  const int64_t s_norm = 0, s_gate = s_norm + even(L.dim), s_mem = s_gate + even(3 * H), s_pos = s_mem + even(2 * mems),
                s_b1 = s_pos + even(2 * pos), s_b2 = s_b1 + even(2 * hid), s_end = s_b2 + even(2 * d);
  const int64_t a_counters = 2 * k_elems + 2 * c_elems, a_small = even(a_counters + nsa::gate_sums_counters((int)(3 * H)));
  const bool apart = type == at::kFloat;
  Tensor acc = empty({apart ? a_small : a_small + s_end}, x, at::kFloat);
  Tensor rounded = apart ? empty({s_end}, x, at::kFloat) : Tensor();
  float* const dk = ptr<float>(acc);
  float* const dck = dk + 2 * k_elems;
  float* const small = apart ? ptr<float>(rounded) : dk + a_small;

  // output projection and gated combine
  dout = dout.reshape({BN, L.dim}).contiguous();
  // (what a later step does not need is given back as soon as it has been used: the partial results of the branches are
  // larger than all of it together)
  std::vector<OptTensor> g(1 + kWeights);
  Tensor d_merged = at::empty({BN, c.heads * d}, x.options());
  {
    Products p(type, L.status);
    p.add(Op::NN, dout, w.out, d_merged);
    if (needs[5]) {
      g[5] = at::empty({L.dim, c.heads * d}, x.options());
      p.add(Op::TN, dout, merged, *g[5]);
    }
    p.run(st);
  }
  Slab tmp;
  const int64_t t_delta = tmp.add(3 * L.rows(H) * 4), t_gates = tmp.add(nsa::gate_sums_partial((int)(3 * H)) * 4);
  tmp.allocate(x);
  Tensor d_outs[3], dqs[3];
  for (Tensor& t : d_outs) t = bytes(q_bytes, x);
  const Tensor d_logits = at::empty({BN, 3 * H}, x.options());
  {
    void* const outs[3] = {kp + at_o, kp + at_o + q_bytes, kp + at_o + 2 * q_bytes};
    nsa::CombineParams p = L.combine_params(outs, logits.data_ptr());
    p.dout = d_merged.data_ptr();
    for (int s = 0; s < 3; ++s) p.d_o[s] = d_outs[s].data_ptr();
    p.delta = reinterpret_cast<float*>(tmp.at(t_delta));
    p.d_logits = d_logits.data_ptr();
    p.clear[0] = dk; p.clear_pieces[0] = acc.numel() / 4;
    if (apart) { p.clear[1] = small; p.clear_pieces[1] = s_end / 4; }
    check(nsa::launch_combine(p, L.dt, true, st));
    d_merged = Tensor();
  }

  // the three branches
  nsa::QkvGrad qg = {};
  const nsa_tensor kr = L.heads_of(kp + at_kr, hkv, N), v = L.in_qkv(qkv.data_ptr(), 2);
  auto delta = [&](int s) { return reinterpret_cast<float*>(tmp.at(t_delta)) + s * L.rows(H); };
  auto d_o = [&](int s) { return L.heads_of(d_outs[s].data_ptr(), H, N); };
  // dq of branch s: rows in the layer's type where the kernels store them, else fp32; run(direct) issues the call
  auto with_dq = [&](int s, bool stores, bool need_f32, nsa_tensor& dq_out, float*& dq, auto run) {
    int rc = NSA_ERR_UNSUPPORTED;
    if (stores && !need_f32) {
      dqs[s] = bytes(q_bytes, x);
      dq_out = L.heads_of(dqs[s].data_ptr(), H, N);
      rc = run();
      if (rc == 0) qg.dq[s] = dqs[s].data_ptr();
    }
    if (rc == NSA_ERR_UNSUPPORTED) {
      dqs[s] = bytes(q_elems * 4, x);
      dq_out = no_tensor();
      dq = ptr<float>(dqs[s]);
      rc = run();
      if (rc == 0) qg.dq_f32[s] = dq;
    }
    check(rc);
    d_outs[s] = Tensor();
  };
  Tensor slots;
  {
    nsa_sel_bwd_args a = {};
    a.fwd = L.sel_args(kp + at_qr, kr, v, kp + at_o + q_bytes, lse + L.rows(H),
                       L.k_sel > 0 ? reinterpret_cast<int64_t*>(kp + at_idx) : nullptr, L.k_sel > 0 ? kp + at_mask : nullptr);
    const Tensor ws = scratch(a.fwd, nsa_sel_workspace_bytes, 1, x);
    a.dout = d_o(1); a.dk = dk; a.dv = dk + k_elems; a.accumulate_kv = 1; a.delta = delta(1);
    if (index.defined()) { a.index = index.data_ptr(); a.index_bytes = index.numel(); }
    if (c.diff_topk && L.k_sel > 0) {
      slots = at::zeros({B, L.hs, N, L.k_sel}, x.options().dtype(at::kFloat));
      a.slot_grads = ptr<float>(slots);
    }
    with_dq(1, nsa_sel_bwd_stores_dq(&a.fwd) == 1, false, a.dq_out, a.dq, [&] { return nsa_sel_bwd(&a, st); });
  }
  std::vector<OptTensor> built(2);
  {
    nsa_swa_bwd_args a = {};
    a.fwd = L.swa_args(kp + at_qr, kr, v, kp + at_o + 2 * q_bytes, lse + 2 * L.rows(H));
    const Tensor ws = scratch(a.fwd, nsa_swa_workspace_bytes, 1, x);
    a.dout = d_o(2); a.dk = dk; a.dv = dk + k_elems; a.accumulate_kv = 1; a.delta = delta(2);
    if (swa_index.has_value()) { a.index = swa_index->data_ptr(); a.index_bytes = swa_index->numel(); }
    with_dq(2, nsa_swa_bwd_stores_dq(&a.fwd) == 1, false, a.dq_out, a.dq, [&] { return nsa_swa_bwd(&a, st); });
    const int64_t n = !keep_built || swa_index.has_value() || !ws.defined() ? 0 : nsa_swa_index_bytes(&a.fwd);
    if (n > 0) built[0] = ws.narrow(0, 0, n).clone();
  }
  const bool through_topk = slots.defined();
  {
    nsa_cmp_bwd_args a = {};
    a.fwd = L.cmp_args(qkv.data_ptr(), kp + at_ckv, kp + at_o, lse);
    const Tensor ws = scratch(a.fwd, nsa_cmp_workspace_bytes, 1, x);
    a.dout = d_o(0); a.dck = dck; a.dcv = dck + c_elems; a.accumulate_kv = 1; a.delta = delta(0);
    if (cmp_index.has_value()) { a.index = cmp_index->data_ptr(); a.index_bytes = cmp_index->numel(); }
    with_dq(0, nsa_cmp_bwd_stores_dq(&a.fwd) == 1, through_topk, a.dq_out, a.dq, [&] { return nsa_cmp_bwd(&a, st); });
    const int64_t n = !keep_built || cmp_index.has_value() || !ws.defined() ? 0 : nsa_cmp_index_bytes(&a.fwd);
    if (n > 0) built[1] = ws.narrow(0, 0, n).clone();
  }
  if (through_topk) {
    const Tensor dlog = at::empty({B, L.hs, N, L.ncb}, importance.options());
    nsa::TopkGrad t = {};
    t.importance = ptr<float>(importance); t.idx = reinterpret_cast<const int64_t*>(kp + at_idx); t.dvals = ptr<float>(slots); t.dlog = ptr<float>(dlog);
    t.qkv = qkv.data_ptr(); t.ck = kp + at_ckv; t.dq = ptr<float>(dqs[0]); t.dck = dck;
    t.batch = B; t.seq = N; t.heads = H; t.kv_heads = hkv; t.sel_heads = L.hs; t.d = d; t.ncb = L.ncb; t.num_mem = c.num_mem;
    t.cpf = c.block / c.stride; t.k = L.k_sel; t.block = c.block; t.stride = c.stride; t.causal = c.causal;
    t.scale = L.scale / (float)(H / L.hs);
    check(nsa::launch_topk_grad(t, L.dt, st));
  }

  // compress networks
  const int64_t wins = B * hkv * L.ncb, width = c.cbs * d;
  const Tensor dc = at::empty({2, wins, d}, x.options());
  check(nsa::launch_split_mem(L.shape, dck, dc.data_ptr(), small + s_mem, small + s_b2, L.dt, st));
  const Tensor dck_rows = dc.select(0, 0), dcv_rows = dc.select(0, 1);
  Tensor dhk = at::empty({wins, hid}, x.options()), dhv = at::empty({wins, hid}, x.options());
  auto weight_grad = [&](Products& p, int i, const Tensor& dy, const Tensor& in) {   // of a weight [features of dy, features of in]
    if (!needs[i]) return;
    g[i] = at::empty({dy.size(1), in.size(1)}, x.options());
    p.add(Op::TN, dy, in, *g[i]);
  };
  {
    Products p(type, L.status);
    auto hidden_grad = [&](const Tensor& dy, const Tensor& weight, const Tensor& act, const Tensor& dh, float* sums) {
      auto& q = p.add(Op::NN, dy, weight, dh);
      q.act = act;
      q.sums = sums;
    };
    hidden_grad(dck_rows, w.k2, hk, dhk, small + s_b1);
    hidden_grad(dcv_rows, w.v2, hv, dhv, small + s_b1 + hid);
    weight_grad(p, 11, dck_rows, hk);
    weight_grad(p, 15, dcv_rows, hv);
    if (!p.run(st)) {
      nsa::ColumnSums r = {};
      r.x[0] = dhk.data_ptr(); r.x[1] = dhv.data_ptr(); r.act[0] = hk.data_ptr(); r.act[1] = hv.data_ptr();
      r.out[0] = small + s_b1; r.out[1] = small + s_b1 + hid;
      r.rows = wins; r.cols = hid; r.sets = 2;
      check(nsa::launch_relu_sums(r, L.dt, st));
    }
  }
  const Tensor kw = kept_view(at_win, {wins, width}, type), vw = kept_view(at_win + wins * width * el, {wins, width}, type);
  Tensor dkw = at::empty({wins, width}, x.options()), dvw = at::empty({wins, width}, x.options());
  {
    Products p(type, L.status);
    weight_grad(p, 9, dhk, kw);
    weight_grad(p, 13, dhv, vw);
    p.add(Op::NN, dhk, w.k1, dkw);
    p.add(Op::NN, dhv, w.v1, dvw);
    p.run(st);
  }
  dhk = dhv = Tensor();

  // qkv, gates, norm
  const Tensor d_qkv = at::empty({BN, L.F}, x.options());
  qg.dk = dk; qg.dv = dk + k_elems; qg.dkw = dkw.data_ptr(); qg.dvw = dvw.data_ptr(); qg.inv_freq = ptr<float>(inv_freq); qg.out = d_qkv.data_ptr();
  {
    nsa::GateSums sums = {};
    sums.x = d_logits.data_ptr(); sums.out = small + s_gate; sums.rows = BN; sums.cols = (int)(3 * H);
    sums.partial = reinterpret_cast<float*>(tmp.at(t_gates)); sums.arrived = reinterpret_cast<unsigned*>(dk + a_counters);
    check(nsa::launch_layer_tail(L.shape, qg, sums, small + s_pos, L.dt, st));
  }
  for (Tensor& t : dqs) t = Tensor();
  dkw = dvw = Tensor();
  Tensor dxn;
  {
    Products p(type, L.status);
    weight_grad(p, 2, d_qkv, xn);
    // (in bf16 the library splits this sum over the rows and adds its parts in bf16, and so do the modules: 1 x 515 rows, dim 256,
    // off by 0.9 % from fp32, this kernel's by 0.5)
    if (type == at::kFloat) weight_grad(p, 3, d_logits, xn);
    else if (needs[3]) g[3] = product(Op::TN, d_logits, xn);
    if (needs[0] || needs[1]) {
      dxn = at::empty({BN, L.dim}, x.options());
      auto& q = p.add(Op::NN, d_qkv, w.qkv, dxn);
      q.A2 = d_logits;
      q.B2 = w.gate;
    }
    p.run(st);
  }
  if (needs[0] || needs[1]) {
    if (w.norm.defined()) {
      const Tensor dx = at::empty({BN, L.dim}, x.options());
      nsa::NormParams p = {};
      p.x = x.data_ptr(); p.weight = w.norm.data_ptr(); p.rstd = ptr<float>(rstd); p.dy = dxn.data_ptr(); p.dx = dx.data_ptr();
      p.dweight = small + s_norm; p.rows = BN; p.x_stride = L.dim; p.dim = L.dim; p.eps = (float)eps; p.accumulate = 1;
      check(nsa::launch_rmsnorm(p, L.dt, true, st));
      dxn = dx;
    }
    if (needs[0]) g[0] = dxn.view(x.sizes());
  }
  // the small gradients in the layer's type
  if (!apart) {
    rounded = at::empty({s_end}, x.options());
    check(nsa::launch_round(small, rounded.data_ptr(), s_end, st));
  }
  auto give = [&](int i, int64_t off, const Tensor& like) {
    if (needs[i]) g[i] = rounded.narrow(0, off, like.numel()).view(like.sizes());
  };
  if (w.norm.defined()) give(1, s_norm, w.norm);
  give(4, s_gate, w.gate_b);
  give(6, s_mem, w.mem);
  give(7, s_pos, w.pos_k);
  give(8, s_pos + pos, w.pos_v);
  give(10, s_b1, w.kb1);
  give(14, s_b1 + hid, w.vb1);
  give(12, s_b2, w.kb2);
  give(16, s_b2 + d, w.vb2);
  g.push_back(built[0]);
  g.push_back(built[1]);
  return g;
}

// The index of the sliding and of the compressed backward depends on the sizes only: kept for the last few shapes, per
// stream (so that none is read by another stream than the one that built it).  Not while the stream is being captured:
// what a graph builds exists only once it is replayed, and what it was handed would have to live as long as the graph.  A
// captured step builds its indexes itself, in the graph's own memory.
class IndexCache {
 public:
  using Key = std::vector<int64_t>;
  static IndexCache& instance() {
    static IndexCache* cache = new IndexCache;   // never destroyed: tensors must not outlive the CUDA context's teardown order
    return *cache;
  }
  OptTensor find(const Key& key) {
    const std::lock_guard<std::mutex> lock(mutex_);
    for (const auto& e : entries_)
      if (e.first == key) return e.second;
    return {};
  }
  void keep(Key key, const Tensor& index) {
    const std::lock_guard<std::mutex> lock(mutex_);
    if (entries_.size() >= kMost) entries_.pop_front();
    entries_.emplace_back(std::move(key), index);
  }

 private:
  static constexpr size_t kMost = 16;
  std::mutex mutex_;
  std::list<std::pair<Key, Tensor>> entries_;
};

// The autograd node.  A Python function in its place cost 80 us per backward (the call from the engine's thread, saved
// tensors and gradients crossing the language border one by one).
struct NativeLayerBackward : torch::autograd::Node {
  std::vector<torch::autograd::SavedVariable> weights, saved;
  double eps = 0;
  Tensor inv_freq;
  std::vector<int64_t> cfg;
  int64_t status = 0;

  void release_variables() override {
    for (auto& v : weights) v.reset_data();
    for (auto& v : saved) v.reset_data();
  }

  torch::autograd::variable_list apply(torch::autograd::variable_list&& grads) override {
    torch::autograd::variable_list out(1 + kWeights);
    if (!grads[0].defined()) return out;
    try {
      const at::NoGradGuard no_grad;
      auto unpack = [&](std::vector<torch::autograd::SavedVariable>& vs) {
        std::vector<OptTensor> ts;
        ts.reserve(vs.size());
        for (auto& v : vs) {
          Tensor t = v.unpack(getptr());
          ts.emplace_back(t.defined() ? OptTensor(std::move(t)) : OptTensor());
        }
        return ts;
      };
      const std::vector<OptTensor> w = unpack(weights), sv = unpack(saved);
      std::vector<bool> needs(1 + kWeights);
      for (int i = 0; i < 1 + kWeights; ++i) needs[i] = task_should_compute_output(i);
      const Tensor& x = *sv.at(0);
      const LayerConfig c = config_of(cfg);
      const IndexCache::Key base = {x.get_device(), reinterpret_cast<int64_t>(stream_of(x)), x.size(0), c.heads, c.kv_heads, x.size(1), c.d,
                                    c.causal};
      IndexCache::Key swa = base, cmp = base;
      swa.insert(swa.end(), {0, c.window});
      cmp.insert(cmp.end(), {1, c.num_mem, c.stride});
      auto& cache = IndexCache::instance();
      cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
      if (cudaStreamIsCapturing((cudaStream_t)stream_of(x), &capture) != cudaSuccess) throw Error("layer: the state of the stream cannot be read");
      const bool eager = capture == cudaStreamCaptureStatusNone;
      std::vector<OptTensor> g = layer_backward(grads[0], w, sv, eps, inv_freq, cfg, status, std::move(needs), eager ? cache.find(swa) : OptTensor(),
                                                eager ? cache.find(cmp) : OptTensor(), eager);
      note_backward(x);
      for (int i = 0; i < 1 + kWeights; ++i)
        if (g[i].has_value()) out[i] = std::move(*g[i]);
      if (g[1 + kWeights].has_value()) cache.keep(std::move(swa), *g[1 + kWeights]);
      if (g[2 + kWeights].has_value()) cache.keep(std::move(cmp), *g[2 + kWeights]);
    } catch (const Error& e) {
      raise_python_error(e.what());
    }
    if (at::GradMode::is_enabled()) {   // create_graph: the gradients are there, their own gradients are not
      for (auto& t : out)
        if (t.defined()) t.set_requires_grad(true);
      torch::autograd::DelayedError fail("trying to differentiate twice the layer's native backward", (int64_t)out.size());
      return fail.apply(std::move(out));
    }
    return out;
  }
};

static Tensor layer_apply(Tensor x, std::vector<OptTensor> weights, double eps, Tensor inv_freq, std::vector<int64_t> cfg, int64_t status) {
  auto node = std::shared_ptr<NativeLayerBackward>(new NativeLayerBackward, torch::autograd::deleteNode);
  torch::autograd::edge_list edges = {torch::autograd::impl::gradient_edge(x)};
  node->weights.reserve(kWeights);
  for (const auto& w : weights) {
    edges.push_back(w.has_value() ? torch::autograd::impl::gradient_edge(*w) : torch::autograd::Edge());
    node->weights.emplace_back(w.value_or(Tensor()), false);
  }
  node->set_next_edges(std::move(edges));
  node->eps = eps;
  node->inv_freq = inv_freq;
  node->cfg = cfg;
  node->status = status;
  std::vector<OptTensor> r;
  {
    const at::NoGradGuard no_grad;
    r = layer_forward(x, std::move(weights), eps, inv_freq, std::move(cfg), status, true, false);
  }
  node->saved.reserve(r.size() - 1);
  for (size_t i = 1; i < r.size(); ++i) node->saved.emplace_back(i == 1 && r[i]->is_same(x) ? x : r[i].value_or(Tensor()), false);
  Tensor out = *r[0];
  torch::autograd::set_history(out, node);
  return out;
}

// One launch of the grouped products on dense matrices, for tests: (op, A, B, act, A2, B2) each -> C and, with
// act, the column sums of C; cols and split as in GemmGroup
static std::vector<Tensor> products_together(
    std::vector<std::tuple<int64_t, Tensor, Tensor, OptTensor, OptTensor, OptTensor>> tasks, int64_t status, int cols, int split) {
  std::vector<Tensor> result;
  if (tasks.empty() || tasks.size() > (size_t)nsa::GemmGroup::kMost) throw Error("products: one to four of them");
  const Tensor& like = std::get<1>(tasks[0]);
  require_cuda(like);
  const c10::cuda::CUDAGuard guard(like.device());
  Products p(like.scalar_type(), reinterpret_cast<int32_t*>(status));
  for (const auto& [op_code, A, B, act, A2, B2] : tasks) {
    const Op op = op_code == 0 ? Op::NT : op_code == 1 ? Op::NN : Op::TN;
    auto rows = [&](const Tensor& a) { return a.size(op == Op::TN ? 1 : 0); };
    auto cols = [&](const Tensor& b) { return b.size(op == Op::NT ? 0 : 1); };
    auto deep = [&](const Tensor& a, const Tensor& b) {
      return a.dim() == 2 && b.dim() == 2 && a.is_contiguous() && b.is_contiguous() && a.scalar_type() == like.scalar_type() &&
             b.scalar_type() == like.scalar_type() && a.device() == like.device() && b.device() == like.device() &&
             a.size(op == Op::TN ? 0 : 1) == b.size(op == Op::NT ? 1 : 0) && a.numel() < INT_MAX && b.numel() < INT_MAX;
    };
    if (!deep(A, B) || A2.has_value() != B2.has_value() || (A2.has_value() && (!deep(*A2, *B2) || rows(*A2) != rows(A) || cols(*B2) != cols(B))) ||
        (act.has_value() && !fits(act, like, {rows(A), cols(B)})))
      throw Error("products: matrices that do not go together");
    const Tensor C = at::empty({rows(A), cols(B)}, like.options()), sums = at::zeros({cols(B)}, like.options().dtype(at::kFloat));
    auto& q = p.add(op, A, B, C);
    q.act = act.value_or(Tensor());
    q.A2 = A2.value_or(Tensor()); q.B2 = B2.value_or(Tensor());
    if (act.has_value()) q.sums = ptr<float>(sums);
    result.insert(result.end(), {C, sums});
  }
  nsa::GemmGroup g;
  p.grouped(g);
  g.cols = cols;
  g.split = split;
  check(nsa::launch_gemm(g, dtype_code(like), (cudaStream_t)stream_of(like)));
  return result;
}

void bind_layer(pybind11::module_& m) {
  namespace py = pybind11;
  m.def("products_together", &products_together, py::call_guard<py::gil_scoped_release>());
  m.def("layer_takes", &layer_takes);
  m.def("layer_forward", &layer_forward, py::call_guard<py::gil_scoped_release>());
  m.def("layer_apply", &layer_apply, py::call_guard<py::gil_scoped_release>());
}

}  // namespace nsa_host
