// Selected-block attention: the bodies of the autograd function's two directions.

#include <algorithm>
#include <numeric>

#include "nsa_host.h"

namespace nsa_host {

Tensor empty_in_order_of(const Tensor& t) {
  const int64_t nd = t.dim();
  std::vector<int64_t> order(nd), sizes(nd), back(nd);
  std::iota(order.begin(), order.end(), 0);
  std::stable_sort(order.begin(), order.end() - 1, [&](int64_t a, int64_t b) { return t.stride(a) > t.stride(b); });
  for (int64_t i = 0; i < nd; ++i) {
    sizes[i] = t.size(order[i]);
    back[order[i]] = i;
  }
  return at::empty(sizes, t.options()).permute(back);
}

static nsa_sel_fwd_args sel_args(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& out, const Tensor& idx,
                                 const Tensor& mask, const Tensor& lse, int64_t block, int64_t diag, int64_t impl,
                                 double scale, int64_t status) {
  nsa_sel_fwd_args a = {};
  a.q = t4(q); a.k = t4(k); a.v = t4(v); a.out = t4(out);
  a.idx = ptr<int64_t>(idx); a.mask = ptr<uint8_t>(mask); a.lse = ptr<float>(lse);
  a.batch = q.size(0); a.q_heads = q.size(1); a.kv_heads = k.size(1); a.sel_heads = idx.defined() ? idx.size(1) : k.size(1);
  a.seq = q.size(2); a.dim_head = q.size(3);
  a.block = block; a.nsel = idx.defined() ? idx.size(3) : 0; a.diag = diag; a.dtype = dtype_code(q); a.impl = impl;
  a.scale = scale;
  a.status = reinterpret_cast<int32_t*>(status);
  return a;
}

// -> q, k, v, idx, mask as the kernels read them (what the backward needs), out, lse, the index (where the tensor-core
// kernels built or were given one and `keep_index` asks for it)
static std::vector<OptTensor> sel_forward(Tensor q, Tensor k, Tensor v, OptTensor idx_, OptTensor mask_, int64_t block,
                                          int64_t diag, int64_t impl, double scale, int64_t status, OptTensor index_,
                                          bool keep_index) {
  Tensor idx = idx_.value_or(Tensor()), mask = mask_.value_or(Tensor()), index = index_.value_or(Tensor());
  for (const Tensor* t : {&q, &k, &v, &idx, &mask}) require_cuda(*t);
  const c10::cuda::CUDAGuard guard(q.device());
  q = rowwise(q); k = rowwise(k); v = rowwise(v);
  if (idx.defined()) {
    idx = idx.to(at::kLong).contiguous();
    mask = mask.to(at::kBool).contiguous().view(at::kByte);
  }
  Tensor out = at::empty(q.sizes(), q.options());
  Tensor lse = empty({q.size(0), q.size(1), q.size(2)}, q, at::kFloat);
  nsa_sel_fwd_args a = sel_args(q, k, v, out, idx, mask, lse, block, diag, impl, scale, status);
  Tensor ws;
  const int64_t need = nsa_sel_workspace_bytes(&a, 0);
  if (need < 0) check(need);
  if (need > 0) {
    ws = bytes(need, q);
    a.workspace = ws.data_ptr();
    a.workspace_bytes = need;
    if (index.defined()) {
      a.index = index.data_ptr();
      a.index_bytes = index.numel();
    } else if (keep_index) {   // in a buffer of its own, so that keeping it does not keep the partial results
      index = bytes(nsa_sel_index_bytes(&a), q);
      a.index_out = index.data_ptr();
      a.index_out_bytes = index.numel();
    }
  }
  check(nsa_sel_fwd(&a, stream_of(q)));
  if (need <= 0) index = Tensor();
  auto opt = [](const Tensor& t) { return t.defined() ? OptTensor(t) : OptTensor(); };
  return {q, k, v, opt(idx), opt(mask), out, lse, opt(index)};
}

// -> dq, dk, dv, slot gradients
static std::vector<OptTensor> sel_backward(Tensor q, Tensor k, Tensor v, OptTensor idx_, OptTensor mask_, Tensor out,
                                           Tensor lse, Tensor dout, OptTensor delta, OptTensor index_, int64_t block,
                                           int64_t diag, int64_t impl, double scale, int64_t status, bool want_slots) {
  Tensor idx = idx_.value_or(Tensor()), mask = mask_.value_or(Tensor()), index = index_.value_or(Tensor());
  const c10::cuda::CUDAGuard guard(q.device());
  dout = rowwise(dout);
  nsa_sel_bwd_args a = {};
  a.fwd = sel_args(q, k, v, out, idx, mask, lse, block, diag, impl, scale, status);
  Tensor ws;
  const int64_t need = nsa_sel_workspace_bytes(&a.fwd, 1);
  if (need < 0) check(need);
  if (need > 0) {
    ws = bytes(need, q);
    a.fwd.workspace = ws.data_ptr();
    a.fwd.workspace_bytes = need;
  }
  // dk and dv side by side: one clearing, one conversion
  Tensor dkv = empty({2, k.size(0), k.size(1), k.size(2), k.size(3)}, k, at::kFloat);
  Tensor slots = want_slots ? at::zeros(idx.sizes(), q.options().dtype(at::kFloat)) : Tensor();
  a.dout = t4(dout);
  a.dk = ptr<float>(dkv);
  a.dv = a.dk + k.numel();
  a.accumulate_kv = 1;
  if (cudaMemsetAsync(a.dk, 0, 2 * k.numel() * sizeof(float), (cudaStream_t)stream_of(k)) != cudaSuccess) throw Error("clearing dk and dv failed");
  a.slot_grads = ptr<float>(slots);
  a.index = index.defined() ? index.data_ptr() : nullptr;
  a.index_bytes = index.defined() ? index.numel() : 0;
  a.delta = delta.has_value() ? ptr<float>(*delta) : nullptr;
  Tensor dq;
  int rc = NSA_ERR_UNSUPPORTED;
  if (q.scalar_type() == at::kBFloat16 && nsa_sel_bwd_stores_dq(&a.fwd) == 1) {
    dq = empty_in_order_of(q);
    a.dq_out = t4(dq);
    rc = nsa_sel_bwd(&a, stream_of(q));
  }
  if (rc == NSA_ERR_UNSUPPORTED) {   // no direct dq, or the tensor-core kernels declined these tensors: fp32 dq
    Tensor dq32 = empty(q.sizes(), q, at::kFloat);
    a.dq_out = no_tensor();
    a.dq = ptr<float>(dq32);
    rc = nsa_sel_bwd(&a, stream_of(q));
    if (rc == 0) dq = dq32.to(q.scalar_type());
  }
  check(rc);
  dkv = dkv.to(k.scalar_type());
  return {dq, dkv.select(0, 0), dkv.select(0, 1), want_slots ? OptTensor(slots) : OptTensor()};
}

void bind_selected(pybind11::module_& m) {
  namespace py = pybind11;
  m.def("sel_forward", &sel_forward, py::call_guard<py::gil_scoped_release>());
  m.def("sel_backward", &sel_backward, py::call_guard<py::gil_scoped_release>());
}

}  // namespace nsa_host
