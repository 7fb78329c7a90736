// Selected-block attention: the bodies of the two directions, and the autograd node around them.

#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_cpp_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>

#include <algorithm>
#include <cmath>
#include <numeric>

#include "nsa_host.h"
#include "nsa_kernels.h"

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
  // dk and dv side by side: one clearing, one conversion; in the tensor-core family both are part of other launches
  Tensor dkv = empty({2, k.size(0), k.size(1), k.size(2), k.size(3)}, k, at::kFloat);
  Tensor slots = want_slots ? at::zeros(idx.sizes(), q.options().dtype(at::kFloat)) : Tensor();
  a.dout = t4(dout);
  a.dk = ptr<float>(dkv);
  a.dv = a.dk + k.numel();
  a.accumulate_kv = 1;
  a.slot_grads = ptr<float>(slots);
  a.index = index.defined() ? index.data_ptr() : nullptr;
  a.index_bytes = index.defined() ? index.numel() : 0;
  a.delta = delta.has_value() ? ptr<float>(*delta) : nullptr;
  Tensor dq;
  if (q.scalar_type() == at::kBFloat16 && nsa_sel_bwd_stores_dq(&a.fwd) == 1) {
    dq = empty_in_order_of(q);
    a.dq_out = t4(dq);
    Tensor rounded = at::empty(dkv.sizes(), k.options());
    const int rc = nsa::sel_bwd_rounded(a, rounded.data_ptr(), (cudaStream_t)stream_of(q));
    if (rc != NSA_ERR_UNSUPPORTED) {
      check(rc);
      return {dq, rounded.select(0, 0), rounded.select(0, 1), want_slots ? OptTensor(slots) : OptTensor()};
    }
  }
  // the generic kernels, or tensors the tensor-core ones declined: fp32 dq
  if (cudaMemsetAsync(a.dk, 0, 2 * k.numel() * sizeof(float), (cudaStream_t)stream_of(k)) != cudaSuccess) throw Error("clearing dk and dv failed");
  Tensor dq32 = empty(q.sizes(), q, at::kFloat);
  a.dq_out = no_tensor();
  a.dq = ptr<float>(dq32);
  check(nsa_sel_bwd(&a, stream_of(q)));
  dq = dq32.to(q.scalar_type());
  dkv = dkv.to(k.scalar_type());
  return {dq, dkv.select(0, 0), dkv.select(0, 1), want_slots ? OptTensor(slots) : OptTensor()};
}

// The autograd node of native_sparse_attend: 137 -> 110 us for forward and backward of 1 x 1024 positions against the same
// calls behind a Python function.
struct NativeSelectedBackward : torch::autograd::Node {
  torch::autograd::SavedVariable q, k, v, idx, mask, out, lse;
  Tensor index;            // which queries attend which key block, as the forward built it; `grad_fn.index` in Python
  int64_t block = 0, diag = 0, impl = 0, status = 0;
  double scale = 0;
  std::optional<at::ScalarType> slot_type;

  void release_variables() override {
    for (auto* t : {&q, &k, &v, &idx, &mask, &out, &lse}) t->reset_data();
    index = Tensor();
  }

  // The row sums sum_d out * dout that the gated combine's backward attaches to the branch gradient it returns
  static OptTensor handed_over_delta(const Tensor& dout, const Tensor& lse) {
    if (dout.unsafeGetTensorImpl()->pyobj_slot()->load_pyobj() == nullptr) return {};   // never seen by Python
    const pybind11::gil_scoped_acquire gil;
    const pybind11::object t = pybind11::reinterpret_steal<pybind11::object>(THPVariable_Wrap(dout));
    const pybind11::object d = pybind11::getattr(t, "_nsa_delta", pybind11::none());
    if (d.is_none()) return {};
    Tensor delta = THPVariable_Unpack(d.ptr());
    if (delta.sizes() != lse.sizes() || delta.scalar_type() != at::kFloat || !delta.is_contiguous() || delta.device() != dout.device()) return {};
    return delta;
  }

  torch::autograd::variable_list apply(torch::autograd::variable_list&& grads) override {
    torch::autograd::variable_list g(4);
    if (!grads[0].defined()) return g;
    try {
      const at::NoGradGuard no_grad;
      auto opt = [&](const torch::autograd::SavedVariable& s) {
        Tensor t = s.unpack(getptr());
        return t.defined() ? OptTensor(std::move(t)) : OptTensor();
      };
      const Tensor l = lse.unpack(getptr());
      std::vector<OptTensor> r = sel_backward(q.unpack(getptr()), k.unpack(getptr()), v.unpack(getptr()), opt(idx), opt(mask), out.unpack(getptr()), l,
                                              grads[0], handed_over_delta(grads[0], l), index.defined() ? OptTensor(index) : OptTensor(), block,
                                              diag, impl, scale, status, slot_type.has_value());
      note_backward(l);
      for (int i = 0; i < 3; ++i) g[i] = std::move(*r[i]);
      if (r[3].has_value()) g[3] = r[3]->to(*slot_type);
    } catch (const Error& e) {
      raise_python_error(e.what());
    }
    if (at::GradMode::is_enabled()) {   // create_graph: the gradients are there, their own gradients are not
      for (auto& t : g)
        if (t.defined()) t.set_requires_grad(true);
      torch::autograd::DelayedError fail("trying to differentiate twice the native backward of selected-block attention", 4);
      return fail.apply(std::move(g));
    }
    return g;
  }
};

// -> out, lse
static std::vector<Tensor> sel_attend(Tensor q, Tensor k, Tensor v, OptTensor idx, OptTensor mask, OptTensor slot_scale, int64_t block,
                                      int64_t diag, int64_t impl, int64_t status, bool reuse_index) {
  const double scale = 1.0 / std::sqrt((double)q.size(3));
  const bool slots = slot_scale.has_value() && slot_scale->requires_grad();
  const bool direct = q.requires_grad() || k.requires_grad() || v.requires_grad();
  const bool wanted = at::GradMode::is_enabled() && (direct || slots);
  std::vector<OptTensor> r;
  {
    const at::NoGradGuard no_grad;
    r = sel_forward(q, k, v, std::move(idx), std::move(mask), block, diag, impl, scale, status, {}, wanted && direct && reuse_index);
  }
  Tensor out = *r[5], lse = *r[6];
  if (!wanted) return {out, lse};
  using torch::autograd::SavedVariable;
  auto node = std::shared_ptr<NativeSelectedBackward>(new NativeSelectedBackward, torch::autograd::deleteNode);
  torch::autograd::edge_list edges = {torch::autograd::impl::gradient_edge(q), torch::autograd::impl::gradient_edge(k),
                                      torch::autograd::impl::gradient_edge(v),
                                      slot_scale.has_value() ? torch::autograd::impl::gradient_edge(*slot_scale) : torch::autograd::Edge()};
  node->set_next_edges(std::move(edges));
  auto saved = [&](int i) { return r[i].value_or(Tensor()); };
  node->q = SavedVariable(saved(0), false); node->k = SavedVariable(saved(1), false); node->v = SavedVariable(saved(2), false);
  node->idx = SavedVariable(saved(3), false); node->mask = SavedVariable(saved(4), false); node->lse = SavedVariable(lse, false);
  node->index = saved(7);
  node->block = block; node->diag = diag; node->impl = impl; node->status = status; node->scale = scale;
  if (slot_scale.has_value()) node->slot_type = slot_scale->scalar_type();
  torch::autograd::set_history(out, node);
  node->out = SavedVariable(out, true);
  return {out, lse};
}

static PyObject* node_index(PyObject* self, void*) {
  const auto* node = dynamic_cast<NativeSelectedBackward*>(reinterpret_cast<torch::autograd::THPCppFunction*>(self)->cdata.get());
  if (node == nullptr || !node->index.defined()) Py_RETURN_NONE;
  return THPVariable_Wrap(node->index);
}

static void register_node() {
  namespace ta = torch::autograd;
  using namespace torch::autograd;   // the property table's names
  static PyTypeObject type;
  static PyGetSetDef properties[] = {THP_FUNCTION_DEFAULT_PROPERTIES,
                                     {(char*)"index", node_index, nullptr, nullptr, nullptr},
                                     {nullptr, nullptr, nullptr, nullptr, nullptr}};
  static PyMethodDef methods[] = {{"_register_hook_dict", ta::THPCppFunction_register_hook_dict, METH_O, nullptr},
                                  {"register_hook", ta::THPCppFunction_register_hook, METH_O, nullptr},
                                  {"register_prehook", ta::THPCppFunction_register_prehook, METH_O, nullptr},
                                  {"name", ta::THPCppFunction_name, METH_NOARGS, nullptr},
                                  {"_sequence_nr", ta::THPCppFunction_sequence_nr, METH_NOARGS, nullptr},
                                  {nullptr, nullptr, 0, nullptr}};
  ta::_initFunctionPyTypeObject(type, "NativeSelectedBackward", properties, methods);
  ta::registerCppFunction(typeid(NativeSelectedBackward), &type);
}

void bind_selected(pybind11::module_& m) {
  namespace py = pybind11;
  register_node();
  m.def("sel_attend", &sel_attend, py::call_guard<py::gil_scoped_release>());
  m.def("sel_forward", &sel_forward, py::call_guard<py::gil_scoped_release>());
  m.def("sel_backward", &sel_backward, py::call_guard<py::gil_scoped_release>());
}

}  // namespace nsa_host
