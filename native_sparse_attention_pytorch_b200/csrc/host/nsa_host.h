// Shared pieces of the native host side: what stands between PyTorch tensors and the C ABI of libnsa_b200.so.
//
// The Python operators issue one call of this extension per direction.  Filling the argument structs, sizing and
// allocating the buffers and issuing the launches from Python cost 100 to 150 us per operator and direction (ctypes
// structs, stream look-ups, allocator calls through the dispatcher), several times what the GPU needs at ordinary
// sizes; here it is a few microseconds plus the launches.
#pragma once

#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/utils/pybind.h>

#include <optional>
#include <stdexcept>
#include <string>
#include <vector>

#include "nsa_b200.h"

namespace nsa_host {

using at::Tensor;
using OptTensor = std::optional<Tensor>;

// An NSA_ERR_* or CUDA error code with its message; reaches Python as the package's NsaError.
struct Error : std::runtime_error {
  explicit Error(const std::string& what) : std::runtime_error(what) {}
};

[[noreturn]] void raise_python_error(const char* what);   // as the package's NsaError, from a thread of the autograd engine

inline void check(int64_t rc) {
  if (rc != 0) throw Error("libnsa_b200 returned " + std::to_string(rc) + ": " + nsa_last_error());
}

inline void require_cuda(const Tensor& t) {
  if (t.defined() && !t.is_cuda())
    throw Error("the NSA kernels run on CUDA tensors only; there is no CPU implementation in this package");
}

inline int dtype_code(const Tensor& t) {
  if (t.scalar_type() == at::kFloat) return NSA_F32;
  if (t.scalar_type() == at::kBFloat16) return NSA_BF16;
  throw Error(std::string("unsupported dtype ") + c10::toString(t.scalar_type()) + ": the kernels take float32 or bfloat16");
}

// t itself if its last axis is contiguous and its rows are 16-byte aligned, else a contiguous copy
inline Tensor rowwise(const Tensor& t) {
  const int64_t per16 = 16 / t.element_size();
  const auto st = t.strides();
  bool ok = st.back() == 1 && reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0;
  for (size_t i = 0; ok && i + 1 < st.size(); ++i) ok = st[i] % per16 == 0;
  return ok ? t : t.contiguous();
}

// A parameter the kernels can read as it is next to activations x: of these sizes, of x's type and device, dense, and on the
// 16-byte boundary their loads need (a view into a flat buffer of many parameters often is not)
inline bool fits(const OptTensor& t, const Tensor& x, at::IntArrayRef sizes) {
  return t.has_value() && t->defined() && t->has_storage() && t->scalar_type() == x.scalar_type() && t->device() == x.device() &&
         t->sizes() == sizes && t->is_contiguous() && reinterpret_cast<uintptr_t>(t->data_ptr()) % 16 == 0;
}

// Can the native layer calls take this input and these parameters (all, or the first six for a decoding step)?
bool layer_takes(const Tensor& x, const std::vector<OptTensor>& w, int64_t heads, int64_t kv_heads, int64_t d, int64_t cbs, int64_t num_mem);

inline nsa_tensor t4(const Tensor& t) { return {t.data_ptr(), t.stride(0), t.stride(1), t.stride(2)}; }
inline nsa_tensor no_tensor() { return {nullptr, 0, 0, 0}; }

template <typename T>
T* ptr(const Tensor& t) { return t.defined() ? static_cast<T*>(t.data_ptr()) : nullptr; }

inline Tensor empty(at::IntArrayRef sizes, const Tensor& like, at::ScalarType type) {
  return at::empty(sizes, like.options().dtype(type));
}
inline Tensor bytes(int64_t n, const Tensor& like) { return at::empty({n}, like.options().dtype(at::kByte)); }

inline void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

// Uninitialised tensor of t's shape and dtype whose dimensions lie in memory in the order t's do: a [b, h, n, d] view
// of a [b, n, (h d)] projection output gives a [b, n, h, d] buffer seen as [b, h, n, d], so that the gradient of the
// view that made t is a view again instead of a copy.
Tensor empty_in_order_of(const Tensor& t);

// A native backward has launched kernels that report through the device's status word: the next poll has to copy it (the
// operators' Python side notes its own calls)
void note_backward(const Tensor& t);

void bind_status(pybind11::module_& m);
void bind_selected(pybind11::module_& m);
void bind_decode(pybind11::module_& m);
void bind_layer(pybind11::module_& m);

}  // namespace nsa_host
