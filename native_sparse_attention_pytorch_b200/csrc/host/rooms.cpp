#include "rooms.h"

#include "nsa_kernels.h"

#include <ATen/core/LegacyTypeDispatch.h>

#include <array>

namespace nsa_host {

Rooms& Rooms::instance() {
  static Rooms* r = new Rooms;   // outlives the interpreter's tensors
  return *r;
}

// (what as_strided makes of it below autograd, without the dispatch: four of them are made per step)
static Tensor rows_of(const Tensor& buf, int64_t first, int64_t rows) {
  Tensor t = at::detail::make_tensor<c10::TensorImpl>(c10::TensorImpl::VIEW, c10::Storage(buf.storage()), buf.key_set(), buf.dtype());
  t.unsafeGetTensorImpl()->set_sizes_and_strides(std::array<int64_t, 4>{buf.size(0), buf.size(1), rows, buf.size(3)}, buf.strides(),
                                                 first * buf.size(3));
  return t;
}

Rooms::Owner Rooms::current_owner(const Tensor& t) {
  Owner o;
  o.stream = stream_of(t);
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  if (cudaStreamGetCaptureInfo((cudaStream_t)o.stream, &status, &o.capture) != cudaSuccess) {
    cudaGetLastError();
    return o;
  }
  if (status == cudaStreamCaptureStatusNone) o.capture = 0;
  o.known = true;
  return o;
}

GrownPair Rooms::fresh(const Tensor& like, int64_t batch, int64_t heads, int64_t rows, int64_t room, int64_t d) {
  at::AutoDispatchBelowADInplaceOrView no_view_tracking;   // a tracked view would keep its base
  GrownPair g;
  const Tensor k_buf = at::empty({batch, heads, rows + room, d}, like.options());
  const Tensor v_buf = at::empty({batch, heads, rows + room, d}, like.options());
  g.k = rows_of(k_buf, 0, rows);
  g.v = rows_of(v_buf, 0, rows);
  g.k_buf = k_buf.data_ptr();
  g.v_buf = v_buf.data_ptr();
  g.row = rows - 1;
  std::lock_guard<std::mutex> lock(mutex_);
  if (entries_.size() >= 256)      // forget the buffers that are gone
    for (auto it = entries_.begin(); it != entries_.end();) it = it->second.k.expired() ? entries_.erase(it) : std::next(it);
  const c10::StorageImpl* key = k_buf.storage().unsafeGetStorageImpl();
  auto weak = [](const Tensor& t) {
    return c10::weak_intrusive_ptr<c10::StorageImpl>(
        c10::intrusive_ptr<c10::StorageImpl>::reclaim_copy(t.storage().unsafeGetStorageImpl()));
  };
  entries_.erase(key);             // the address of a storage that is gone may come back
  entries_.emplace(key, Entry{weak(k_buf), weak(v_buf), rows, current_owner(like)});
  return g;
}

// The rows of k and v to the front of the buffers of g.  Caches whose heads are runs of whole 16-byte pieces at one distance
// from each other (all that come from here) go in one launch.
static void copy_rows(const GrownPair& g, const Tensor& k, const Tensor& v) {
  const int64_t B = k.size(0), H = k.size(1), rows = k.size(2), d = k.size(3), el = k.element_size();
  if (B * H * rows == 0) return;
  auto whole = [&](const void* p, int64_t step) { return reinterpret_cast<uintptr_t>(p) % 16 == 0 && step * el % 16 == 0; };
  const bool runs = k.strides() == v.strides() && k.stride(3) == 1 && (rows == 1 || k.stride(2) == d) && (B == 1 || k.stride(0) == k.stride(1) * H) &&
                    d * el % 16 == 0 && whole(k.data_ptr(), k.stride(1)) && whole(v.data_ptr(), k.stride(1)) && k.scalar_type() == g.k.scalar_type() &&
                    v.scalar_type() == g.k.scalar_type();
  if (!runs) {
    rows_of(g.k, 0, rows).copy_(k);
    rows_of(g.v, 0, rows).copy_(v);
    return;
  }
  nsa::CacheCopy c = {};
  c.src[0] = k.data_ptr(); c.src[1] = v.data_ptr(); c.dst[0] = g.k_buf; c.dst[1] = g.v_buf;
  c.src_step = k.stride(1) * el / 16; c.dst_step = g.k.stride(1) * el / 16; c.pieces = rows * d * el / 16; c.heads = (int)(B * H);
  check(nsa::launch_cache_copy(c, (cudaStream_t)stream_of(k)));
}

GrownPair Rooms::extend(const Tensor& k, const Tensor& v, int64_t room) {
  at::AutoDispatchBelowADInplaceOrView no_view_tracking;
  const int64_t B = k.size(0), H = k.size(1), rows = k.size(2), d = k.size(3);
  const c10::StorageImpl* ks = k.storage().unsafeGetStorageImpl();
  const c10::StorageImpl* vs = v.storage().unsafeGetStorageImpl();
  {
    std::lock_guard<std::mutex> lock(mutex_);
    auto it = entries_.find(ks);
    if (it != entries_.end() && !it->second.k.expired() && it->second.v._unsafe_get_target() == vs && k.strides() == v.strides() &&
        k.storage_offset() == v.storage_offset() && k.sizes() == v.sizes() && k.stride(3) == 1 && k.stride(2) == d &&
        k.stride(0) == k.stride(1) * H && k.scalar_type() == v.scalar_type()) {
      const int64_t capacity = k.stride(1) / d, first = k.storage_offset() / d, end = first + rows;
      if (it->second.used == end && end < capacity && it->second.owner == current_owner(k) &&
          (int64_t)k.storage().nbytes() == B * H * capacity * d * k.element_size()) {
        it->second.used = end + 1;
        GrownPair g;
        g.k_buf = k.storage().mutable_data();
        g.v_buf = v.storage().mutable_data();
        g.k = rows_of(k, first, rows + 1);
        g.v = rows_of(v, first, rows + 1);
        g.row = end;
        return g;
      }
    }
  }
  GrownPair g = fresh(k, B, H, rows + 1, room, d);
  copy_rows(g, k, v);
  return g;
}

}  // namespace nsa_host
