// Caches that grow in place.
//
// A decoding step appends one row per head to [B, H, T, d] key and value caches and returns the longer caches.  Copying
// them for every token costs the whole cache per step; instead the rows live in buffers with some room behind the last
// row, and the returned caches are views of them.  The views a caller holds never change: a row is only appended where
// no live tensor reaches -- either the cache that is being extended is the longest view of its buffer, or its buffer
// has no other tensor on it.  Otherwise (two continuations of one cache, a cache from elsewhere, no room left) the rows
// are copied into a new buffer.
#pragma once

#include <mutex>
#include <unordered_map>

#include "nsa_host.h"

namespace nsa_host {

struct GrownPair {
  Tensor k, v;        // views of `rows` rows, the last of them not written yet
  int64_t row;        // index of that row in the buffers
  void *k_buf, *v_buf;   // the buffers [B, H, capacity, d]; the views' strides are theirs
};

class Rooms {
 public:
  // Buffers for caches of `rows` rows with `room` rows behind them; registered, contents uninitialised.
  GrownPair fresh(const Tensor& like, int64_t batch, int64_t heads, int64_t rows, int64_t room, int64_t d);
  // The caches one row longer, in place where that is safe.
  GrownPair extend(const Tensor& k, const Tensor& v, int64_t room);
  static Rooms& instance();

 private:
  struct Entry {
    c10::weak_intrusive_ptr<c10::StorageImpl> k, v;
    int64_t used;
  };
  std::mutex mutex_;
  std::unordered_map<const c10::StorageImpl*, Entry> entries_;   // by the storage of the key buffer; holds nothing alive
};

}  // namespace nsa_host
