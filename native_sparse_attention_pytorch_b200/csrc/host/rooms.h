// Caches that grow in place.
//
// A decoding step appends one row per head to [B, H, T, d] key and value caches and returns the longer caches.  Copying
// them for every token costs the whole cache per step; instead the rows live in buffers with some room behind the last
// row, and the returned caches are views of them.  A row is appended in place only where no tensor ever reached: by the
// cache that is the longest view its buffer has given out, on the stream the buffer was allocated on.  Everything else is
// copied into a new buffer: a second continuation of one cache, also when the first one has been dropped (kernels of other
// streams may still read its rows, which the allocator knows and this table does not); a continuation on another stream
// (whose tensors have to be that stream's own); a cache from elsewhere; no room left.  A step that is recorded into a CUDA
// graph appends only to buffers of the same recording: a replay writes the same rows again.  The copy is one
// launch (cache_copy_kernel).
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
  // Where a buffer comes from, and so who may append to it: the stream, and the recording of a CUDA graph (0: none)
  struct Owner {
    void* stream = nullptr;
    unsigned long long capture = 0;
    bool known = false;      // false: the stream cannot be asked at this moment
    bool operator==(const Owner& o) const { return known && o.known && stream == o.stream && capture == o.capture; }
  };
  static Owner current_owner(const Tensor& t);
  struct Entry {
    c10::weak_intrusive_ptr<c10::StorageImpl> k, v;
    int64_t used;            // rows given out
    Owner owner;
  };
  std::mutex mutex_;
  std::unordered_map<const c10::StorageImpl*, Entry> entries_;   // by the storage of the key buffer; holds nothing alive
};

}  // namespace nsa_host
