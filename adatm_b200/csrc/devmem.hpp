// devmem.hpp -- device buffers, and a pool of the ones that come and go.
//
// Building an engine takes and returns about a hundred buffers, and cudaMalloc
// and cudaFree (which waits for the whole device) cost more than the kernels
// in between: a 5th-order engine of 3.5M nonzeros and its first MTTKRP took 51
// ms, of which the device worked 4; with the pool 11.8.
//
// A buffer taken for a stream of the library is used by work on that stream
// (or work ordered with it) alone. Returned, it is kept for later requests of
// its size on the same stream, which the stream itself orders; when the stream
// is closed, it is waited for and its buffers are free for any stream. The
// pool keeps at most kPoolKept bytes, gives the oldest back beyond that, gives
// everything back when one of its own allocations fails, when the last stream
// closes or when it is told to (dev_trim: the memory is missing to somebody
// else), and takes no block above kPoolBlock. Buffers without a stream, or of a
// stream that is not the library's, go straight to cudaMalloc and cudaFree.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

#include "check.hpp"

namespace adatm {

constexpr size_t kPoolBlock = (size_t)64 << 20;
constexpr size_t kPoolKept = (size_t)512 << 20;

void *dev_alloc(size_t bytes, cudaStream_t stream);
void dev_free(void *p);
void dev_trim();

// A stream that buffers may be taken for, from its creation to just before its
// destruction.
void stream_opened(cudaStream_t s);
void stream_closed(cudaStream_t s);

// A device buffer of n elements.
template <typename T>
struct DevBuf {
  T *p = nullptr;
  size_t n = 0;
  DevBuf() = default;
  explicit DevBuf(size_t count, cudaStream_t s = nullptr) { alloc(count, s); }
  DevBuf(const DevBuf &) = delete;
  DevBuf &operator=(const DevBuf &) = delete;
  DevBuf(DevBuf &&o) noexcept : p(o.p), n(o.n) {
    o.p = nullptr;
    o.n = 0;
  }
  DevBuf &operator=(DevBuf &&o) noexcept {
    if (this != &o) {
      reset();
      p = o.p;
      n = o.n;
      o.p = nullptr;
      o.n = 0;
    }
    return *this;
  }
  ~DevBuf() { reset(); }
  void alloc(size_t count, cudaStream_t s = nullptr) {
    reset();
    if (count) p = static_cast<T *>(dev_alloc(count * sizeof(T), s));
    n = count;
  }
  void reset() {
    dev_free(p);
    p = nullptr;
    n = 0;
  }
  T *get() const { return p; }
  size_t bytes() const { return n * sizeof(T); }
};

}  // namespace adatm
