// devmem.cu -- device memory kept for reuse (see devmem.hpp).
#include "devmem.hpp"

#include <algorithm>
#include <list>
#include <map>
#include <mutex>
#include <set>
#include <unordered_map>

namespace adatm {

namespace {

// A block returned to the pool: free for work that follows on its stream, or
// (stream nullptr) for anybody.
struct Kept {
  void *p;
  size_t bytes;
  int dev;
  cudaStream_t stream;
};

struct Live {
  size_t bytes;
  int dev;
  cudaStream_t stream;
};

struct Pool {
  std::mutex mu;
  std::set<cudaStream_t> streams;         // between stream_opened and stream_closed
  std::unordered_map<void *, Live> live;  // blocks of the pool that are in use
  std::list<Kept> kept;                   // oldest first
  size_t kept_bytes = 0;
};

Pool &pool() {
  static Pool *p = new Pool();  // never destroyed: buffers may outlive static objects
  return *p;
}

// Sizes that blocks come in: eight steps per power of two, 512 bytes at least,
// so that a block fits the next request of about its size.
size_t block_size(size_t bytes) {
  size_t top = 512;
  while (top < bytes) top <<= 1;
  const size_t step = std::max<size_t>(512, top >> 4);
  return (bytes + step - 1) / step * step;
}

void give_back(Pool &p, std::list<Kept>::iterator it) {
  cudaFree(it->p);
  p.kept_bytes -= it->bytes;
  p.kept.erase(it);
}

}  // namespace

void *dev_alloc(size_t bytes, cudaStream_t stream) {
  void *out = nullptr;
  const size_t size = block_size(bytes);
  Pool &p = pool();
  bool pooled = false;
  int dev = 0;
  if (stream != nullptr && size <= kPoolBlock) {
    ADATM_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lk(p.mu);
    pooled = p.streams.count(stream) != 0;
    if (pooled)
      for (auto it = p.kept.begin(); it != p.kept.end(); ++it)
        if (it->bytes == size && it->dev == dev && (it->stream == nullptr || it->stream == stream)) {
          out = it->p;
          p.kept_bytes -= size;
          p.kept.erase(it);
          p.live[out] = {size, dev, stream};
          return out;
        }
  }
  cudaError_t err = cudaMalloc(&out, pooled ? size : bytes);
  if (err == cudaErrorMemoryAllocation) {
    // what the pool keeps may be what is missing
    cudaGetLastError();
    std::lock_guard<std::mutex> lk(p.mu);
    while (!p.kept.empty()) give_back(p, p.kept.begin());
    err = cudaMalloc(&out, pooled ? size : bytes);
  }
  ADATM_CUDA(err);
  if (pooled) {
    std::lock_guard<std::mutex> lk(p.mu);
    p.live[out] = {size, dev, stream};
  }
  return out;
}

void dev_free(void *ptr) {
  if (!ptr) return;
  Pool &p = pool();
  std::unique_lock<std::mutex> lk(p.mu);
  const auto it = p.live.find(ptr);
  if (it == p.live.end()) {
    lk.unlock();
    cudaFree(ptr);
    return;
  }
  const Live b = it->second;
  p.live.erase(it);
  if (p.streams.count(b.stream) == 0) {
    // its stream is closed: nothing orders its last use any more
    lk.unlock();
    cudaFree(ptr);
    return;
  }
  p.kept.push_back({ptr, b.bytes, b.dev, b.stream});
  p.kept_bytes += b.bytes;
  while (p.kept_bytes > kPoolKept) give_back(p, p.kept.begin());
}

void dev_trim() {
  Pool &p = pool();
  std::lock_guard<std::mutex> lk(p.mu);
  while (!p.kept.empty()) give_back(p, p.kept.begin());
}

void stream_opened(cudaStream_t s) {
  std::lock_guard<std::mutex> lk(pool().mu);
  pool().streams.insert(s);
}

void stream_closed(cudaStream_t s) {
  Pool &p = pool();
  const bool idle = cudaStreamSynchronize(s) == cudaSuccess;
  std::lock_guard<std::mutex> lk(p.mu);
  p.streams.erase(s);
  for (auto it = p.kept.begin(); it != p.kept.end();) {
    auto at = it++;
    if (at->stream != s) continue;
    if (idle) at->stream = nullptr;
    else give_back(p, at);
  }
  // the last user of the library's streams leaves: nothing stays behind
  if (p.streams.empty())
    while (!p.kept.empty()) give_back(p, p.kept.begin());
}

}  // namespace adatm
