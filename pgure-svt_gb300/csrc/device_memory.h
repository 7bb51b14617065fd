// device_memory.h — device memory of a call (capi.cu): arrays carved out of blocks
// that a process-wide cache keeps between calls.  Host code on the CUDA runtime
// API alone.
#ifndef PGSVT_DEVICE_MEMORY_H
#define PGSVT_DEVICE_MEMORY_H

#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <exception>
#include <mutex>
#include <stdexcept>
#include <string>
#include <vector>

#include "pgsvt.h"

namespace pgsvt {

// identifier of the calling thread's current CUDA context (0: none yet)
unsigned long long current_context_id();

struct Fail : std::runtime_error {
  int code;
  int cuda;
  Fail(int c, const std::string& m, int ce = 0) : std::runtime_error(m), code(c), cuda(ce) {}
};

#define PGSVT_CK(x)                                                                  \
  do {                                                                               \
    cudaError_t e_ = (x);                                                            \
    if (e_ != cudaSuccess)                                                           \
      throw Fail(e_ == cudaErrorMemoryAllocation ? PGSVT_ERR_OOM : PGSVT_ERR_CUDA,   \
                 std::string(#x) + ": " + cudaGetErrorString(e_), (int)e_);          \
  } while (0)

// Device memory of a call.  A call needs 25 to 90 arrays; allocating and freeing
// each took 0.9 of 1.8 ms on a 32 x 32 x 16 sequence and 11 of 203 ms on 256 x
// 256 x 100, so arrays are carved out of blocks, and the blocks of a finished
// call stay in a process-wide cache for the next one.  The cache is bounded
// (kCacheBytes over all devices, the blocks longest unused are freed first) and
// is given back by pgsvt_release_memory(), when an allocation fails, and at the end
// of any call that leaves the device with little free memory.  Blocks enter it only
// when the call's device work has completed, so any thread and stream may take them.
constexpr size_t kCacheBytes = (size_t)16 << 30;
constexpr size_t kBlock = (size_t)4 << 20;  // least block; sizes are multiples of half of it

struct MemBlock {
  void* p;
  size_t n;
  int dev;
  unsigned long long ctx;  // the context that owns it (a device reset destroys it)
};

class BlockCache {
 public:
  // a block of at least n bytes on the current device
  MemBlock take(size_t n) {
    n = std::max(kBlock, (n + kBlock / 2 - 1) / (kBlock / 2) * (kBlock / 2));
    int dev = 0;
    PGSVT_CK(cudaGetDevice(&dev));
    if (current_context_id() == 0) PGSVT_CK(cudaSetDevice(dev));  // a thread's first CUDA call
    const unsigned long long ctx = current_context_id();
    {
      std::lock_guard<std::mutex> lk(mu_);
      size_t best = free_.size();
      for (size_t i = 0; i < free_.size(); ++i) {
        const MemBlock& b = free_[i];
        if (b.dev == dev && b.ctx == ctx && b.n >= n && b.n <= 2 * n &&
            (best == free_.size() || b.n < free_[best].n))
          best = i;
      }
      if (best < free_.size()) {
        const MemBlock b = free_[best];
        free_.erase(free_.begin() + (long)best);
        bytes_ -= b.n;
        return b;
      }
    }
    MemBlock b{nullptr, n, dev, 0};
    cudaError_t e = cudaMalloc(&b.p, n);
    if (e == cudaErrorMemoryAllocation) {
      cudaGetLastError();
      trim(0);
      e = cudaMalloc(&b.p, n);
    }
    PGSVT_CK(e);
    b.ctx = current_context_id();  // (the allocation made a context current)
    return b;
  }
  void give(const MemBlock& b) {
    if (b.ctx == 0 || b.ctx != current_context_id()) {  // not known to be alive and reusable
      cudaFree(b.p);
      return;
    }
    {
      std::lock_guard<std::mutex> lk(mu_);
      free_.push_back(b);
      bytes_ += b.n;
    }
    trim(kCacheBytes);
  }
  // bytes cached for the current device
  size_t cached() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    const unsigned long long ctx = current_context_id();
    std::lock_guard<std::mutex> lk(mu_);
    size_t t = 0;
    for (const MemBlock& b : free_) t += (b.dev == dev && b.ctx == ctx) ? b.n : 0;
    return t;
  }
  // Free the blocks longest unused until at most `keep` bytes are cached; on any
  // thread, so one without a current context gets the device's first.
  void trim(size_t keep) {
    for (;;) {
      MemBlock b{};
      {
        std::lock_guard<std::mutex> lk(mu_);
        if (bytes_ <= keep || free_.empty()) return;
        b = free_.front();
        free_.erase(free_.begin());
        bytes_ -= b.n;
      }
      int dev = 0;
      cudaGetDevice(&dev);
      if (dev != b.dev || current_context_id() == 0) cudaSetDevice(b.dev);
      if (b.ctx == current_context_id()) cudaFree(b.p);  // else it went with its context
      if (dev != b.dev) cudaSetDevice(dev);
    }
  }

 private:
  std::mutex mu_;
  std::vector<MemBlock> free_;  // least recently used first
  size_t bytes_ = 0;
};

// (never destroyed: calls may still run on other threads at exit)
inline BlockCache& block_cache() {
  static BlockCache* c = new BlockCache;
  return *c;
}

// The arrays of one call.  The owner's device work has completed when it is
// destroyed, except when an exception ends the call.
struct DevMem {
  std::vector<MemBlock> blocks;
  size_t used = 0;  // of the last block
  const int depth = std::uncaught_exceptions();
  void* get(size_t bytes) {
    bytes = (std::max<size_t>(bytes, 16) + 255) / 256 * 256;
    if (blocks.empty() || used + bytes > blocks.back().n) {
      const MemBlock b = block_cache().take(bytes);
      // go on filling whichever block has more room left
      if (blocks.empty() || b.n - bytes >= blocks.back().n - used) {
        blocks.push_back(b);
        used = bytes;
      } else {
        blocks.insert(blocks.end() - 1, b);
      }
      return b.p;
    }
    void* p = (char*)blocks.back().p + used;
    used += bytes;
    return p;
  }
  template <typename T>
  T* arr(size_t n) { return (T*)get(n * sizeof(T)); }
  void release() {
    if (blocks.empty()) return;
    if (std::uncaught_exceptions() > depth) cudaDeviceSynchronize();
    for (const MemBlock& b : blocks) block_cache().give(b);
    blocks.clear();
    size_t freeb = 0, totb = 0;
    if (cudaMemGetInfo(&freeb, &totb) == cudaSuccess && freeb < totb / 8) block_cache().trim(0);
  }
  DevMem() = default;
  DevMem(const DevMem&) = delete;
  DevMem& operator=(const DevMem&) = delete;
  ~DevMem() { release(); }
};

// Run a call, once more if it failed for lack of device memory.  The blocks that a
// call reuses are up to twice as large as it needs; the second run has an empty
// cache and allocates no more than its arrays.  (A call allocates before it writes
// any output.)
template <typename Fn>
void with_retry(Fn&& fn) {
  try {
    fn();
    return;
  } catch (const Fail& f) {
    if (f.cuda != (int)cudaErrorMemoryAllocation) throw;
    cudaGetLastError();
  }
  block_cache().trim(0);
  fn();
}

}  // namespace pgsvt

#endif
