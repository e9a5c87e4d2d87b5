// Device memory of one solver context, taken from the driver in a few large
// blocks.  A context makes about ninety allocations while it loads a deck, and
// every cudaMalloc and cudaFree synchronises the device and costs 0.1 to 0.4 ms
// (tens of ms while other processes of the host allocate too); a block costs about
// as much as one of them.  New deck to first step on a graded 30^3 mesh (27
// Gauss points): 63 ms with an allocation per buffer, 36 ms from the pool.
//
// The pool belongs to its context (single-threaded use).  Blocks that hold nothing go
// back to the driver when a context loads another deck, and when the driver has
// no room for a new block (otherwise a deck of 70 GB after one of 60 would not fit
// 100 GB); everything goes back when the context ends.  A range returned with put() is handed out again
// only after the context's streams have finished what was queued on them, as
// cudaFree would have waited.  PoolScope makes a pool current for the calling
// thread while an entry point runs; buffers allocated meanwhile come from it.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <map>
#include <vector>

namespace cfd {

class DevPool {
 public:
  DevPool() = default;
  DevPool(const DevPool&) = delete;
  DevPool& operator=(const DevPool&) = delete;
  ~DevPool() {
    for (auto& b : blocks_) cudaFree(b.base);
  }
  void streams(cudaStream_t a, cudaStream_t b) {
    s_[0] = a;
    s_[1] = b;
  }
  cudaError_t get(size_t bytes, void** out) {
    bytes = (bytes + kAlign - 1) / kAlign * kAlign;
    for (auto& b : blocks_) {  // first fit
      for (auto it = b.free.begin(); it != b.free.end(); ++it) {
        if (it->second < bytes) continue;
        const size_t at = it->first, left = it->second - bytes;
        b.free.erase(it);
        if (left) b.free[at + bytes] = left;
        b.used[at] = bytes;
        *out = b.base + at;
        return cudaSuccess;
      }
    }
    // a new block: as much as the pool holds already (so their number grows
    // with the logarithm of the total), within bounds, or the request itself
    Block b;
    b.size = std::max(bytes, std::min(kMaxBlock, std::max(kMinBlock, total_)));
    cudaError_t e = cudaMalloc((void**)&b.base, b.size);
    if (e == cudaErrorMemoryAllocation && (trim() || b.size > bytes)) {
      cudaGetLastError();
      b.size = bytes;
      e = cudaMalloc((void**)&b.base, b.size);
    }
    if (e != cudaSuccess) return e;
    total_ += b.size;
    if (b.size > bytes) b.free[bytes] = b.size - bytes;
    b.used[0] = bytes;
    *out = b.base;
    blocks_.push_back(std::move(b));
    return cudaSuccess;
  }
  // Gives the blocks that hold nothing back; whether there were any.
  bool trim() {
    const auto first = std::partition(blocks_.begin(), blocks_.end(), [](const Block& b) { return !b.used.empty(); });
    const bool any = first != blocks_.end();
    for (auto it = first; it != blocks_.end(); ++it) {
      total_ -= it->size;
      cudaFree(it->base);
    }
    blocks_.erase(first, blocks_.end());
    return any;
  }
  size_t held() const { return total_; }
  void put(void* p) {
    if (s_[0]) {
      cudaStreamSynchronize(cudaStreamLegacy);  // plain cudaMemset and cudaMemcpy
      for (cudaStream_t s : s_) cudaStreamSynchronize(s);
    }
    for (auto& b : blocks_) {
      if (p < b.base || p >= b.base + b.size) continue;
      const size_t at = (char*)p - b.base;
      const auto u = b.used.find(at);
      if (u == b.used.end()) return;
      size_t lo = at, n = u->second;
      b.used.erase(u);
      const auto next = b.free.lower_bound(at);
      if (next != b.free.end() && next->first == at + n) {
        n += next->second;
        b.free.erase(next);
      }
      const auto after = b.free.lower_bound(at);
      if (after != b.free.begin()) {
        const auto prev = std::prev(after);
        if (prev->first + prev->second == at) {
          lo = prev->first;
          n += prev->second;
          b.free.erase(prev);
        }
      }
      b.free[lo] = n;
      return;
    }
  }

 private:
  static constexpr size_t kAlign = 512, kMinBlock = size_t(16) << 20, kMaxBlock = size_t(512) << 20;
  struct Block {
    char* base = nullptr;
    size_t size = 0;
    std::map<size_t, size_t> free, used;  // offset -> bytes
  };
  std::vector<Block> blocks_;
  size_t total_ = 0;
  cudaStream_t s_[2] = {nullptr, nullptr};
};

// The calling thread's current pool (null: plain cudaMalloc).
inline DevPool*& current_pool() {
  static thread_local DevPool* p = nullptr;
  return p;
}
struct PoolScope {
  DevPool* before;
  explicit PoolScope(DevPool* p) : before(current_pool()) { current_pool() = p; }
  ~PoolScope() { current_pool() = before; }
  PoolScope(const PoolScope&) = delete;
  PoolScope& operator=(const PoolScope&) = delete;
};

}  // namespace cfd
