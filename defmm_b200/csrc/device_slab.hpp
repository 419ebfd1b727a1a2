// Device memory in pieces of a few large allocations.  A plan build takes and
// drops some 250 arrays, most of them small, and cudaMalloc and cudaFree cost
// up to a millisecond each (cudaFree also waits for the device): they were
// two thirds of prcmpt on a 50,000-point problem.  Pieces come from chunks of
// 4 MB that double up to 128 MB; a piece of 128 MB or more is an allocation
// of its own, given back when dropped, so that the peak of a large build is
// its arrays' (and the chunks').  Everything is given back with the slab.
//
// A dropped piece may be handed out again at once: its users have to be
// ordered on one stream (the plan build's kernels all run on the default
// stream), as with cudaFree followed by cudaMalloc.  Not shared between
// threads.
#pragma once

#include <algorithm>
#include <cstddef>
#include <map>
#include <vector>

#include <cuda_runtime.h>

namespace dfb {

class DeviceSlab {
 public:
  DeviceSlab() = default;
  DeviceSlab(const DeviceSlab&) = delete;
  DeviceSlab& operator=(const DeviceSlab&) = delete;
  ~DeviceSlab() { release(); }

  // nullptr when out of device memory (the CUDA error is cleared), or when no
  // free piece serves and the slab is not to grow
  void* get(size_t bytes, bool grow = true) {
    bytes = (std::max<size_t>(bytes, 1) + 255) / 256 * 256;
    if (bytes >= kBig) {
      if (!grow) return nullptr;
      void* p = alloc(bytes);
      if (p) big_.push_back(p);
      return p;
    }
    for (auto it = free_.begin(); it != free_.end(); ++it)
      if (it->second >= bytes) return carve(it, bytes);
    if (!grow) return nullptr;
    char* c = static_cast<char*>(alloc(std::max(bytes, grow_)));
    size_t size = std::max(bytes, grow_);
    if (!c) {
      size = bytes;
      if (!(c = static_cast<char*>(alloc(size)))) return nullptr;
    }
    grow_ = std::min(kBig, 2 * grow_);
    chunks_.push_back(c);
    return carve(free_.emplace(c, size).first, bytes);
  }

  void drop(void* q) {
    const auto b = std::find(big_.begin(), big_.end(), q);
    if (b != big_.end()) {
      cudaFree(q);
      big_.erase(b);
      return;
    }
    const auto u = used_.find(static_cast<char*>(q));
    if (u == used_.end()) return;
    char* p = u->first;
    size_t n = u->second;
    used_.erase(u);
    auto next = free_.lower_bound(p);  // join with free neighbours of the same chunk
    if (next != free_.end() && next->first == p + n && !chunk_start(next->first)) {
      n += next->second;
      next = free_.erase(next);
    }
    if (next != free_.begin() && !chunk_start(p)) {
      auto prev = std::prev(next);
      if (prev->first + prev->second == p) {
        prev->second += n;
        return;
      }
    }
    free_.emplace(p, n);
  }

  // the allocations behind the pieces: the caller frees them from now on
  std::vector<void*> take() {
    std::vector<void*> v(big_.begin(), big_.end());
    v.insert(v.end(), chunks_.begin(), chunks_.end());
    big_.clear();
    chunks_.clear();
    free_.clear();
    used_.clear();
    grow_ = kFirst;
    return v;
  }

  void release() {
    for (void* p : take()) cudaFree(p);
  }

 private:
  static constexpr size_t kFirst = size_t(4) << 20, kBig = size_t(128) << 20;
  std::vector<void*> big_;
  std::vector<char*> chunks_;
  std::map<char*, size_t> free_, used_;  // pieces by address
  size_t grow_ = kFirst;

  static void* alloc(size_t bytes) {
    void* p = nullptr;
    if (cudaMalloc(&p, bytes) == cudaSuccess) return p;
    cudaGetLastError();
    return nullptr;
  }
  // two chunks can lie next to each other: pieces never span them
  bool chunk_start(const char* p) const { return std::find(chunks_.begin(), chunks_.end(), p) != chunks_.end(); }
  void* carve(std::map<char*, size_t>::iterator it, size_t bytes) {
    char* p = it->first;
    const size_t left = it->second - bytes;
    free_.erase(it);
    if (left) free_.emplace(p + bytes, left);
    used_.emplace(p, bytes);
    return p;
  }
};

}  // namespace dfb
