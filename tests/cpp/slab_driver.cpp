// DeviceSlab against a fake allocator: random pieces never overlap, dropped
// ones are joined and used again, and everything is given back.
#include <cassert>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <set>

#include "../../defmm_b200/csrc/device_slab.hpp"

static std::map<void*, size_t> live;      // the fake device's allocations
static uintptr_t next_addr = 1u << 20;    // adjacent allocations: no gaps between them
static size_t in_use = 0, limit = size_t(4) << 30;

extern "C" cudaError_t cudaMalloc(void** p, size_t n) {
  if (in_use + n > limit) return cudaErrorMemoryAllocation;
  *p = reinterpret_cast<void*>(next_addr);
  next_addr += n;
  live[*p] = n;
  in_use += n;
  return cudaSuccess;
}
extern "C" cudaError_t cudaFree(void* p) {
  const auto it = live.find(p);
  assert(it != live.end());
  in_use -= it->second;
  live.erase(it);
  return cudaSuccess;
}
extern "C" cudaError_t cudaGetLastError() { return cudaSuccess; }

int main(int argc, char** argv) {
  std::mt19937 rng(argc > 1 ? atoi(argv[1]) : 1);
  {
    dfb::DeviceSlab s;
    std::map<uintptr_t, size_t> held;
    for (int step = 0; step < 20000; step++) {
      if (held.size() < 60 && rng() % 3) {
        const size_t n = rng() % 50 == 0 ? size_t(rng()) % (size_t(300) << 20) : size_t(1) << rng() % 24;
        void* q = s.get(n);
        if (!q) {  // out of memory: nothing changed
          assert(in_use + n + 256 > limit);
          continue;
        }
        const uintptr_t a = reinterpret_cast<uintptr_t>(q);
        assert(a % 256 == 0);
        const auto up = held.upper_bound(a);
        assert(up == held.end() || a + n <= up->first);
        if (up != held.begin()) assert(std::prev(up)->first + std::prev(up)->second <= a);
        auto c = live.upper_bound(q);  // inside one allocation
        assert(c != live.begin());
        --c;
        assert(a + n <= reinterpret_cast<uintptr_t>(c->first) + c->second);
        held[a] = n;
      } else if (!held.empty()) {
        auto it = std::next(held.begin(), rng() % held.size());
        s.drop(reinterpret_cast<void*>(it->first));
        held.erase(it);
      }
    }
    for (const auto& h : held) s.drop(reinterpret_cast<void*>(h.first));
    const size_t before = live.size();
    void* q = s.get(size_t(100) << 20);  // joined again: a whole chunk serves it
    assert(q && live.size() == before);
    s.drop(nullptr);
    limit = in_use;
    assert(!s.get(size_t(500) << 20));
  }
  assert(live.empty());
  {
    dfb::DeviceSlab s;
    limit = size_t(1) << 20;  // less than a chunk: the piece alone
    assert(s.get(1000) && in_use == 1024);
    const std::vector<void*> mine = s.take();
    s.release();
    assert(mine.size() == 1 && live.size() == 1);
    cudaFree(mine[0]);
  }
  assert(live.empty());
  std::puts("ok");
  return 0;
}
