// DeviceSlab asked not to grow: a piece of what is free, or nothing.
#include <cassert>
#include <cstdint>
#include <cstdio>

#include "../../defmm_b200/csrc/device_slab.hpp"

static int allocations = 0;
static uintptr_t next_addr = 1u << 20;

extern "C" cudaError_t cudaMalloc(void** p, size_t n) {
  *p = reinterpret_cast<void*>(next_addr);
  next_addr += n;
  allocations++;
  return cudaSuccess;
}
extern "C" cudaError_t cudaFree(void*) {
  allocations--;
  return cudaSuccess;
}
extern "C" cudaError_t cudaGetLastError() { return cudaSuccess; }

int main() {
  dfb::DeviceSlab s;
  assert(!s.get(1000, false) && allocations == 0);  // nothing to take it from
  void* kept = s.get(1000);
  assert(kept && allocations == 1);
  void* q = s.get(size_t(3) << 20, false);  // the rest of the first chunk
  assert(q && q != kept && allocations == 1);
  assert(!s.get(size_t(3) << 20, false));    // not twice
  assert(!s.get(size_t(300) << 20, false));  // an allocation of its own is growth
  assert(allocations == 1);
  s.drop(q);
  assert(s.get(size_t(3) << 20, false) == q);
  s.release();
  assert(allocations == 0);
  std::puts("ok");
  return 0;
}
