// Compaction of the M2L lists at upload: which source slots some target slot
// meets, which target slots have a list, and the lists renumbered to match.
//
// On a sphere of 250,000 points at 45 wavelengths 29% of the source slots and
// of the target slots take no part in M2L (their directions only pass
// through to the next level), so M2F would transform and M2L visit them for
// nothing.
#include "m2l_lists.hpp"

#include <cub/cub.cuh>

#include <algorithm>

namespace dfb {
namespace {

__global__ void k_flag_targets(const int64_t* __restrict__ ptr, int64_t n, int32_t* __restrict__ flag) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i <= n) flag[i] = i < n && ptr[i + 1] > ptr[i] ? 1 : 0;
}

// every writer of a flag writes the same value
__global__ void k_flag_sources(const int32_t* __restrict__ src, int64_t n, int32_t* __restrict__ flag) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x)
    flag[src[e]] = 1;
}

__global__ void k_compact_targets(const int64_t* __restrict__ ptr, int64_t n, const int32_t* __restrict__ rank,
                                  int64_t* __restrict__ cptr, int32_t* __restrict__ list) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i > n) return;
  if (i == n) {
    cptr[rank[n]] = ptr[n];
  } else if (rank[i + 1] > rank[i]) {
    cptr[rank[i]] = ptr[i];
    list[rank[i]] = (int32_t)i;
  }
}

__global__ void k_compact_sources(int64_t n, const int32_t* __restrict__ rank, int32_t* __restrict__ list) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n && rank[i + 1] > rank[i]) list[rank[i]] = (int32_t)i;
}

__global__ void k_rank_entries(int64_t n, const int32_t* __restrict__ rank, int32_t* __restrict__ src) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x)
    src[e] = rank[src[e]];
}

__global__ void k_pick(int64_t n, const int64_t* __restrict__ at, const int32_t* __restrict__ rank,
                       int64_t* __restrict__ out) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) out[i] = rank[at[i]];
}

unsigned blocks(int64_t n) { return (unsigned)((n + 255) / 256); }

}  // namespace

int device_m2l_lists(const int64_t* ptr, int32_t* src, int64_t nent, int64_t nT, int64_t nS,
                     std::vector<int64_t>& atT, std::vector<int64_t>& atS, int64_t* cptr, int32_t* tlist,
                     int32_t* slist, DeviceSlab& slab, std::string& err) {
  const int64_t nmax = std::max(nT, nS) + 1, na = (int64_t)(atT.size() + atS.size());
  size_t scan = 0;
  cudaError_t e = cub::DeviceScan::ExclusiveSum(nullptr, scan, (int32_t*)nullptr, (int32_t*)nullptr, nmax);
  auto up = [](size_t b) { return (b + 255) / 256 * 256; };
  const size_t flag_b = up(nmax * 4), at_b = up(na * 8), need = 2 * flag_b + 2 * at_b + scan;
  DeviceSlab own;  // where the plan's slab has no room left: it would keep the scratch
  char* tmp = (char*)slab.get(need, false);
  char* const borrowed = tmp;
  if (e == cudaSuccess && !tmp && !(tmp = (char*)own.get(need))) e = cudaErrorMemoryAllocation;
  int32_t *flag = (int32_t*)tmp, *rank = (int32_t*)(tmp + flag_b);
  int64_t *at = (int64_t*)(tmp + 2 * flag_b), *got = (int64_t*)(tmp + 2 * flag_b + at_b);
  void* cubtmp = tmp + 2 * flag_b + 2 * at_b;
  std::vector<int64_t> both(atT);
  both.insert(both.end(), atS.begin(), atS.end());
  if (e == cudaSuccess && na) e = cudaMemcpy(at, both.data(), na * 8, cudaMemcpyHostToDevice);
  auto ranks = [&](int64_t n, int64_t a0, int64_t a1) -> cudaError_t {  // scan of flag[0, n], picked at [a0, a1)
    size_t b = scan;
    const cudaError_t r = cub::DeviceScan::ExclusiveSum(cubtmp, b, flag, rank, n + 1);
    if (r == cudaSuccess && a1 > a0) k_pick<<<blocks(a1 - a0), 256>>>(a1 - a0, at + a0, rank, got + a0);
    return r;
  };
  const unsigned ge = (unsigned)std::min<int64_t>(std::max<int64_t>(1, (nent + 255) / 256), 148 * 64);
  if (e == cudaSuccess) {
    k_flag_targets<<<blocks(nT + 1), 256>>>(ptr, nT, flag);
    e = ranks(nT, 0, (int64_t)atT.size());
  }
  if (e == cudaSuccess) {
    k_compact_targets<<<blocks(nT + 1), 256>>>(ptr, nT, rank, cptr, tlist);
    e = cudaMemsetAsync(flag, 0, (nS + 1) * 4, 0);
  }
  if (e == cudaSuccess) {
    if (nent) k_flag_sources<<<ge, 256>>>(src, nent, flag);
    e = ranks(nS, (int64_t)atT.size(), na);
  }
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e == cudaSuccess) {  // the entries last: they are as they were when anything before fails
    if (nS) k_compact_sources<<<blocks(nS), 256>>>(nS, rank, slist);
    if (nent) k_rank_entries<<<ge, 256>>>(nent, rank, src);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess && na) e = cudaMemcpy(both.data(), got, na * 8, cudaMemcpyDeviceToHost);
  const cudaError_t d = cudaDeviceSynchronize();
  if (e == cudaSuccess) e = d;
  if (borrowed) slab.drop(borrowed);
  if (e == cudaSuccess) {
    std::copy(both.begin(), both.begin() + atT.size(), atT.begin());
    std::copy(both.begin() + atT.size(), both.end(), atS.begin());
    return 0;
  }
  cudaGetLastError();
  err = std::string("M2L list compaction: ") + cudaGetErrorString(e);
  return e == cudaErrorMemoryAllocation ? -5 : -4;
}

}  // namespace dfb
