// Whether the eight fields of a state that a caller passed can be copied as one.
//
// Fields that lie one after another are one copy instead of eight (the copies of
// 256 boxes of 8.8k cells took 10 ms as 2,048 of 35 KB), but equal addresses do
// not make them one allocation: buffers allocated or pinned one by one may lie
// back to back, and a copy across two of them may be refused.
#pragma once
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace nmhd {

// The device, managed or pinned allocation that holds an address: [begin, end),
// empty for pageable memory; `known` false where the driver does not say.
struct Allocation {
  bool known;
  uintptr_t begin, end;
};

inline Allocation allocation_of(const void *p) {
  static const PFN_cuPointerGetAttributes_v7000 attributes = [] {
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    const bool ok = cudaGetDriverEntryPointByVersion("cuPointerGetAttributes", &fn, 7000, cudaEnableDefault, &q) ==
                        cudaSuccess &&
                    q == cudaDriverEntryPointSuccess;
    return reinterpret_cast<PFN_cuPointerGetAttributes_v7000>(ok ? fn : nullptr);
  }();
  CUdeviceptr begin = 0;  // both stay 0 for pageable memory
  size_t size = 0;
  CUpointer_attribute what[2] = {CU_POINTER_ATTRIBUTE_RANGE_START_ADDR, CU_POINTER_ATTRIBUTE_RANGE_SIZE};
  void *to[2] = {&begin, &size};
  if (!attributes || attributes(2, what, to, (CUdeviceptr)p) != CUDA_SUCCESS) return Allocation{false, 0, 0};
  return Allocation{true, (uintptr_t)begin, (uintptr_t)begin + size};
}

// Whether fields of n floats each are one run of memory inside one allocation, or
// all in pageable memory.  of: allocation_of(), asked for the first field unless
// `held` (the last answer, for callers with many states) covers it.
template <class Of>
bool one_run(const float *const fields[8], size_t n, Allocation &held, Of &&of) {
  for (int v = 1; v < 8; ++v)
    if (fields[v] != fields[0] + v * n) return false;
  const uintptr_t begin = (uintptr_t)fields[0], end = begin + 8 * n * sizeof(float);
  if (!(held.known && held.begin <= begin && begin < held.end)) held = of(fields[0]);
  if (!held.known) return false;
  if (held.begin < held.end) return held.begin <= begin && end <= held.end;
  for (int v = 1; v < 8; ++v) {
    const Allocation a = of(fields[v]);
    if (!a.known || a.begin < a.end) return false;
  }
  return true;
}

}  // namespace nmhd
