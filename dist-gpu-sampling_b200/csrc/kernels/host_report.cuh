// Sizes of a sequence that the host spins on in pinned memory.
#pragma once
#include <cstdint>

namespace dgs {

// `code`: an error by which the host decides, as soon as the last size has landed, whether the batch counts (0: none).  It has
// to be at the host before the sizes are, so the thread that reports them raises it and fences in between.  (Kernels in
// front leave it in device memory for that.  A fence on every call instead: 2 us more until the host has the sizes.)
__device__ __forceinline__ void report_sizes(int64_t* dst, const int64_t* const* src, int n, int32_t code, int32_t* status) {
  if (code != 0) {
    raise_status(status, code);
    __threadfence_system();
  }
  for (int k = 0; k < n; ++k) dst[k] = *src[k];
  __threadfence_system();
}

}  // namespace dgs
