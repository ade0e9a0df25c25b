// pinned_block.hpp -- a page-locked block that grows on demand: a context's
// staging for uploads, and the one for results.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

namespace nicp {

struct PinnedBlock {
  char *p = nullptr;
  size_t cap = 0;
  // Room for `bytes`.  The old block is freed where it is too small: whoever
  // used it is done.  A block that cannot be had leaves none, and the next call
  // tries again.
  cudaError_t reserve(size_t bytes) {
    if (bytes <= cap) return cudaSuccess;
    release();
    const size_t want = (bytes + bytes / 4 + 0xffff) & ~(size_t)0xffff;
    const cudaError_t e = cudaMallocHost(&p, want);
    if (e != cudaSuccess) {
      p = nullptr;
      return e;
    }
    cap = want;
    return cudaSuccess;
  }
  void release() {
    if (p) cudaFreeHost(p);
    p = nullptr;
    cap = 0;
  }
};

}  // namespace nicp
