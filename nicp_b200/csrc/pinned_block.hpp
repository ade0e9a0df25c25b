// pinned_block.hpp -- a page-locked block that grows on demand: a context's
// staging for uploads, and the one for results.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

namespace nicp {

struct PinnedBlock {
  // Captured loops hold the block's address, so each move costs them: the first
  // block has room for loops of 700 pairs and builds of a thousand frames of
  // 640x480, and from there a larger one is at least twice as large.
  static constexpr size_t kFirst = (size_t)1 << 20;
  char *p = nullptr;
  size_t cap = 0;
  // Room for `bytes`.  The old block is freed where it is too small: whoever
  // used it is done.  A block that cannot be had leaves none, and the next call
  // tries again.
  cudaError_t reserve(size_t bytes) {
    if (bytes <= cap) return cudaSuccess;
    size_t want = cap ? cap : kFirst / 2;
    while (want *= 2, want < bytes) {}
    release();
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
