// Flat cell indices: division by a grid's extents and the loop of a
// one-cell-per-thread pass.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace cfdb {
namespace res {

// Division of a cell index (< 2^31) by a fixed divisor: one 32 x 32 -> 64
// multiply (m = ceil(2^s / d), s = 31 + ceil(log2 d), m < 2^32).
struct FastDiv {
  uint32_t m = 0, s = 31;
  __device__ __forceinline__ uint32_t div(uint32_t c) const {
    return (uint32_t)(((uint64_t)c * m) >> s);
  }
};
__host__ __device__ inline FastDiv fast_div(uint32_t d) {
  FastDiv f;
  uint32_t l = 0;
  while ((1ull << l) < d) ++l;
  f.s = 31 + l;
  f.m = (uint32_t)(((1ull << f.s) + d - 1) / d);
  return f;
}

// f(c, i, j, k) for this thread's cells of n (at most 2^31) in blocks of 256
// threads.  Flat indices are unsigned: past n - gridDim.x * 256 the next
// index, and past 2^31 - a plane the index of a face, leave an int.
template <class F>
__device__ __forceinline__ void gather_cells(uint32_t n, int nx, int ny, FastDiv dx, FastDiv dy, F f) {
  for (uint32_t c = blockIdx.x * 256 + threadIdx.x; c < n; c += gridDim.x * 256) {
    const uint32_t row = dx.div(c), k = dy.div(row);
    f(c, (int)(c - row * (uint32_t)nx), (int)(row - k * (uint32_t)ny), (int)k);
  }
}

}  // namespace res
}  // namespace cfdb
