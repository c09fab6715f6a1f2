// Enough of the device's vocabulary to compile the header-only device routines
// with a host compiler: one thread per block, atomics and fences as plain code.
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>
#include <vector>

using std::max;
using std::min;

static uint3 threadIdx{0, 0, 0}, blockIdx{0, 0, 0};
static dim3 blockDim{1, 1, 1}, gridDim{1, 1, 1};

inline void __syncthreads() {}
inline int __syncthreads_and(int v) { return v; }
inline void __threadfence() {}
inline void __nanosleep(unsigned) {}
template <typename T>
inline T __ldg(const T* p) { return *p; }
template <typename T>
inline T __ldcg(const T* p) { return *p; }
template <typename T>
inline void __stcg(T* p, T v) { *p = v; }
template <typename T>
inline T __shfl_xor_sync(unsigned, T v, int) { return v; }
inline unsigned atomicAdd(unsigned* p, unsigned v) { unsigned o = *p; *p += v; return o; }
inline unsigned atomicExch(unsigned* p, unsigned v) { unsigned o = *p; *p = v; return o; }
inline double __drcp_rn(double x) { return 1.0 / x; }
inline float __frcp_rn(float x) { return 1.0f / x; }
inline size_t __cvta_generic_to_shared(const void* p) { return (size_t)p; }
