// Launch of the on-chip Jacobi-PCG (resident_faces.cu), instantiated for one
// dimension and kind per translation unit: a process loads only the modules
// it runs.  With every variant in one module a process's first solve took
// 70 ms longer; with one of these it takes 5-9 ms longer than the next.
#pragma once

#include <cuda_runtime.h>

#include <type_traits>

#include "pcg_internal.cuh"
#include "resident_launch.cuh"

namespace cfdb {
namespace res {

enum { FP64 = 0, MIXED = 1, FP32 = 2 };
template <int KIND>
using Value = typename std::conditional<KIND == FP32, float, double>::type;

template <int DIM, int KIND>
cfdb_status pcg_on_chip(cfdb_context* ctx, const OpView<Value<KIND>>& V, const Value<KIND>* invd,
                        const IoT<Value<KIND>>& io);

}  // namespace res
}  // namespace cfdb
