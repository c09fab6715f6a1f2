// The 2D FP32 instantiation of the on-chip Jacobi-PCG.
#include "resident_faces_impl.cuh"

namespace cfdb {
namespace res {
template cfdb_status pcg_on_chip<2, FP32>(cfdb_context*, const OpView<float>&, const float*,
                                         const IoT<float>&);
}  // namespace res
}  // namespace cfdb
