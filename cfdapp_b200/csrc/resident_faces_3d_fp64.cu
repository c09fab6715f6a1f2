// The 3D FP64 instantiation of the on-chip Jacobi-PCG.
#include "resident_faces_impl.cuh"

namespace cfdb {
namespace res {
template cfdb_status pcg_on_chip<3, FP64>(cfdb_context*, const OpView<double>&, const double*,
                                         const IoT<double>&);
}  // namespace res
}  // namespace cfdb
