// The 3D mixed-precision instantiation of the on-chip Jacobi-PCG.
#include "resident_faces_impl.cuh"

namespace cfdb {
namespace res {
template cfdb_status pcg_on_chip<3, MIXED>(cfdb_context*, const OpView<double>&, const double*,
                                         const IoT<double>&);
}  // namespace res
}  // namespace cfdb
