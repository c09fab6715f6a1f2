// The 3D instantiations of the on-chip CG over band coefficients.
#include "resident_cg_impl.cuh"

namespace cfdb {
namespace res {
template int cg_cluster_limit<3>();
template cudaError_t launch_cg<3>(cfdb_context*, const BandOp<3>&, const Plan&, uint32_t,
                              const GridWords&, const Io&);
}  // namespace res
}  // namespace cfdb
