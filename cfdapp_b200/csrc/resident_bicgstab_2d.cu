// The 2D instantiations of the on-chip BiCGSTAB.
#include "resident_bicgstab_impl.cuh"

namespace cfdb {
namespace res {
template int bicgstab_cluster_limit<2>();
template cudaError_t launch_bicgstab<2, false>(cfdb_context*, const BandOp<2>&, const Plan&, uint32_t,
                              const GridWords&, const Io&);
template cudaError_t launch_bicgstab<2, true>(cfdb_context*, const BandOp<2>&, const Plan&, uint32_t,
                              const GridWords&, const Io&);
}  // namespace res
}  // namespace cfdb
