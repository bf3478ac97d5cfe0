// k_paths_sum_pyr.cu -- pyramid-level instantiations of the one-volume aggregation.
#include "k_paths_sum.cuh"

namespace pg {

template cudaError_t launch_paths_sum<true, 1>(const Jobs<1>&, const LevelExtent&, cudaStream_t);

}  // namespace pg
