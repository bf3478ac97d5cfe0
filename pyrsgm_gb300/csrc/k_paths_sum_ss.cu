// k_paths_sum_ss.cu -- single-scale instantiations of the one-volume aggregation.
#include "k_paths_sum.cuh"

namespace pg {

template cudaError_t launch_paths_sum<false, 1>(const Jobs<1>&, const LevelExtent&, cudaStream_t);

}  // namespace pg
