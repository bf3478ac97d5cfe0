// k_paths_sum_pyr_batch.cu -- pyramid-level instantiations of the one-volume aggregation for batches.
#include "k_paths_sum.cuh"

namespace pg {

template cudaError_t launch_paths_sum<true, kBatchJobs>(const Jobs<kBatchJobs>&, const LevelExtent&, cudaStream_t);

}  // namespace pg
