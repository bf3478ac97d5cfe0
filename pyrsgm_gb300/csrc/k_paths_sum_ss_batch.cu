// k_paths_sum_ss_batch.cu -- single-scale instantiations of the one-volume aggregation for batches.
#include "k_paths_sum.cuh"

namespace pg {

template cudaError_t launch_paths_sum<false, kBatchJobs>(const Jobs<kBatchJobs>&, const LevelExtent&, cudaStream_t);

}  // namespace pg
