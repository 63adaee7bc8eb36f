// Batched persistent kernel: double-float complex.
#include "fm_batch_launch.cuh"

namespace fmk {

cudaError_t launch_batch_df(const BatchLaunch &b, cudaStream_t s) {
  return launch_batch_one<dfc, 0>(b, s);
}

}  // namespace fmk
