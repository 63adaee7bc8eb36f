// Batched persistent kernel: complex64, every program.
#include "fm_batch_launch.cuh"

namespace fmk {

cudaError_t launch_batch_c64_gen(const BatchLaunch &b, cudaStream_t s) {
  return launch_batch_one<float2, 0>(b, s);
}

}  // namespace fmk
