// Batched persistent kernel: complex64, FFTs of any radix and pointwise work.
#include "fm_batch_launch.cuh"

namespace fmk {

cudaError_t launch_batch_c64(const BatchLaunch &b, cudaStream_t s) {
  return launch_batch_one<float2, 2>(b, s);
}

}  // namespace fmk
