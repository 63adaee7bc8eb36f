// Batched persistent kernel: complex64, power-of-two FFTs and pointwise work.
#include "fm_batch_launch.cuh"

namespace fmk {

cudaError_t launch_batch_c64_pow2(const BatchLaunch &b, cudaStream_t s) {
  return launch_batch_one<float2, 1>(b, s);
}

}  // namespace fmk
