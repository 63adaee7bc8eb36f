// Launcher of the batched persistent kernel (many operators in one
// cooperative launch; see batch_kernel in fm_batch.cuh).  The instantiations
// live in translation units of their own (fm_batch_c64_pow2.cu,
// fm_batch_c64.cu, fm_batch_c64_gen.cu, fm_batch_df.cu), which compile in
// parallel.

#include <cuda_runtime.h>

#include "../../include/fmgpu.h"
#include "fm_launch.cuh"

namespace fmk {

cudaError_t launch_batch_c64_pow2(const BatchLaunch &b, cudaStream_t s);
cudaError_t launch_batch_c64(const BatchLaunch &b, cudaStream_t s);
cudaError_t launch_batch_c64_gen(const BatchLaunch &b, cudaStream_t s);
cudaError_t launch_batch_df(const BatchLaunch &b, cudaStream_t s);

cudaError_t launch_batch(const BatchLaunch &b, cudaStream_t s) {
  switch (b.ctype) {
    case FM_C64:
      return b.cls == 1   ? launch_batch_c64_pow2(b, s)
             : b.cls == 2 ? launch_batch_c64(b, s)
                          : launch_batch_c64_gen(b, s);
    case FM_C128_DF: return launch_batch_df(b, s);
    default: return cudaErrorNotSupported;
  }
}

}  // namespace fmk
