// Instantiations and launcher of rxfft_kernel (fm_rfft.cuh): packed
// double-float.
#include "fm_launch.cuh"
#include "fm_rfft.cuh"

namespace fmk {

cudaError_t launch_rxfft_df(const RxStep &p, cudaStream_t s) {
  switch (p.L) {
    case 32: return rxfft_one<dfq, 32>(p, s);
    case 64: return rxfft_one<dfq, 64>(p, s);
    case 128: return rxfft_one<dfq, 128>(p, s);
    case 256: return rxfft_one<dfq, 256>(p, s);
    case 512: return rxfft_one<dfq, 512>(p, s);
    case 1024: return rxfft_one<dfq, 1024>(p, s);
    default: return cudaErrorInvalidConfiguration;
  }
}

}  // namespace fmk
