// Instantiations and launcher of rxconv_kernel (fm_rfft.cuh): packed
// double-float.
#include "fm_launch.cuh"
#include "fm_rfft.cuh"

namespace fmk {

cudaError_t launch_rxconv_df(const RxStep &p, cudaStream_t s) {
  switch (p.L) {
    case 64: return rxconv_one<dfq, 64>(p, s);
    case 128: return rxconv_one<dfq, 128>(p, s);
    case 256: return rxconv_one<dfq, 256>(p, s);
    case 512: return rxconv_one<dfq, 512>(p, s);
    case 1024: return rxconv_one<dfq, 1024>(p, s);
    case 2048: return rxconv_one<dfq, 2048>(p, s);
    case 4096: return rxconv_one<dfq, 4096>(p, s);
    default: return cudaErrorInvalidConfiguration;
  }
}

}  // namespace fmk
