// One step of iterative soft thresholding in a single pass (fastmat's ISTA
// and FISTA, fastmat/algorithms/ISTA.py:111-160,
// fastmat/algorithms/FISTA.py:120-180):
//
//   step = y - l g
//   x    = m / (m + alpha) step,  m = max(|step| - alpha, 0)
//   ynew = x + beta (x - xold)                          (FISTA's momentum)
//
// elementwise over `count` elements.  Evaluated as separate tensor
// operations the step is about 13 launches over the iterates, each shorter
// than its launch (FISTA on Circulant(4096), 4 complex128 columns: 130 us of
// a 208 us iteration between the two transforms); here it is one launch that
// reads three arrays and writes three, bound by its launch at such sizes
// and by HBM at large ones (96 bytes an element in complex128).

#include <cuda_runtime.h>

#include <algorithm>
#include <string>

#include "../../include/fmgpu.h"
#include "fm_launch.cuh"

namespace {

using i64 = long long;

__device__ __forceinline__ float mag(float a) { return fabsf(a); }
__device__ __forceinline__ double mag(double a) { return fabs(a); }
__device__ __forceinline__ float mag(float2 a) { return hypotf(a.x, a.y); }
__device__ __forceinline__ double mag(double2 a) { return hypot(a.x, a.y); }
__device__ __forceinline__ float mul(float s, float a) { return s * a; }
__device__ __forceinline__ double mul(double s, double a) { return s * a; }
__device__ __forceinline__ float2 mul(float s, float2 a) {
  return make_float2(s * a.x, s * a.y);
}
__device__ __forceinline__ double2 mul(double s, double2 a) {
  return make_double2(s * a.x, s * a.y);
}
__device__ __forceinline__ float add(float a, float b) { return a + b; }
__device__ __forceinline__ double add(double a, double b) { return a + b; }
__device__ __forceinline__ float2 add(float2 a, float2 b) {
  return make_float2(a.x + b.x, a.y + b.y);
}
__device__ __forceinline__ double2 add(double2 a, double2 b) {
  return make_double2(a.x + b.x, a.y + b.y);
}

template <class T, class R>
__global__ void __launch_bounds__(256)
    k_shrink_step(i64 count, const T *__restrict__ y, const T *__restrict__ g,
                  const T *__restrict__ xold, T *__restrict__ step,
                  T *__restrict__ x, T *__restrict__ ynew, R l, R alpha,
                  R beta) {
  for (i64 i = blockIdx.x * (i64)256 + threadIdx.x; i < count;
       i += (i64)gridDim.x * 256) {
    const T s = add(y[i], mul(-l, g[i]));
    R m = mag(s) - alpha;
    if (m < (R)0) m = (R)0;  // (NaN stays)
    const T v = mul(m / (m + alpha), s);
    step[i] = s;
    x[i] = v;
    if (ynew) ynew[i] = add(v, mul(beta, add(v, mul((R)-1, xold[i]))));
  }
}

template <class T, class R>
cudaError_t run(i64 count, const void *y, const void *g, const void *xold,
                void *step, void *x, void *ynew, double l, double alpha,
                double beta, cudaStream_t s) {
  const i64 blocks = std::min<i64>((count + 255) / 256, 152 * 8);
  k_shrink_step<T, R><<<(unsigned)blocks, 256, 0, s>>>(
      count, (const T *)y, (const T *)g, (const T *)xold, (T *)step, (T *)x,
      (T *)ynew, (R)l, (R)alpha, (R)beta);
  return cudaGetLastError();
}

}  // namespace

extern "C" int fm_shrink_step(int64_t count, int32_t type, const void *y,
                              const void *g, const void *xold, void *step,
                              void *x, void *ynew, double l, double alpha,
                              double beta, void *stream) {
  if (count < 0 || (count > 0 && (!y || !g || !step || !x ||
                                  (ynew && !xold)))) {
    fmk::set_last_error("fm_shrink_step: invalid count or NULL pointer");
    return FM_ERR_VALUE;
  }
  if (count == 0) return FM_OK;
  const cudaStream_t s = (cudaStream_t)stream;
  cudaError_t e;
  switch (type) {
    case FM_F32:
      e = run<float, float>(count, y, g, xold, step, x, ynew, l, alpha, beta,
                            s);
      break;
    case FM_F64:
      e = run<double, double>(count, y, g, xold, step, x, ynew, l, alpha,
                              beta, s);
      break;
    case FM_C64:
      e = run<float2, float>(count, y, g, xold, step, x, ynew, l, alpha, beta,
                             s);
      break;
    case FM_C128:
      e = run<double2, double>(count, y, g, xold, step, x, ynew, l, alpha,
                               beta, s);
      break;
    default:
      fmk::set_last_error("fm_shrink_step: unsupported element type");
      return FM_ERR_TYPE;
  }
  if (e != cudaSuccess) {
    fmk::set_last_error(cudaGetErrorString(e));
    return FM_ERR_CUDA;
  }
  return FM_OK;
}
