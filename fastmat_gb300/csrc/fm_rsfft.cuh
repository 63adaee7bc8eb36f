// Register-resident FFT of strided complex vectors: a Fourier factor of a
// Kron applied mode-wise (fastmat/Kron.pyx:284-300 with the transform of
// fastmat/Fourier.pyx), i.e. vectors of L points at an element stride S
// that is a multiple of 32, adjacent vectors adjacent in memory.
//
//   * the lanes take NV adjacent vectors (NV = 32, or fewer for long
//     vectors: NV G <= 256 threads), so each load and store of a warp covers
//     contiguous row segments of 128 bytes or more;
//   * vector v's L points are held by G = L / P threads (P = 16 complex64 or
//     8 double-float complex per thread), thread t of the vector holding
//     points t + G r, exactly the natural-order layout of the register
//     convolution (fm_rconv.cuh), whose radix stages run here unchanged:
//     the in-place DIF over the radices (P, P, ..., rest), twiddles from
//     lane-major tables in shared memory, exchanges between the stages
//     through a buffer per vector (odd stride: the lanes of each wavefront
//     on distinct banks; CTA barriers, the threads of a vector sit in
//     different warps);
//   * the results leave in natural order: each register's digit-reversed
//     position is mapped back at compile time, and the store of a point
//     goes to its row for all NV vectors at once.
// Double-float vectors are scaled by the power of two of their largest
// exponent on the way in (float's exponent range) and back on the way out.
#pragma once

#include "fm_rconv.cuh"

namespace fmk {

struct RsfStep {
  const void *src;
  void *dst;
  i64 ld_src, ld_dst;
  i64 A;   // vectors per column (a S + c: block a, offset c < S)
  i64 es;  // element stride S
  i64 num_cols;
  const void *tw;  // tw[j] = exp(-2 pi i j / L), j < L
  int *err;
  int L;
  int sign;  // -1 forward, +1 inverse (unscaled)
};

#define FM_RSF_THREADS 256
template <class E, int L> struct RsfShape {
  static constexpr int P = RcLane<E>::P;
  static constexpr int G = L / P;  // threads per vector
  static constexpr int NV = FM_RSF_THREADS / G > 32 ? 32
                                                    : FM_RSF_THREADS / G;
  static constexpr int T = NV * G;
  static constexpr int Lx = (L + (L >> RcBuf<E, L>::SH)) | 1;
};
template <class E> struct RsfOcc {
  static constexpr int v = sizeof(E) == 8 ? 3 : 2;
};
// double-float copies the next batch ahead into shared memory while the
// current one transforms (its two CTAs per SM leave the load latency
// uncovered: FFT(256) at stride 32768 on 8 columns 710 -> 615 us, 628 with
// the wider conversions); complex64,
// at 0.93 of the copy peak, loads straight into registers
template <class E> struct RsfAhead { static constexpr bool v = Emu<E>::v; };
template <class E, int L>
__host__ __device__ constexpr size_t rsf_smem() {
  return (size_t)(rc_twlen<E, L, rc_stages(L, RcLane<E>::P)>() +
                  RsfShape<E, L>::NV * RsfShape<E, L>::Lx +
                  (RsfAhead<E>::v ? RsfShape<E, L>::NV * L : 0)) *
             sizeof(E) +
         32 * sizeof(int);
}

template <class E, int L, int SG>
__global__ void __launch_bounds__(RsfShape<E, L>::T, (RsfOcc<E>::v))
    rsfft_kernel(const __grid_constant__ RsfStep p) {
  typedef RsfShape<E, L> Sh;
  constexpr int P = Sh::P, G = Sh::G, NV = Sh::NV;
  constexpr int S = rc_stages(L, P);
  static_assert(G >= 2 && NV >= 1 && NV <= 32, "vector layout");
  typedef typename std::conditional<Emu<E>::v, double2, float2>::type Raw;
  extern __shared__ __align__(128) unsigned char fm_smem[];
  constexpr int TWN = rc_twlen<E, L, S>();
  E *stw = reinterpret_cast<E *>(fm_smem);
  E *xb = stw + TWN;
  constexpr bool ahead = RsfAhead<E>::v;
  // thread-private slots of the next batch's points
  Raw *const slot =
      reinterpret_cast<Raw *>(xb + NV * Sh::Lx) + threadIdx.x;
  int *sexp =
      reinterpret_cast<int *>(xb + NV * Sh::Lx + (ahead ? NV * L : 0));
  rc_fill_tw<E, L, 0>(stw, p.tw);
  __syncthreads();
  const int v = threadIdx.x % NV, t = threadIdx.x / NV;
  E *buf = xb + v * Sh::Lx;
  const i64 Sx = p.es;
  const i64 nb = p.A * p.num_cols / NV;  // batches of NV adjacent vectors
  const FDiv dA((unsigned)p.A), dS((unsigned)Sx);
  // column and row of point 0 of this thread's vector in batch bt
  auto where = [&](i64 bt, unsigned &m) {
    const unsigned gv = (unsigned)(bt * NV);
    m = dA.div(gv);
    const unsigned v0 = gv - m * (unsigned)p.A;
    const unsigned a = dS.div(v0), c0 = v0 - a * (unsigned)Sx;
    return (i64)a * L * Sx + c0 + v;
  };
  auto prefetch = [&](i64 bt) {
    unsigned m;
    const i64 row0 = where(bt, m);
    const Raw *q = (const Raw *)p.src + (i64)m * p.ld_src + row0 + (i64)t * Sx;
#pragma unroll
    for (int r = 0; r < P; ++r, q += G * Sx)
      cp_async<sizeof(Raw)>(slot + Sh::T * r, q, true);
    cp_async_commit();
  };
  if (ahead && blockIdx.x < nb) prefetch(blockIdx.x);
  for (i64 bt = blockIdx.x; bt < nb; bt += gridDim.x) {
    unsigned m;
    const i64 row0 = where(bt, m);
    Raw d[P];
    if constexpr (ahead) {
      cp_async_wait<0>();
      __syncwarp();
#pragma unroll
      for (int r = 0; r < P; ++r) d[r] = slot[Sh::T * r];
      __syncwarp();
      if (bt + gridDim.x < nb) prefetch(bt + gridDim.x);
    } else {
      const Raw *q = (const Raw *)p.src + (i64)m * p.ld_src + row0 +
                     (i64)t * Sx;
#pragma unroll
      for (int r = 0; r < P; ++r, q += G * Sx) d[r] = *q;
    }
    E x[P];
    int s = 0;
    if constexpr (Emu<E>::v) {
      const int emax = rx_max<P>(d);
      if (threadIdx.x < NV) sexp[threadIdx.x] = 0;
      __syncthreads();
      if (emax > 0) atomicMax(sexp + v, emax);
      __syncthreads();
      s = df_scale<false>(sexp[v] >> 20);
      rx_in<false>(x, d, s);
    } else {
#pragma unroll
      for (int r = 0; r < P; ++r) x[r] = E{d[r].x, d[r].y};
    }
    // (S >= 2: the stages hold at least one exchange, whose barriers also
    // separate this batch's reads of sexp from the next batch's reset)
    rc_forward<E, L, 0, SG, 1>(x, buf, t, stw);
    // register u R + r of the last stage (radix R) holds the natural index
    // of the thread's base plus u R + r L / R
    constexpr int R = rc_radix(S - 1, L, P);
    Raw *dst = (Raw *)p.dst + (i64)m * p.ld_dst + row0 +
               (i64)rc_nat<E, L>(rc_base<E, L, S - 1>(t)) * Sx;
    rx_out<P>(x, s, [&](int j, Raw y) {
      dst[((i64)((j / R) * R) + (j % R) * (L / R)) * Sx] = y;
    });
  }
}

}  // namespace fmk
