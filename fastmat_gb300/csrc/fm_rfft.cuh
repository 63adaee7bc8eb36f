// Register transforms of long complex vectors (complex64 and packed
// double-float): the passes of four-step transforms and convolutions of
// whole columns, i.e. fastmat's Fourier, Circulant and Toeplitz (and the
// chirp form of any length) above the lengths one warp holds
// (fastmat/Fourier.pyx, fastmat/Circulant.pyx:127-133,
// fastmat/Toeplitz.pyx:255-268).
//
// A vector's L points sit in the registers of G = L / P threads (P = 8
// per thread, thread t holding points t + G r),
// and the radix stages, exchanges and digit order are those of the register
// convolution (fm_rconv.cuh), with CTA barriers where a vector spans several
// warps.  Two mappings:
//
//   rxfft_kernel: one FFT; the lanes take NV adjacent vectors, so the loads
//     and stores of strided vectors are row segments of 64 bytes or more
//     (contiguous input vectors come in coalesced along their points and
//     turn through the exchange buffer, for the transposing second pass of
//     a long Fourier); optional four-step twiddle on the results;
//   rxconv_kernel: FFT, spectrum product (one spectrum per vector of the
//     column or one for all), inverse FFT on contiguous vectors, the lanes
//     along a vector's points; optional four-step twiddle.
//
// Both read and write any I/O type, apply the loader's gather, conjugation
// and product and the storer's product, scalar, conjugation, scatter and
// accumulation, and clip to the rows that exist.  An inverse FFT is the
// conjugate of the forward FFT of the conjugate: the host folds that into
// the conjugation flags.  The stage twiddles, spectra and four-step twiddles
// are tables in the kernels' own element type, in the order the lanes read
// them (consecutive lanes, consecutive entries).
//
// Measured against the stage kernel's tiles (vprog_kernel, every radix stage
// a pass over shared memory with run-time index arithmetic), microseconds
// per launch: 32 columns of 2^18 points, double-float, strided 512 points
// 347 -> 132 (with gathers and products around), convolution of 512 points
// 558 -> 207 (185 before products were normalised and heads rounded); the
// same in complex64 118 -> 35 and 62 -> 43; convolution of 4096 points, 4
// columns, double-float 57 -> 22.  Eight points a thread in
// complex64 too: 16 (the radices 16, 16, 2) measured 6 % further from 64-bit
// results over 2^18 points, and spilled in the convolution.  The next batch
// is copied ahead (strided complex64 38 -> 35, gathered double-float 168 ->
// 134).  Bounds: the FMA pipe in double-float (66 % busy in the convolution,
// 46 to 50 % in the FFT passes, whose table loads and barriers 16 warps a
// multiprocessor do not cover), the shared-memory / L1 pipe in complex64 (50
// to 69 %).  Measured and left out, in double-float: intermediates as packed
// double-floats instead of float64 words (no change: the conversions run in
// the integer pipe's spare cycles), half the vectors a CTA (2^18 x 32 chain
// 463 -> 478 us), 96 registers a thread (convolution 185 -> 196), barriers
// per vector (185 -> 188).
#pragma once

#include <map>
#include <mutex>

#include "fm_rconv.cuh"

namespace fmk {

struct RxStep {
  const void *src;
  void *dst;
  i64 ld_src, ld_dst;
  int src_type, dst_type;
  i64 V;                // vectors per column
  i64 in_n, in_cc;      // input view: vector v = a cc + c has point j at
  i64 out_n, out_cc;    // row (a n + j) cc + c
  i64 in_rows, out_rows;  // rows that exist / are written
  i64 num_cols;
  const i64 *map_in, *map_out;  // gather of the loader, scatter of the storer
  const void *pre, *post;  // products of the loader / storer, by row
  const void *spec;     // conv: spectra in the order of the last forward
  i64 spec_stride;      // stage's registers (j G + g), per vector or 0
  const void *tw;       // stage twiddle tables (rc_twoff)
  const void *wtab;     // four-step twiddle of point j of vector v at
  i64 wq, wj;           // v wq + j wj
  int in_len, out_len;
  int pre_by_point, post_by_point;  // products by point instead of row
  int conj_in, conj_out, pre_conj, post_conj, spec_conj, w_conj;
  int has_scale, accumulate;
  double scale_re, scale_im;
  int L;
};

constexpr int kRxP = 8;  // points per thread
template <class E, int L> struct RxShape {
  static constexpr int P = RcLane<E>::P;
  static_assert(P == kRxP, "points per thread");
  static constexpr int G = L / P;
  // rxfft: adjacent vectors per CTA (row segments of at least 64 bytes up
  // to 512 points), and the stride of their exchange buffers: the lanes of
  // one shared-memory phase (128 bytes) are NV vectors times 1 or more
  // consecutive threads, which this stride puts on distinct banks
  static constexpr int NVmin = 64 / (int)sizeof(E);
  static constexpr int NV0 = 256 / G;
  static constexpr int NV1 = NV0 > 32 ? 32 : NV0 < NVmin ? NVmin : NV0;
  static constexpr int NV = NV1 * G > 512 ? 512 / G : NV1;
  static constexpr int TF = NV * G;
  static constexpr int EP = 128 / (int)sizeof(E);
  static constexpr int Lb = L + (L >> RcBuf<E, L>::SH);
  static constexpr int Lx = NV >= EP ? (Lb | 1) : Lb + EP / NV;
  // rxconv: vectors per CTA
  static constexpr int TC = G > 128 ? G : 128;
  static constexpr int VPC = TC / G;
  static constexpr int Lc = RcBuf<E, L>::Lp;
};
// threads per SM the register budget aims at: 128 registers a thread in
// double-float; complex64 64 for one FFT, 80 for the convolution
template <class E, bool CONV> struct RxTPS {
  static constexpr int v = sizeof(E) != 8 ? 512 : CONV ? 768 : 1024;
};
template <class E, int L>
__host__ __device__ constexpr size_t rxfft_smem() {
  typedef RxShape<E, L> S;
  return (size_t)2 * S::NV * S::Lx * sizeof(E) + 32 * sizeof(int);
}
template <class E, int L>
__host__ __device__ constexpr size_t rxconv_smem() {
  typedef RxShape<E, L> S;
  return (size_t)S::VPC * (S::Lc + L) * sizeof(E) + S::VPC * sizeof(int);
}

template <class E> struct RxRaw {
  typedef typename std::conditional<Emu<E>::v, double2, float2>::type type;
};
// conjugation of raw words by a sign mask (0 or 0x80000000)
__device__ __forceinline__ double2 rx_conj(double2 v, unsigned m) {
  v.y = __hiloint2double((int)((unsigned)__double2hiint(v.y) ^ m),
                         __double2loint(v.y));
  return v;
}
__device__ __forceinline__ float2 rx_conj(float2 v, unsigned m) {
  v.y = __int_as_float((int)((unsigned)__float_as_int(v.y) ^ m));
  return v;
}
__device__ __forceinline__ double2 rx_zero(double2) {
  return make_double2(0., 0.);
}
__device__ __forceinline__ float2 rx_zero(float2) {
  return make_float2(0.f, 0.f);
}

// P points j0 + dj r of one vector of the input view (row of point 0: rb,
// column offset col) from any type, zero outside the vector or the column
template <class E, int L>
__device__ __forceinline__ void rx_load(
    typename RxRaw<E>::type (&d)[RcLane<E>::P], const RxStep &p, bool act,
    i64 col, i64 rb, int j0, int dj) {
  typedef typename RxRaw<E>::type Raw;
  constexpr int P = RcLane<E>::P;
  const i64 cc = p.in_cc;
#pragma unroll
  for (int r = 0; r < P; ++r) {
    const int j = j0 + dj * r;
    const i64 row = rb + (i64)j * cc;
    Raw v = rx_zero(Raw());
    if (act && j < p.in_len && row < p.in_rows) {
      const i64 srow = p.map_in ? p.map_in[row] : row;
      if (srow >= 0) v = load_as<Raw>(p.src, p.src_type, col + srow);
    }
    d[r] = v;
  }
  const unsigned m = p.conj_in ? 0x80000000u : 0u;
#pragma unroll
  for (int r = 0; r < P; ++r) d[r] = rx_conj(d[r], m);
}

// copy points j0 + dj r of one vector ahead into shared memory (dst + ds r),
// zeros outside the vector or the column and where the gather has none;
// buffers already in the kernel's type only
template <class E, int L>
__device__ __forceinline__ void rx_ahead(const RxStep &p, bool act, i64 col,
                                         i64 rb, int j0, int dj,
                                         typename RxRaw<E>::type *dst,
                                         int ds) {
  typedef typename RxRaw<E>::type Raw;
  constexpr int P = RcLane<E>::P;
  const i64 cc = p.in_cc;
  const Raw *q = (const Raw *)p.src + col + rb + (i64)j0 * cc;
  const i64 step = (i64)dj * cc;
  if (p.map_in) {
    i64 row[P];
#pragma unroll
    for (int r = 0; r < P; ++r) {
      const int j = j0 + dj * r;
      const i64 k = rb + (i64)j * cc;
      row[r] = act && j < p.in_len && k < p.in_rows ? p.map_in[k] : -1;
    }
#pragma unroll
    for (int r = 0; r < P; ++r)
      cp_async<sizeof(Raw)>(
          dst + ds * r,
          row[r] >= 0 ? (const void *)((const Raw *)p.src + col + row[r])
                      : p.src,
          row[r] >= 0);
  } else if (act && p.in_len == L && rb + (L - 1) * cc < p.in_rows) {
#pragma unroll
    for (int r = 0; r < P; ++r)
      cp_async<sizeof(Raw)>(dst + ds * r, q + r * step, true);
  } else {
#pragma unroll
    for (int r = 0; r < P; ++r) {
      const int j = j0 + dj * r;
      const bool ok = act && j < p.in_len && rb + (i64)j * cc < p.in_rows;
      cp_async<sizeof(Raw)>(dst + ds * r,
                            ok ? (const void *)(q + r * step) : p.src, ok);
    }
  }
}

// the loader's product on points j0 + dj r
template <class E, int L>
__device__ __forceinline__ void rx_pre(E (&x)[RcLane<E>::P], const RxStep &p,
                                       bool act, i64 rb, int j0, int dj) {
  if (!p.pre || !act) return;
#pragma unroll
  for (int r = 0; r < RcLane<E>::P; ++r) {
    const int j = j0 + dj * r;
    const i64 row = rb + (i64)j * p.in_cc;
    if (j < p.in_len && row < p.in_rows)
      x[r] = mulv(x[r], tab_get<E>(p.pre, p.pre_by_point ? (i64)j : row),
                  p.pre_conj != 0);
  }
}

// registers to the output view: register r holds point j0 + jo(r)
// (RAW: plain stores in the kernel's own type, no scalar)
template <class E, int L, bool RAW = false, class JO>
__device__ __forceinline__ void rx_store(E (&x)[RcLane<E>::P], int s,
                                         const RxStep &p, i64 v, i64 col,
                                         i64 rb, int j0, JO jo) {
  typedef typename RxRaw<E>::type Raw;
  constexpr int P = RcLane<E>::P;
  const i64 cc = p.out_cc;
  if (p.wtab) {
    const E *w = (const E *)p.wtab + v * p.wq + (i64)j0 * p.wj;
#pragma unroll
    for (int r = 0; r < P; ++r) {
      const E f = tw_get<true>(w + (i64)jo(r) * p.wj, 0);
      x[r] = mulv(x[r], f, p.w_conj != 0);
    }
  }
  if (p.post) {
#pragma unroll
    for (int r = 0; r < P; ++r) {
      const int j = j0 + jo(r);
      const i64 row = rb + (i64)j * cc;
      if (j < p.out_len && row < p.out_rows)
        x[r] = mulv(x[r], tab_get<E>(p.post, p.post_by_point ? (i64)j : row),
                    p.post_conj != 0);
    }
  }
  if (!RAW && p.has_scale) {
    const E c = scalar_of<E>(p.scale_re, p.scale_im);
#pragma unroll
    for (int r = 0; r < P; ++r) x[r] = mulv(x[r], c, false);
  }
  if (RAW || (p.dst_type == Tr<E>::code && !p.accumulate)) {
    const unsigned m = p.conj_out ? 0x80000000u : 0u;
    Raw *const dst = (Raw *)p.dst + col;
    if (p.map_out) {
      rx_out<P>(x, s, [&](int r, Raw y) {
        const int j = j0 + jo(r);
        const i64 row = rb + (i64)j * cc;
        const i64 drow =
            j < p.out_len && row < p.out_rows ? p.map_out[row] : -1;
        if (drow >= 0) dst[drow] = rx_conj(y, m);
      });
      return;
    }
    Raw *q = dst + rb + (i64)j0 * cc;
    if (p.out_len == L && rb + (L - 1) * cc < p.out_rows) {
      rx_out<P>(x, s, [&](int r, Raw y) {
        q[(i64)jo(r) * cc] = rx_conj(y, m);
      });
    } else {
      rx_out<P>(x, s, [&](int r, Raw y) {
        const int j = j0 + jo(r);
        if (j < p.out_len && rb + (i64)j * cc < p.out_rows)
          q[(i64)jo(r) * cc] = rx_conj(y, m);
      });
    }
    return;
  }
  if constexpr (!RAW) {
#pragma unroll
    for (int r = 0; r < P; ++r) {
      const int j = j0 + jo(r);
      const i64 row = rb + (i64)j * cc;
      if (j >= p.out_len || row >= p.out_rows) continue;
      const i64 drow = p.map_out ? p.map_out[row] : row;
      if (drow < 0) continue;
      store_elem<E>(p.dst, p.dst_type, col + drow,
                    p.conj_out ? conjv(x[r]) : x[r], p.accumulate != 0, s);
    }
  }
}

template <class E, int L>
__global__ void __launch_bounds__(RxShape<E, L>::TF,
                                  RxTPS<E, false>::v / RxShape<E, L>::TF)
    rxfft_kernel(const __grid_constant__ RxStep p) {
  typedef RxShape<E, L> Sh;
  typedef typename RxRaw<E>::type Raw;
  constexpr int P = Sh::P, G = Sh::G, NV = Sh::NV, T = Sh::TF;
  constexpr int S = rc_stages(L, P);
  constexpr int R = rc_radix(S - 1, L, P);
  static_assert(S >= 2 && T <= 512 && T * P == NV * L, "vector layout");
  extern __shared__ __align__(128) unsigned char fm_smem[];
  E *xb = reinterpret_cast<E *>(fm_smem);
  Raw *slot = reinterpret_cast<Raw *>(xb + NV * Sh::Lx);  // the next batch
  int *sexp = reinterpret_cast<int *>(slot + NV * Sh::Lx);
  const int lane = threadIdx.x % NV, t = threadIdx.x / NV;
  E *buf = xb + lane * Sh::Lx;
  const unsigned nbc = (unsigned)((p.V + NV - 1) / NV);  // batches per column
  const unsigned nb = nbc * (unsigned)p.num_cols;
  const FDiv dB(nbc), dI((unsigned)p.in_cc), dO((unsigned)p.out_cc);
  const int jn = rc_nat<E, L>(rc_base<E, L, S - 1>(t));
  // contiguous vectors are loaded along their points (thread k takes point
  // k + T i of the batch's NV L points) and turned on the way through shared
  // memory; strided ones by the thread that uses them
  const bool turn = p.in_cc == 1;
  const bool ahead = p.src_type == Tr<E>::code && !(turn && p.map_in);
  auto prefetch = [&](unsigned bt) {
    const unsigned m = dB.div(bt), v0 = (bt - m * nbc) * NV;
    const i64 col = (i64)m * p.ld_src;
    if (turn) {
#pragma unroll
      for (int i = 0; i < P; ++i) {
        const int k = threadIdx.x + T * i, vv = k / L, j = k % L;
        const i64 row = (i64)(v0 + vv) * p.in_n + j;
        const bool ok = v0 + vv < p.V && j < p.in_len && row < p.in_rows;
        cp_async<sizeof(Raw)>(
            slot + vv * Sh::Lx + rc_pad<E, L>(j),
            ok ? (const void *)((const Raw *)p.src + col + row) : p.src, ok);
      }
    } else {
      const unsigned v = v0 + lane;
      const unsigned a = dI.div(v), c = v - a * (unsigned)p.in_cc;
      rx_ahead<E, L>(p, v < p.V, col, (i64)a * p.in_n * p.in_cc + c, t, G,
                     slot + threadIdx.x, T);
    }
    cp_async_commit();
  };
  if (ahead && blockIdx.x < nb) prefetch(blockIdx.x);
  for (unsigned bt = blockIdx.x; bt < nb; bt += gridDim.x) {
    const unsigned m = dB.div(bt), v0 = (bt - m * nbc) * NV;
    const unsigned v = v0 + lane;
    const bool act = v < p.V;
    const unsigned a = dI.div(v), c = v - a * (unsigned)p.in_cc;
    const i64 rb = (i64)a * p.in_n * p.in_cc + c;
    const i64 col = (i64)m * p.ld_src;
    Raw d[P];
    if (turn) {
      if (ahead) {
        cp_async_wait<0>();
      } else {
#pragma unroll
        for (int i = 0; i < P; ++i) {
          const int k = threadIdx.x + T * i, vv = k / L, j = k % L;
          const i64 rv = (i64)(v0 + vv) * p.in_n;
          Raw y = rx_zero(Raw());
          if (v0 + vv < p.V && j < p.in_len && rv + j < p.in_rows) {
            const i64 srow = p.map_in ? p.map_in[rv + j] : rv + j;
            if (srow >= 0) y = load_as<Raw>(p.src, p.src_type, col + srow);
          }
          slot[vv * Sh::Lx + rc_pad<E, L>(j)] = y;
        }
      }
      __syncthreads();
      // (t < G, so t and G r occupy disjoint bits)
      const Raw *rr = slot + lane * Sh::Lx + rc_pad<E, L>(t);
      const unsigned mask = p.conj_in ? 0x80000000u : 0u;
#pragma unroll
      for (int r = 0; r < P; ++r)
        d[r] = rx_conj(rr[rc_pad<E, L>(G * r)], mask);
      __syncthreads();
    } else if (ahead) {
      cp_async_wait<0>();
      __syncwarp();
      const unsigned mask = p.conj_in ? 0x80000000u : 0u;
#pragma unroll
      for (int r = 0; r < P; ++r)
        d[r] = rx_conj(slot[threadIdx.x + T * r], mask);
      __syncwarp();
    } else {
      rx_load<E, L>(d, p, act, col, rb, t, G);
    }
    if (ahead && bt + gridDim.x < nb) prefetch(bt + gridDim.x);
    E x[P];
    int s = 0;
    if constexpr (Emu<E>::v) {
      const int emax = rx_max<P>(d);
      if (threadIdx.x < NV) sexp[threadIdx.x] = 0;
      __syncthreads();
      if (emax > 0) atomicMax(sexp + lane, emax);
      __syncthreads();
      s = df_scale<true>(sexp[lane] >> 20);
      rx_in<true>(x, d, s);
    } else {
#pragma unroll
      for (int r = 0; r < P; ++r) x[r] = E{d[r].x, d[r].y};
    }
    rx_pre<E, L>(x, p, act, rb, t, G);
    // (S >= 2: the exchanges' barriers also separate this batch's reads of
    // sexp from the next batch's reset)
    rc_forward<E, L, 0, -1, 1, true>(x, buf, t, (const E *)p.tw);
    if (act) {
      const unsigned ao = dO.div(v), co = v - ao * (unsigned)p.out_cc;
      // register u R + r holds natural index jn + u R + r L / R
      rx_store<E, L>(x, s, p, v, (i64)m * p.ld_dst,
                     (i64)ao * p.out_n * p.out_cc + co, jn, [](int j) {
                       return (j / R) * R + (j % R) * (L / R);
                     });
    }
  }
}

template <class E, int L>
__global__ void __launch_bounds__(RxShape<E, L>::TC,
                                  RxTPS<E, true>::v / RxShape<E, L>::TC)
    rxconv_kernel(const __grid_constant__ RxStep p) {
  typedef RxShape<E, L> Sh;
  typedef typename RxRaw<E>::type Raw;
  constexpr int P = Sh::P, G = Sh::G, VPC = Sh::VPC;
  constexpr int S = rc_stages(L, P);
  constexpr bool CTA = G > 32;
  static_assert(S >= 2 && Sh::TC <= 512, "vector layout");
  extern __shared__ __align__(128) unsigned char fm_smem[];
  E *xb = reinterpret_cast<E *>(fm_smem);
  Raw *slot = reinterpret_cast<Raw *>(xb + VPC * Sh::Lc) + threadIdx.x;
  int *sexp = reinterpret_cast<int *>(fm_smem) +
              VPC * (Sh::Lc + L) * (sizeof(E) / sizeof(int));
  const int q = threadIdx.x / G, g = threadIdx.x % G;
  E *buf = xb + q * Sh::Lc;
  const unsigned NV = (unsigned)(p.V * p.num_cols);
  const FDiv dV((unsigned)p.V);
  // the next batch's points, copied ahead by the threads that use them
  const bool ahead = p.src_type == Tr<E>::code;
  auto prefetch = [&](unsigned vb) {
    const unsigned gv = vb + q;
    const unsigned m = dV.div(gv), v = gv - m * (unsigned)p.V;
    rx_ahead<E, L>(p, gv < NV, (i64)m * p.ld_src, (i64)v * p.in_n, g, G,
                   slot, Sh::TC);
    cp_async_commit();
  };
  if (ahead && blockIdx.x * VPC < NV) prefetch(blockIdx.x * VPC);
  for (unsigned vb = blockIdx.x * VPC; vb < NV; vb += gridDim.x * VPC) {
    const unsigned gv = vb + q;
    const bool act = gv < NV;
    const unsigned m = dV.div(gv), v = gv - m * (unsigned)p.V;
    const i64 rb = (i64)v * p.in_n;
    Raw d[P];
    if (ahead) {
      cp_async_wait<0>();
      __syncwarp();
      const unsigned mask = p.conj_in ? 0x80000000u : 0u;
#pragma unroll
      for (int r = 0; r < P; ++r) d[r] = rx_conj(slot[Sh::TC * r], mask);
      __syncwarp();
      const unsigned nx = vb + gridDim.x * VPC;
      if (nx < NV) prefetch(nx);
    } else {
      rx_load<E, L>(d, p, act, (i64)m * p.ld_src, rb, g, G);
    }
    E x[P];
    int s = 0;
    if constexpr (Emu<E>::v) {
      int emax = rx_max<P>(d);
      constexpr int WV = G < 32 ? G : 32;
#pragma unroll
      for (int o = WV / 2; o >= 1; o /= 2)
        emax = max(emax, __shfl_xor_sync(0xffffffffu, emax, o, WV));
      if constexpr (CTA) {
        if (g == 0) sexp[q] = 0;
        __syncthreads();
        if (g % WV == 0 && emax > 0) atomicMax(sexp + q, emax);
        __syncthreads();
        emax = sexp[q];
      }
      s = df_scale<true>(emax >> 20);
      rx_in<true>(x, d, s);
    } else {
#pragma unroll
      for (int r = 0; r < P; ++r) x[r] = E{d[r].x, d[r].y};
    }
    rx_pre<E, L>(x, p, act, rb, g, G);
    rc_forward<E, L, 0, -1, CTA ? 1 : 0, true>(x, buf, g, (const E *)p.tw);
    if (act) {
      const E *sp = (const E *)p.spec + (i64)v * p.spec_stride + g;
#pragma unroll
      for (int j = 0; j < P; ++j)
        x[j] = mulv(x[j], tw_get<true>(sp, j * G), p.spec_conj != 0);
    }
    rc_inverse<E, L, S - 1, CTA ? 1 : 0, true>(x, buf, g, (const E *)p.tw);
    if (act)
      rx_store<E, L>(x, s, p, v, (i64)m * p.ld_dst, (i64)v * p.out_n, g,
                     [](int r) { return G * r; });
  }
}

// one kernel's CTA count: the work, at most one resident grid
template <class K>
cudaError_t rx_launch(K fn, int threads, size_t smem, i64 want,
                      std::map<int, int> &resident, std::mutex &mu,
                      const RxStep &p, cudaStream_t s) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  i64 cap = 0;
  {
    std::lock_guard<std::mutex> lock(mu);
    auto it = resident.find(dev);
    if (it == resident.end()) {
      e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)smem);
      if (e != cudaSuccess) return e;
      int per_sm = 0, sms = 0;
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads,
                                                        smem);
      if (e != cudaSuccess) return e;
      e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
      if (e != cudaSuccess) return e;
      it = resident.emplace(dev, (per_sm < 1 ? 1 : per_sm) * sms).first;
    }
    cap = it->second;
  }
  const i64 grid = want > cap ? cap : want < 1 ? 1 : want;
  fn<<<(unsigned)grid, threads, smem, s>>>(p);
  return cudaGetLastError();
}
template <class E, int L>
cudaError_t rxfft_one(const RxStep &p, cudaStream_t s) {
  typedef RxShape<E, L> S;
  static std::mutex mu;
  static std::map<int, int> resident;
  return rx_launch(rxfft_kernel<E, L>, S::TF, rxfft_smem<E, L>(),
                   (p.V + S::NV - 1) / S::NV * p.num_cols, resident, mu, p,
                   s);
}
template <class E, int L>
cudaError_t rxconv_one(const RxStep &p, cudaStream_t s) {
  typedef RxShape<E, L> S;
  static std::mutex mu;
  static std::map<int, int> resident;
  return rx_launch(rxconv_kernel<E, L>, S::TC, rxconv_smem<E, L>(),
                   (p.V * p.num_cols + S::VPC - 1) / S::VPC, resident, mu, p,
                   s);
}

}  // namespace fmk
