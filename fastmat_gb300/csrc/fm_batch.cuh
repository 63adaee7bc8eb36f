// The batched persistent kernel (see the batch section of fm_vprog.cuh) and
// the register transforms it runs on tiles.
//
// The passes of long transforms carry nearly all bytes of a batch (30.8 M of
// 34.6 M element passes for 64 Circulant / Toeplitz / Fourier operators of
// 64..65536 points).  As vector programs their tiles were bound by the
// integer work of the generic loads and stores (about 45 % of the time) and
// by the barriers between load, program and store; the register transforms
// of fm_rfft.cuh take a tile's points, copied ahead, into registers,
// transform and store them directly, 8 points on each of the CTA's 512
// threads.
// 64 operators of 64..65536 points: 425 -> 327 us with direct loads, 321
// with the points copied ahead, 309 with barriers of the threads that
// exchange only.  Per tile they still take 1.7 times what the separate
// launches of fm_rfft.cuh take: 64 registers hold the records' fields and
// the transform, barriers and load latency lead the stalls.  Measured and
// left out: one CTA of 128 registers a thread (385 us), runs of one step's
// tiles without CTA barriers and with host-made divisors (312), all factors
// of a product loaded before use (323: spills).
#pragma once

#include "fm_rfft.cuh"

namespace fmk {

// Modes of a batch step's register transform
enum {
  RXM_NONE = 0,
  RXM_FFT = 1,    // as rxfft_kernel, 64..512 points
  RXM_CONV = 2    // as rxconv_kernel, 128..4096 points
};
// The lengths built, for the dispatch on the device and for the rule that
// sends a step there: a step never meets a length that is not built.
#define FM_RXB_FFT(X) X(64) X(128) X(256) X(512)
#define FM_RXB_CONV(X) X(128) X(256) X(512) X(1024) X(2048) X(4096)
inline bool rxb_built(int mode, int L) {
#define FM_RXB_IS(N) || L == N
  return mode == RXM_FFT    ? false FM_RXB_FFT(FM_RXB_IS)
         : mode == RXM_CONV ? false FM_RXB_CONV(FM_RXB_IS)
                            : false;
#undef FM_RXB_IS
}
constexpr int kRxbPoints = FM_MAX_THREADS * kRxP;  // points per tile
// shared memory of a tile's exchange buffers
constexpr size_t kRxbBytes = 38400;

// rxb_fft works in groups of threads with barriers of their own: 256
// threads up to 256 points (rows of 64 bytes or more), all 512 above
__host__ __device__ constexpr int rxb_group(int L) {
  return L <= 256 ? 256 : FM_MAX_THREADS;
}
// adjacent vectors of a group, and the stride of their exchange buffers
// (the rule of RxShape::Lx)
__host__ __device__ constexpr int rxb_nv(int L) {
  return rxb_group(L) * kRxP / L;
}
__host__ __device__ constexpr int rxb_lx(int L) {
  return rxb_nv(L) >= 16 ? ((L + (L >> 3)) | 1)
                         : L + (L >> 3) + 16 / rxb_nv(L);
}
// words between the groups' buffers
__host__ __device__ constexpr int rxb_region(int L) {
  return rxb_nv(L) * rxb_lx(L);
}

// Copy a tile's points ahead into its buffer (cp.async, zeros where there
// are none).  FFT: the points of thread k of a group at k + T r of the
// group's region, or, for contiguous vectors that rxb_fft turns, along the
// vectors at their padded positions; convolution: point j of a vector at j of
// its exchange buffer.
__device__ __forceinline__ void rxb_issue(const RxStep &p, int mode,
                                          float2 *slot, unsigned tile) {
  const int L = p.L, G = L / kRxP;
  const int tid = threadIdx.x;
  unsigned m, v;
  int j0, step;
  if (mode == RXM_FFT) {
    const int T = rxb_group(L), NV = rxb_nv(L), grp = tid / T, k0 = tid % T;
    const unsigned nbc = ((unsigned)p.V + NV - 1) / NV;
    const unsigned bt = tile * (FM_MAX_THREADS / T) + grp;
    m = bt / nbc;
    v = (bt - m * nbc) * NV;  // first vector
    if (m >= (unsigned)p.num_cols) v = (unsigned)p.V;  // none
    slot += grp * rxb_region(L);
    if (p.in_cc == 1) {
      const int lg = __ffs(L) - 1, Lx = rxb_lx(L);
      const i64 col = (i64)m * p.ld_src;
#pragma unroll
      for (int i = 0; i < kRxP; ++i) {
        const int k = k0 + T * i, vv = k >> lg, j = k & (L - 1);
        const i64 row = (i64)(v + vv) * p.in_n + j;
        i64 at = v + vv < p.V && j < p.in_len && row < p.in_rows ? row : -1;
        if (p.map_in && at >= 0) at = p.map_in[at];
        cp_async<8>(slot + vv * Lx + j + (j >> 3),
                    at >= 0 ? (const void *)((const float2 *)p.src + col + at)
                            : p.src,
                    at >= 0);
      }
      return;
    }
    v += k0 & (NV - 1);
    j0 = k0 / NV;
    slot += k0;
    step = T;
  } else {
    const int q = tid / G;
    const unsigned gv = tile * (kRxbPoints / L) + q;
    m = gv / (unsigned)p.V;
    v = gv - m * (unsigned)p.V;
    if (gv >= (unsigned)(p.V * p.num_cols)) v = (unsigned)p.V;  // none
    j0 = tid & (G - 1);
    slot += q * (L + (L >> 3)) + j0;
    step = G;
  }
  const i64 cc = p.in_cc;
  const unsigned a = v / (unsigned)cc, c = v - a * (unsigned)cc;
  const i64 rb = (i64)a * p.in_n * cc + c;
  const float2 *src = (const float2 *)p.src + (i64)m * p.ld_src;
  if (v < p.V && !p.map_in && p.in_len == L &&
      rb + (i64)(L - 1) * cc < p.in_rows) {
    const float2 *s = src + rb + (i64)j0 * cc;
    const i64 d = (i64)G * cc;
#pragma unroll
    for (int r = 0; r < kRxP; ++r, s += d)
      cp_async<8>(slot + step * r, s, true);
  } else {
#pragma unroll
    for (int r = 0; r < kRxP; ++r) {
      const int j = j0 + G * r;
      const i64 row = rb + (i64)j * cc;
      i64 at = v < p.V && j < p.in_len && row < p.in_rows ? row : -1;
      if (p.map_in && at >= 0) at = p.map_in[at];
      cp_async<8>(slot + step * r,
                  at >= 0 ? (const void *)(src + at) : p.src, at >= 0);
    }
  }
}

template <int L>
__device__ __forceinline__ void rxb_fft(const RxStep &p, cfp<8> *xb,
                                        unsigned tile) {
  typedef cfp<8> E;
  constexpr int P = kRxP, G = L / P, T = rxb_group(L), NV = rxb_nv(L);
  constexpr int SY = T == FM_MAX_THREADS ? 1 : T;
  constexpr int S = rc_stages(L, P);
  constexpr int R = rc_radix(S - 1, L, P);
  constexpr int Lx = rxb_lx(L);
  static_assert(RcBuf<E, L>::SH == 3, "padding of rxb_issue");
  static_assert((size_t)FM_MAX_THREADS / T * rxb_region(L) * sizeof(E) <=
                    kRxbBytes,
                "exchange buffers");
  const int grp = threadIdx.x / T, k0 = threadIdx.x % T;
  const int lane = k0 % NV, t = k0 / NV;
  xb += grp * rxb_region(L);
  E *buf = xb + lane * Lx;
  const unsigned nbc = (unsigned)((p.V + NV - 1) / NV);
  const unsigned bt = tile * (FM_MAX_THREADS / T) + grp;
  const unsigned m = bt / nbc, v = (bt - m * nbc) * NV + lane;
  const bool act = v < p.V && m < p.num_cols;
  const unsigned mask = p.conj_in ? 0x80000000u : 0u;
  const float2 *raw = reinterpret_cast<const float2 *>(xb);
  E x[P];
  if (p.in_cc == 1) {
    const float2 *rr = raw + lane * Lx + rc_pad<E, L>(t);
#pragma unroll
    for (int r = 0; r < P; ++r) {
      const float2 d = rx_conj(rr[rc_pad<E, L>(G * r)], mask);
      x[r] = E{d.x, d.y};
    }
  } else {
#pragma unroll
    for (int r = 0; r < P; ++r) {
      const float2 d = rx_conj(raw[k0 + T * r], mask);
      x[r] = E{d.x, d.y};
    }
  }
  rc_sync<SY>();  // the exchanges reuse the buffer
  if (p.pre) {
    const unsigned a = v / (unsigned)p.in_cc, c = v - a * (unsigned)p.in_cc;
    rx_pre<E, L>(x, p, act, (i64)a * p.in_n * p.in_cc + c, t, G);
  }
  rc_forward<E, L, 0, -1, SY, true>(x, buf, t, (const E *)p.tw);
  if (act) {
    const unsigned ao = v / (unsigned)p.out_cc,
                   co = v - ao * (unsigned)p.out_cc;
    rx_store<E, L, true>(x, 0, p, v, (i64)m * p.ld_dst,
                         (i64)ao * p.out_n * p.out_cc + co,
                         rc_nat<E, L>(rc_base<E, L, S - 1>(t)), [](int j) {
                           return (j / R) * R + (j % R) * (L / R);
                         });
  }
}

template <int L>
__device__ __forceinline__ void rxb_conv(const RxStep &p, cfp<8> *xb,
                                         unsigned tile) {
  typedef cfp<8> E;
  constexpr int P = kRxP, G = L / P, VPC = kRxbPoints / L;
  // the threads of one vector: a warp or less, a group, the CTA
  constexpr int SY = G <= 32 ? 0 : G == FM_MAX_THREADS ? 1 : G;
  constexpr int S = rc_stages(L, P);
  constexpr int Lc = RcBuf<E, L>::Lp;
  static_assert(Lc == L + (L >> 3), "buffers of rxb_issue");
  static_assert((size_t)VPC * Lc * sizeof(E) <= kRxbBytes, "exchange buffers");
  const int q = threadIdx.x / G, g = threadIdx.x % G;
  E *buf = xb + q * Lc;
  const unsigned gv = tile * VPC + q;
  const bool act = gv < (unsigned)(p.V * p.num_cols);
  const unsigned m = gv / (unsigned)p.V, v = gv - m * (unsigned)p.V;
  const unsigned mask = p.conj_in ? 0x80000000u : 0u;
  const float2 *raw = reinterpret_cast<const float2 *>(buf) + g;
  E x[P];
#pragma unroll
  for (int r = 0; r < P; ++r) {
    const float2 d = rx_conj(raw[G * r], mask);
    x[r] = E{d.x, d.y};
  }
  rc_sync<SY>();  // the exchanges reuse the buffer
  rx_pre<E, L>(x, p, act, (i64)v * p.in_n, g, G);
  rc_forward<E, L, 0, -1, SY, true>(x, buf, g, (const E *)p.tw);
  if (act) {
    const E *sp = (const E *)p.spec + (i64)v * p.spec_stride + g;
#pragma unroll
    for (int j = 0; j < P; ++j)
      x[j] = mulv(x[j], tw_get<true>(sp, j * G), p.spec_conj != 0);
  }
  rc_inverse<E, L, S - 1, SY, true>(x, buf, g, (const E *)p.tw);
  if (act)
    rx_store<E, L, true>(x, 0, p, v, (i64)m * p.ld_dst, (i64)v * p.out_n, g,
                         [](int r) { return G * r; });
}

// one tile of a register step (complex64; called by all 512 threads, a
// barrier follows)
__device__ __forceinline__ void rx_batch_tile(const RxStep &p, int mode,
                                           cfp<8> *xb, unsigned tile) {
  switch (mode * 8192 + p.L) {
#define FM_RXB_CASE(N) \
  case RXM_FFT * 8192 + N: rxb_fft<N>(p, xb, tile); break;
    FM_RXB_FFT(FM_RXB_CASE)
#undef FM_RXB_CASE
#define FM_RXB_CASE(N) \
  case RXM_CONV * 8192 + N: rxb_conv<N>(p, xb, tile); break;
    FM_RXB_CONV(FM_RXB_CASE)
#undef FM_RXB_CASE
    default: break;
  }
}

// Loads of one batch tile into a slot: cp.async when the source already
// has the compute type and needs no gather (completion is awaited later,
// so the copy overlaps the previous tile's program), synchronous loads with
// conversion and gather otherwise.
// The launch record is first copied into shared memory (read there by
// every op of the tile program instead of from global memory).
template <class E>
__device__ __forceinline__ void batch_issue_load(const Step *gp, Step *slot,
                                                 E *sm, VInfo *vi, i64 tile,
                                                 int tid, int T) {
  {
    static_assert(sizeof(Step) % 16 == 0, "launch record size");
    const int4 *src = reinterpret_cast<const int4 *>(gp);
    int4 *dst = reinterpret_cast<int4 *>(slot);
    for (int i = tid; i < (int)(sizeof(Step) / 16); i += T) dst[i] = src[i];
  }
  __syncthreads();
  const Step &p = *slot;
  const i64 nvec = p.V * p.num_cols;
  const FDivF dV((unsigned)p.V), dci((unsigned)p.vin.Cc),
      dco((unsigned)p.vout.Cc);
  setup_tile(p, vi, tile, dV, dci, dco, nvec, tid, T);
  __syncthreads();
  if (p.src_type == Tr<E>::code && !p.map_in)
    load_async<E, 0>(p, sm, vi, tid, T);
  else
    load_general<E, 0>(p, sm, vi, tid, T);
  cp_async_commit();
}

template <class E, int CLS>
__global__ void __launch_bounds__(FM_MAX_THREADS, (MinBlocks<E, CLS>::v))
    batch_kernel(const Step *__restrict__ steps, const i64 *__restrict__ start,
                 const int *__restrict__ level, const RxStep *__restrict__ rx,
                 const int *__restrict__ rxmode, int nlev, unsigned *bar,
                 int *err, int max_B, size_t max_tile, long long wait_limit) {
  extern __shared__ __align__(128) unsigned char fm_smem[];
  const int tid = threadIdx.x, T = blockDim.x;
  Step *const sst = reinterpret_cast<Step *>(fm_smem);
  unsigned char *const h = fm_smem + batch_steps_bytes();
  i64 *sq = reinterpret_cast<i64 *>(h);
  // slot k: launch record, per-vector records, exponents and tile buffer
  // (addresses recomputed on use to keep registers free)
  const unsigned rec = (unsigned)((sizeof(VInfo) + 4) * max_B);
  auto vis = [&](int k) {
    return reinterpret_cast<VInfo *>(h + 8 * max_B + k * rec);
  };
  auto sexps = [&](int k) {
    return reinterpret_cast<int *>(h + 8 * max_B + k * rec +
                                   sizeof(VInfo) * max_B);
  };
  auto bufs = [&](int k) {
    return reinterpret_cast<E *>(fm_smem + batch_head_bytes(max_B) +
                                 k * max_tile);
  };
  const i64 G = gridDim.x;
  // complex64: whether a step's tiles run as register transforms
  auto mode = [&](int k) {
    return std::is_same<E, float2>::value ? __ldg(rxmode + k) : 0;
  };
  // records of the register steps in the two slots, and which steps
  __shared__ RxStep srx[2];
  int rxk[2] = {-1, -1};
  // loads of tile `at` of step k into slot c (one cp.async group)
  auto issue = [&](int k, int c, i64 at) {
    const int md = mode(k);
    if (md == 0) {
      batch_issue_load<E>(steps + k, sst + c, bufs(c), vis(c), at, tid, T);
      return;
    }
    if constexpr (std::is_same<E, float2>::value) {
      if (rxk[c] != k) {
        static_assert(sizeof(RxStep) % 8 == 0, "record size");
        for (int i = tid; i < (int)(sizeof(RxStep) / 8); i += T)
          reinterpret_cast<unsigned long long *>(srx + c)[i] =
              reinterpret_cast<const unsigned long long *>(rx + k)[i];
        rxk[c] = k;
        __syncthreads();
      }
      rxb_issue(srx[c], md, bufs(c), (unsigned)at);
      cp_async_commit();
    }
  };
  for (int l = 0; l < nlev; ++l) {
    const int s0 = level[l], s1 = level[l + 1];
    const i64 t1 = start[s1];
    // two-slot pipeline: the loads of tile g + G are issued before tile g
    // is transformed and stored
    i64 g = start[s0] + blockIdx.x;
    int kc = s0, cur = 0;
    if (g < t1) {
      while (start[kc + 1] <= g) ++kc;
      issue(kc, 0, g - start[kc]);
    }
    for (; g < t1; g += G) {
      const i64 gn = g + G;
      int kn = kc;
      if (gn < t1) {
        while (start[kn + 1] <= gn) ++kn;
        issue(kn, cur ^ 1, gn - start[kn]);
        cp_async_wait<1>();
      } else {
        cp_async_wait<0>();
      }
      if constexpr (std::is_same<E, float2>::value) {
        const int md = mode(kc);
        if (md != 0) {
          __syncthreads();
          rx_batch_tile(srx[cur], md, reinterpret_cast<cfp<8> *>(bufs(cur)),
                        (unsigned)(g - start[kc]));
          __syncthreads();
          cur ^= 1;
          kc = kn;
          continue;
        }
      }
      __syncthreads();
      const Step &p = sst[cur];
      E *sm = bufs(cur);
      VInfo *vi = vis(cur);
      int *sexp = sexps(cur);
      const bool async = p.src_type == Tr<E>::code && !p.map_in;
      if constexpr (Emu<E>::v) {
        if (async) {
          emu_in<E, 0>(p, sm, vi, sexp, tid, T);
        } else {
          for (int b = tid; b < p.B; b += T) sexp[b] = 0;
        }
        __syncthreads();
      }
      if (async && (p.conj_in || p.pre)) {
        load_fixup<E, 0>(p, sm, vi, tid, T);
        __syncthreads();
      }
      const int nwarps = T >> 5;
      bool natural = false, stored = false;
      if constexpr (std::is_same<E, float2>::value) {
        if (p.rprog) {
          // the program on registers; results in natural order (or already
          // stored)
          rt_program(p, sm, vi, tid, T);
          natural = true;
          stored = (p.rprog & RT_DIRECT) != 0;
        }
      }
      if (natural) {
      } else if (warp_mode<E, CLS, 0>(p.B, p.L, nwarps)) {
        const int w = tid >> 5, vw = p.B / nwarps;
        run_program<E, CLS, 0>(p, sm + w * vw * p.Lp, p.Lp, vw, vi + w * vw,
                               sq + w * vw, tid & 31, 32);
        __syncthreads();
      } else {
        run_program<E, CLS, 0>(p, sm, p.Lp, p.B, vi, sq, tid, T);
      }
      if (!stored) store_tile<E, 0>(p, sm, vi, sexp, tid, T, natural);
      __syncthreads();
      cur ^= 1;
      kc = kn;
    }
    if (l + 1 < nlev &&
        !grid_barrier(bar, (unsigned)(l + 1) * gridDim.x, err, wait_limit))
      return;
  }
}

}  // namespace fmk
