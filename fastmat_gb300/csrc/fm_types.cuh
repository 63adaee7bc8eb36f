// Element types, arithmetic and dtype conversion for the matvec kernels.
//
// The engine computes in one of five element types: float, double (real
// operators such as Hadamard/Diag on real data), float2, double2 (complex,
// stored interleaved exactly like numpy complex64/complex128) and long long
// (integer-only operator trees; results are narrowed to the fastmat output
// type on store, which reproduces fastmat's wrap-around integer arithmetic
// because wrapping is a ring homomorphism).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/fmgpu.h"

namespace fmk {

typedef long long i64;

// ---------------------------------------------------------------- double-float
// A double-float number is an unevaluated sum h + l of two floats with
// |l| <= ulp(h) / 2, carrying a 48-bit significand (relative precision about
// 2^-48) on the FP32 pipes.  Sums use Knuth's TwoSum, products Dekker's
// TwoProduct through the fused multiply-add (both error-free
// transformations), each followed by a renormalisation (Fast2Sum).  The
// sum is the "sloppy" variant: its error is bounded by 2^-46 (|a| + |b|),
// the norm-wise bound an FFT error analysis needs.
struct df {
  float h, l;
  df() = default;
  __host__ __device__ constexpr df(float h_, float l_) : h(h_), l(l_) {}
  // compile-time constants: split a double literal into two floats
  __host__ __device__ constexpr df(double d)
      : h((float)d), l((float)(d - (double)(float)d)) {}
  __host__ __device__ constexpr df(int i) : h((float)i), l(0.f) {}
};
struct dfc {
  df x, y;  // real, imaginary
};

__device__ __forceinline__ df fast_two_sum(float a, float b) {
  const float s = a + b;
  return df(s, b - (s - a));
}
__device__ __forceinline__ df operator+(df a, df b) {
  const float s = a.h + b.h;
  const float bb = s - a.h;
  const float e = (a.h - (s - bb)) + (b.h - bb) + (a.l + b.l);
  return fast_two_sum(s, e);
}
__device__ __forceinline__ df operator-(df a) { return df(-a.h, -a.l); }
__device__ __forceinline__ df operator-(df a, df b) { return a + (-b); }
__device__ __forceinline__ df operator*(df a, df b) {
  const float p = a.h * b.h;
  float e = fmaf(a.h, b.h, -p);
  e = fmaf(a.h, b.l, e);
  e = fmaf(a.l, b.h, e);
  return fast_two_sum(p, e);
}
// sign * x for sign = +1 / -1
__device__ __forceinline__ df operator*(int s, df a) { return s < 0 ? -a : a; }
__device__ __forceinline__ float smul(int s, float a) { return s < 0 ? -a : a; }
__device__ __forceinline__ double smul(int s, double a) {
  return s < 0 ? -a : a;
}
__device__ __forceinline__ df smul(int s, df a) { return s < 0 ? -a : a; }

__device__ __forceinline__ dfc operator+(dfc a, dfc b) {
  return dfc{a.x + b.x, a.y + b.y};
}
__device__ __forceinline__ dfc operator-(dfc a, dfc b) {
  return dfc{a.x - b.x, a.y - b.y};
}
__device__ __forceinline__ dfc cmul(dfc a, dfc b) {
  return dfc{a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x};
}
__device__ __forceinline__ dfc cmulc(dfc a, dfc b) {
  return dfc{a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y};
}

// Unnormalised double-float, for the additions inside one butterfly: the
// head is the rounded sum of the heads (TwoSum keeps its rounding error
// exactly) and the tail collects tails and errors without renormalising,
// 8 FP32 operations per addition instead of 11; a product skips the final
// renormalisation too (4 instead of 7).  Tails stay a few units of 2^-24
// of the magnitudes that entered the chain, so a chain of k operations
// keeps the norm-wise error bound of about k 2^-48 times the sum of those
// magnitudes (the bound an FFT error analysis uses).  Values are
// renormalised (Fast2Sum) when they leave the butterfly.
struct dfu {
  float h, l;
  dfu() = default;
  __host__ __device__ constexpr dfu(float h_, float l_) : h(h_), l(l_) {}
  __host__ __device__ constexpr dfu(double d)
      : h((float)d), l((float)(d - (double)(float)d)) {}
};
struct dfcu {
  dfu x, y;
};
__device__ __forceinline__ dfu operator+(dfu a, dfu b) {
  const float s = a.h + b.h;
  const float bb = s - a.h;
  const float e = (a.h - (s - bb)) + (b.h - bb);
  return dfu(s, (a.l + b.l) + e);
}
__device__ __forceinline__ dfu operator-(dfu a) { return dfu(-a.h, -a.l); }
__device__ __forceinline__ dfu operator-(dfu a, dfu b) { return a + (-b); }
__device__ __forceinline__ dfu operator*(dfu a, dfu b) {
  const float p = a.h * b.h;
  float e = fmaf(a.h, b.h, -p);
  e = fmaf(a.h, b.l, e);
  e = fmaf(a.l, b.h, e);
  return dfu(p, e);
}
__device__ __forceinline__ dfu smul(int s, dfu a) { return s < 0 ? -a : a; }
__device__ __forceinline__ dfcu operator+(dfcu a, dfcu b) {
  return dfcu{a.x + b.x, a.y + b.y};
}
__device__ __forceinline__ dfcu operator-(dfcu a, dfcu b) {
  return dfcu{a.x - b.x, a.y - b.y};
}

// ---- complex double-float in packed form: the heads of real and imaginary
// part as one float2, the tails as another, so that every operation on both
// parts is one packed FP32 instruction (add / sub / mul / fma .rn.f32x2:
// each half rounds exactly as the scalar operation).  The packed forms run
// at the scalar FP32 rate but take half the issue slots (measured: 64
// packed or 128 scalar additions per clock and SM), which the register
// kernels' conversion and exchange instructions then use.  dfq is
// normalised as dfc is, dfqu unnormalised as dfcu is.
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 r;
  asm("{\n .reg .b64 a, b, c;\n mov.b64 a, {%2, %3};\n mov.b64 b, {%4, %5};\n"
      " add.rn.f32x2 c, a, b;\n mov.b64 {%0, %1}, c;\n}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
  float2 r;
  asm("{\n .reg .b64 a, b, c;\n mov.b64 a, {%2, %3};\n mov.b64 b, {%4, %5};\n"
      " sub.rn.f32x2 c, a, b;\n mov.b64 {%0, %1}, c;\n}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  float2 r;
  asm("{\n .reg .b64 a, b, c;\n mov.b64 a, {%2, %3};\n mov.b64 b, {%4, %5};\n"
      " mul.rn.f32x2 c, a, b;\n mov.b64 {%0, %1}, c;\n}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 d) {
  float2 r;
  asm("{\n .reg .b64 a, b, c, d;\n mov.b64 a, {%2, %3};\n"
      " mov.b64 b, {%4, %5};\n mov.b64 d, {%6, %7};\n"
      " fma.rn.f32x2 c, a, b, d;\n mov.b64 {%0, %1}, c;\n}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(d.x), "f"(d.y));
  return r;
}
__device__ __forceinline__ float2 neg2(float2 a) {
  return make_float2(-a.x, -a.y);
}
struct dfq {
  float2 h, l;  // (re, im) heads, (re, im) tails
};
struct dfqu {
  float2 h, l;
};
__device__ __forceinline__ dfq pack(dfc a) {
  return dfq{make_float2(a.x.h, a.y.h), make_float2(a.x.l, a.y.l)};
}
__device__ __forceinline__ dfc unpack(dfq a) {
  return dfc{df(a.h.x, a.l.x), df(a.h.y, a.l.y)};
}
__device__ __forceinline__ dfqu operator+(dfqu a, dfqu b) {
  const float2 s = add2(a.h, b.h);
  const float2 bb = sub2(s, a.h);
  const float2 e = add2(sub2(a.h, sub2(s, bb)), sub2(b.h, bb));
  return dfqu{s, add2(add2(a.l, b.l), e)};
}
__device__ __forceinline__ dfqu operator-(dfqu a, dfqu b) {
  const float2 s = sub2(a.h, b.h);
  const float2 bb = sub2(s, a.h);
  const float2 e = sub2(sub2(a.h, sub2(s, bb)), add2(b.h, bb));
  return dfqu{s, add2(sub2(a.l, b.l), e)};
}
// complex64 with packed additions, NP points per thread in the register
// transforms (the results of every operation are float2's)
template <int NP> struct alignas(8) cfp {
  float x, y;
};
template <int NP>
__device__ __forceinline__ cfp<NP> operator+(cfp<NP> a, cfp<NP> b) {
  const float2 r = add2(make_float2(a.x, a.y), make_float2(b.x, b.y));
  return cfp<NP>{r.x, r.y};
}
template <int NP>
__device__ __forceinline__ cfp<NP> operator-(cfp<NP> a, cfp<NP> b) {
  const float2 r = sub2(make_float2(a.x, a.y), make_float2(b.x, b.y));
  return cfp<NP>{r.x, r.y};
}
template <int NP>
__device__ __forceinline__ cfp<NP> cmul(cfp<NP> a, cfp<NP> b) {
  return cfp<NP>{fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x)};
}
template <int NP>
__device__ __forceinline__ cfp<NP> cmulc(cfp<NP> a, cfp<NP> b) {
  return cfp<NP>{fmaf(a.x, b.x, a.y * b.y), fmaf(a.y, b.x, -a.x * b.y)};
}
template <int NP>
__device__ __forceinline__ cfp<NP> mulv(cfp<NP> a, cfp<NP> b, bool c) {
  return c ? cmulc(a, b) : cmul(a, b);
}
template <int NP> __device__ __forceinline__ cfp<NP> conjv(cfp<NP> a) {
  return cfp<NP>{a.x, -a.y};
}
// product with a real factor (h, l) common to both parts
__device__ __forceinline__ dfqu rmul(dfqu a, float h, float l) {
  const float2 bh = make_float2(h, h), bl = make_float2(l, l);
  const float2 p = mul2(a.h, bh);
  float2 e = fma2(a.h, bh, neg2(p));
  e = fma2(a.h, bl, e);
  e = fma2(a.l, bh, e);
  return dfqu{p, e};
}
// a times i (sign > 0) or -i
__device__ __forceinline__ dfqu rot90(dfqu a, int sign) {
  if (sign > 0)
    return dfqu{make_float2(-a.h.y, a.h.x), make_float2(-a.l.y, a.l.x)};
  return dfqu{make_float2(a.h.y, -a.h.x), make_float2(a.l.y, -a.l.x)};
}

// double -> double-float with integer operations only (the FP64 pipe of
// this GPU is slow): h is d rounded to 24 bits, l the float nearest to the
// exact remainder d - h.  Zeros, subnormals and values outside the float
// exponent range map to (0, 0) / (+-inf, 0).
__device__ __forceinline__ df d2df(double d) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(d);
  const unsigned sgn = (unsigned)(b >> 63) << 31;
  const int ex = (int)((b >> 52) & 0x7FF);
  if (ex == 0) return df(0.f, 0.f);
  int e = ex - 1023;
  if (ex == 0x7FF || e > 127)
    return df(__int_as_float((int)(sgn | 0x7F800000u)), 0.f);
  if (e < -126) return df(0.f, 0.f);
  const unsigned long long m = (b & 0xFFFFFFFFFFFFFull) | (1ull << 52);
  unsigned long long mh = m >> 29;  // 24 bits
  const unsigned long long rem = m & 0x1FFFFFFFull;
  const unsigned long long half = 1ull << 28;
  if (rem > half || (rem == half && (mh & 1))) ++mh;
  // remainder relative to the rounded head: m - mh * 2^29 (|.| <= 2^28)
  const long long r = (long long)m - (long long)(mh << 29);
  if (mh == (1ull << 24)) {  // rounding carried into the next binade
    mh >>= 1;
    ++e;
    if (e > 127) return df(__int_as_float((int)(sgn | 0x7F800000u)), 0.f);
  }
  const float h = __int_as_float(
      (int)(sgn | ((unsigned)(e + 127) << 23) | (unsigned)(mh & 0x7FFFFF)));
  // l = r * 2^(e0 - 52) with e0 the exponent before any carry
  const int el = ex - 1023 - 52;
  float l = (float)(int)r;  // |r| <= 2^28: rounds to 24 bits
  if (el >= -126) {
    l *= __int_as_float((el + 127) << 23);
  } else if (el >= -126 - 23) {
    l *= __int_as_float((el + 127 + 24) << 23);
    l *= __int_as_float((127 - 24) << 23);
  } else {
    l = 0.f;
  }
  if (sgn) l = -l;
  return df(h, l);
}

// ---------------------------------------------------------------- traits
template <class E> struct Tr;
template <> struct Tr<float> {
  static constexpr bool cplx = false;
  static constexpr int code = FM_F32;
  typedef float R;
};
template <> struct Tr<double> {
  static constexpr bool cplx = false;
  static constexpr int code = FM_F64;
  typedef double R;
};
template <> struct Tr<float2> {
  static constexpr bool cplx = true;
  static constexpr int code = FM_C64;
  typedef float R;
};
template <> struct Tr<double2> {
  static constexpr bool cplx = true;
  static constexpr int code = FM_C128;
  typedef double R;
};
template <> struct Tr<i64> {
  static constexpr bool cplx = false;
  static constexpr int code = FM_I64;
  typedef i64 R;
};
// double-float types hold (complex) float64 data: their buffers in global
// memory are float64 / complex128, converted on load and store (emu)
template <> struct Tr<df> {
  static constexpr bool cplx = false;
  static constexpr int code = FM_F64;
  typedef df R;
};
template <> struct Tr<dfc> {
  static constexpr bool cplx = true;
  static constexpr int code = FM_C128;
  typedef df R;
};
template <> struct Tr<dfu> {
  static constexpr bool cplx = false;
  static constexpr int code = FM_F64;
  typedef dfu R;
};
template <> struct Tr<dfcu> {
  static constexpr bool cplx = true;
  static constexpr int code = FM_C128;
  typedef dfu R;
};
template <int NP> struct Tr<cfp<NP>> {
  static constexpr bool cplx = true;
  static constexpr int code = FM_C64;
  typedef float R;
};
template <> struct Tr<dfq> {
  static constexpr bool cplx = true;
  static constexpr int code = FM_C128;
  typedef df R;
};
template <> struct Tr<dfqu> {
  static constexpr bool cplx = true;
  static constexpr int code = FM_C128;
  typedef dfu R;
};
// the type a butterfly computes in: unnormalised for double-float
template <class C> struct Lazy { typedef C type; };
template <> struct Lazy<df> { typedef dfu type; };
template <> struct Lazy<dfc> { typedef dfcu type; };
template <> struct Lazy<dfq> { typedef dfqu type; };
template <class C> __device__ __forceinline__ C to_lazy(C a) { return a; }
template <class C> __device__ __forceinline__ C from_lazy(C a) { return a; }
__device__ __forceinline__ dfu to_lazy(df a) { return dfu(a.h, a.l); }
__device__ __forceinline__ dfcu to_lazy(dfc a) {
  return dfcu{dfu(a.x.h, a.x.l), dfu(a.y.h, a.y.l)};
}
__device__ __forceinline__ df from_lazy(dfu a) {
  return fast_two_sum(a.h, a.l);
}
__device__ __forceinline__ dfc from_lazy(dfcu a) {
  return dfc{fast_two_sum(a.x.h, a.x.l), fast_two_sum(a.y.h, a.y.l)};
}
__device__ __forceinline__ dfqu to_lazy(dfq a) { return dfqu{a.h, a.l}; }
__device__ __forceinline__ dfq from_lazy(dfqu a) {
  const float2 s = add2(a.h, a.l);
  return dfq{s, sub2(a.l, sub2(s, a.h))};
}
__device__ __forceinline__ dfq operator+(dfq a, dfq b) {
  return from_lazy(to_lazy(a) + to_lazy(b));
}
template <class E> struct Emu { static constexpr bool v = false; };
template <> struct Emu<dfq> { static constexpr bool v = true; };
template <> struct Emu<df> { static constexpr bool v = true; };
template <> struct Emu<dfc> { static constexpr bool v = true; };

// shared-memory padding: one spare 16-byte granule per 128 bytes keeps
// strided butterfly accesses spread over the banks while every 128-byte
// chunk of a vector stays 16-byte aligned (a bulk-copy destination)
template <class E> struct PadShift {
  static constexpr int v = sizeof(E) == 4 ? 5 : (sizeof(E) == 8 ? 4 : 3);
  static constexpr int mul = 16 / (int)sizeof(E);
};

template <class E> __host__ __device__ __forceinline__ int pidx(int i) {
  return i + PadShift<E>::mul * (i >> PadShift<E>::v);
}

// ---------------------------------------------------------------- arithmetic
__device__ __forceinline__ float2 operator+(float2 a, float2 b) {
  return make_float2(a.x + b.x, a.y + b.y);
}
__device__ __forceinline__ float2 operator-(float2 a, float2 b) {
  return make_float2(a.x - b.x, a.y - b.y);
}
__device__ __forceinline__ double2 operator+(double2 a, double2 b) {
  return make_double2(a.x + b.x, a.y + b.y);
}
__device__ __forceinline__ double2 operator-(double2 a, double2 b) {
  return make_double2(a.x - b.x, a.y - b.y);
}

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
// a * conj(b)
__device__ __forceinline__ float2 cmulc(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, a.y * b.y), fmaf(a.y, b.x, -a.x * b.y));
}
__device__ __forceinline__ double2 cmulc(double2 a, double2 b) {
  return make_double2(fma(a.x, b.x, a.y * b.y), fma(a.y, b.x, -a.x * b.y));
}

// generic multiply for all element types (conj applies to b)
__device__ __forceinline__ float mulv(float a, float b, bool) { return a * b; }
__device__ __forceinline__ double mulv(double a, double b, bool) {
  return a * b;
}
__device__ __forceinline__ i64 mulv(i64 a, i64 b, bool) { return a * b; }
__device__ __forceinline__ float2 mulv(float2 a, float2 b, bool c) {
  return c ? cmulc(a, b) : cmul(a, b);
}
__device__ __forceinline__ double2 mulv(double2 a, double2 b, bool c) {
  return c ? cmulc(a, b) : cmul(a, b);
}

__device__ __forceinline__ df mulv(df a, df b, bool) { return a * b; }
__device__ __forceinline__ dfc mulv(dfc a, dfc b, bool c) {
  return c ? cmulc(a, b) : cmul(a, b);
}
// (packed form: the operations of cmul / cmulc, each product and the sum
// normalised; renormalising once after an unnormalised sum measured 1.3
// times the error of a product)
__device__ __forceinline__ dfq mulv(dfq a, dfq b, bool c) {
  const float2 by = c ? make_float2(-b.h.y, -b.l.y)
                      : make_float2(b.h.y, b.l.y);
  const dfqu u = to_lazy(a);
  return from_lazy(rmul(u, b.h.x, b.l.x)) +
         from_lazy(rmul(rot90(u, +1), by.x, by.y));
}
__device__ __forceinline__ dfq conjv(dfq a) {
  return dfq{make_float2(a.h.x, -a.h.y), make_float2(a.l.x, -a.l.y)};
}
__device__ __forceinline__ df conjv(df a) { return a; }
__device__ __forceinline__ dfc conjv(dfc a) { return dfc{a.x, -a.y}; }
__device__ __forceinline__ df addv(df a, df b) { return a + b; }
__device__ __forceinline__ dfc addv(dfc a, dfc b) { return a + b; }
__device__ __forceinline__ df subv(df a, df b) { return a - b; }
__device__ __forceinline__ dfc subv(dfc a, dfc b) { return a - b; }
__device__ __forceinline__ dfu addv(dfu a, dfu b) { return a + b; }
__device__ __forceinline__ dfcu addv(dfcu a, dfcu b) { return a + b; }
__device__ __forceinline__ dfu subv(dfu a, dfu b) { return a - b; }
__device__ __forceinline__ dfcu subv(dfcu a, dfcu b) { return a - b; }

__device__ __forceinline__ float conjv(float a) { return a; }
__device__ __forceinline__ double conjv(double a) { return a; }
__device__ __forceinline__ i64 conjv(i64 a) { return a; }
__device__ __forceinline__ float2 conjv(float2 a) {
  return make_float2(a.x, -a.y);
}
__device__ __forceinline__ double2 conjv(double2 a) {
  return make_double2(a.x, -a.y);
}

template <class E> __device__ __forceinline__ E zero();
template <> __device__ __forceinline__ float zero<float>() { return 0.f; }
template <> __device__ __forceinline__ double zero<double>() { return 0.; }
template <> __device__ __forceinline__ i64 zero<i64>() { return 0; }
template <> __device__ __forceinline__ float2 zero<float2>() {
  return make_float2(0.f, 0.f);
}
template <> __device__ __forceinline__ double2 zero<double2>() {
  return make_double2(0., 0.);
}
template <> __device__ __forceinline__ df zero<df>() { return df(0.f, 0.f); }
template <> __device__ __forceinline__ dfc zero<dfc>() {
  return dfc{df(0.f, 0.f), df(0.f, 0.f)};
}

// a (complex) scalar given in double precision, in the element type E;
// for double-float types this is the host-free integer split
template <class E> __device__ __forceinline__ E scalar_of(double re, double im) {
  return E{(float)re, (float)im};
}
template <> __device__ __forceinline__ float scalar_of<float>(double re, double) {
  return (float)re;
}
template <> __device__ __forceinline__ double scalar_of<double>(double re, double) {
  return re;
}
template <> __device__ __forceinline__ i64 scalar_of<i64>(double re, double) {
  return (i64)re;
}
template <> __device__ __forceinline__ float2 scalar_of<float2>(double re, double im) {
  return make_float2((float)re, (float)im);
}
template <> __device__ __forceinline__ double2 scalar_of<double2>(double re, double im) {
  return make_double2(re, im);
}
template <> __device__ __forceinline__ df scalar_of<df>(double re, double) {
  return d2df(re);
}
template <> __device__ __forceinline__ dfc scalar_of<dfc>(double re, double im) {
  return dfc{d2df(re), d2df(im)};
}
template <> __device__ __forceinline__ dfq scalar_of<dfq>(double re, double im) {
  return pack(dfc{d2df(re), d2df(im)});
}

__device__ __forceinline__ float addv(float a, float b) { return a + b; }
__device__ __forceinline__ double addv(double a, double b) { return a + b; }
__device__ __forceinline__ i64 addv(i64 a, i64 b) { return a + b; }
__device__ __forceinline__ float2 addv(float2 a, float2 b) { return a + b; }
__device__ __forceinline__ double2 addv(double2 a, double2 b) { return a + b; }
__device__ __forceinline__ float subv(float a, float b) { return a - b; }
__device__ __forceinline__ double subv(double a, double b) { return a - b; }
__device__ __forceinline__ i64 subv(i64 a, i64 b) { return a - b; }
__device__ __forceinline__ float2 subv(float2 a, float2 b) { return a - b; }
__device__ __forceinline__ double2 subv(double2 a, double2 b) { return a - b; }

// scale by a (possibly complex) scalar given in double precision
__device__ __forceinline__ float scalev(float a, double sr, double) {
  return a * (float)sr;
}
__device__ __forceinline__ double scalev(double a, double sr, double) {
  return a * sr;
}
__device__ __forceinline__ i64 scalev(i64 a, double sr, double) {
  return a * (i64)sr;
}
__device__ __forceinline__ float2 scalev(float2 a, double sr, double si) {
  return cmul(a, make_float2((float)sr, (float)si));
}
__device__ __forceinline__ double2 scalev(double2 a, double sr, double si) {
  return cmul(a, make_double2(sr, si));
}

// ---------------------------------------------------------------- conversion
// A loaded source element, widened to (re, im) doubles or an integer.
struct Wide {
  double re, im;
  i64 iv;
  bool is_int;
};

__device__ __forceinline__ Wide load_wide(const void *p, int type, i64 idx) {
  Wide w;
  w.im = 0.;
  w.is_int = false;
  w.iv = 0;
  switch (type) {
    case FM_I8: w.iv = ((const int8_t *)p)[idx]; w.is_int = true; break;
    case FM_I16: w.iv = ((const int16_t *)p)[idx]; w.is_int = true; break;
    case FM_I32: w.iv = ((const int32_t *)p)[idx]; w.is_int = true; break;
    case FM_I64: w.iv = ((const i64 *)p)[idx]; w.is_int = true; break;
    case FM_F32: w.re = ((const float *)p)[idx]; break;
    case FM_F64: w.re = ((const double *)p)[idx]; break;
    case FM_C64: {
      float2 v = ((const float2 *)p)[idx];
      w.re = v.x;
      w.im = v.y;
      break;
    }
    default: {
      double2 v = ((const double2 *)p)[idx];
      w.re = v.x;
      w.im = v.y;
      break;
    }
  }
  if (w.is_int) w.re = (double)w.iv;
  return w;
}

template <class E> __device__ __forceinline__ E from_wide(const Wide &w);
template <> __device__ __forceinline__ float from_wide<float>(const Wide &w) {
  return (float)w.re;
}
template <> __device__ __forceinline__ double from_wide<double>(const Wide &w) {
  return w.re;
}
template <> __device__ __forceinline__ i64 from_wide<i64>(const Wide &w) {
  return w.is_int ? w.iv : (i64)w.re;
}
template <> __device__ __forceinline__ float2 from_wide<float2>(const Wide &w) {
  return make_float2((float)w.re, (float)w.im);
}
template <>
__device__ __forceinline__ double2 from_wide<double2>(const Wide &w) {
  return make_double2(w.re, w.im);
}

template <> __device__ __forceinline__ df from_wide<df>(const Wide &w) {
  return d2df(w.re);
}
template <> __device__ __forceinline__ dfc from_wide<dfc>(const Wide &w) {
  return dfc{d2df(w.re), d2df(w.im)};
}

// Load element idx of a buffer of element type `type` as E.  The common case
// (buffer already in the compute type) is a single typed load.
template <class E>
__device__ __forceinline__ E load_as(const void *p, int type, i64 idx) {
  if constexpr (Emu<E>::v) {
    return from_wide<E>(load_wide(p, type, idx));
  } else {
    if (type == Tr<E>::code) return ((const E *)p)[idx];
    return from_wide<E>(load_wide(p, type, idx));
  }
}

__device__ __forceinline__ void split(float v, double &re, double &im) {
  re = v;
  im = 0.;
}
__device__ __forceinline__ void split(double v, double &re, double &im) {
  re = v;
  im = 0.;
}
__device__ __forceinline__ void split(i64 v, double &re, double &im) {
  re = (double)v;
  im = 0.;
}
__device__ __forceinline__ void split(float2 v, double &re, double &im) {
  re = v.x;
  im = v.y;
}
__device__ __forceinline__ void split(double2 v, double &re, double &im) {
  re = v.x;
  im = v.y;
}
// exponent field of a double (0 for zero / subnormal)
__device__ __forceinline__ int dexp(double d) {
  return (int)(((unsigned long long)__double_as_longlong(d) >> 52) & 0x7FF);
}
// in-place conversions of a double-float tile element and its float64 /
// complex128 bit pattern (same size)
// (s: power-of-two scale of the vector, removed on load, restored on store)
__device__ __forceinline__ int raw_exp(df raw) {
  return dexp(*reinterpret_cast<const double *>(&raw));
}
__device__ __forceinline__ int raw_exp(dfc raw) {
  const double2 d = *reinterpret_cast<const double2 *>(&raw);
  const int a = dexp(d.x), b = dexp(d.y);
  return a > b ? a : b;
}
// Tile conversions, branch-free (they run once per element on every load
// and store of the double-float kernels).
// float64 d times 2^-s -> double-float: h keeps the leading 24 significand
// bits (truncated), l is the other 29 bits rounded to a float, so h + l is
// within 2^-48 |d|.  s is the vector's largest exponent minus the bias (so
// every element's rebased float exponent is at most 127): elements more
// than 2^126 below that flush to zero, their l more than 2^74 below it;
// Inf and NaN stay Inf and NaN.
__device__ __forceinline__ df d2df_scaled(double d, int s) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(d);
  const unsigned hi = (unsigned)(b >> 32), lo = (unsigned)b;
  const unsigned sg = hi & 0x80000000u;
  const int ex = (int)((hi >> 20) & 0x7FFu);
  // biased float exponent of h (zeros and subnormals flush whatever s is)
  const int ef = ex ? ex - s - 896 : 0;
  const unsigned mh = __funnelshift_l(lo, hi, 3) & 0x7FFFFFu;
  float h = __int_as_float((int)(sg | ((unsigned)ef << 23) | mh));
  // the remaining bits weigh 2^(ef - 127 - 52) each
  float l = (float)(lo & 0x1FFFFFFFu) * __int_as_float((ef - 52) << 23);
  l = __int_as_float(__float_as_int(l) | (int)sg);
  if (ef < 53) l = 0.f;
  if (ef < 1) h = 0.f;
  if (ex == 0x7FF) {
    h = __int_as_float((int)(sg | (((hi & 0xFFFFFu) | lo) ? 0x7FC00000u
                                                           : 0x7F800000u)));
    l = 0.f;
  }
  return df(h, l);
}
// float -> float64, exact for normal floats; zero and subnormal floats give
// a signed zero, Inf and NaN stay Inf and NaN
__device__ __forceinline__ double f2d_fast(float f) {
  const unsigned u = (unsigned)__float_as_int(f);
  const unsigned ex = (u >> 23) & 0xFFu;
  // exponent rebased by 1023 - 127 = 896 (0x38000000 = 896 << 20)
  unsigned hi = (u & 0x80000000u) | (((u & 0x7FFFFFFFu) >> 3) + 0x38000000u);
  unsigned lo = u << 29;
  if (ex == 0) {
    hi = u & 0x80000000u;
    lo = 0u;
  }
  if (ex == 0xFFu) hi |= 0x7FF00000u;
  return __hiloint2double((int)hi, (int)lo);
}
// d * 2^s by exponent arithmetic: zero, Inf and NaN unchanged, results
// beyond the float64 range saturate to Inf or flush to a signed zero
__device__ __forceinline__ double dscale_fast(double d, int s) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(d);
  const unsigned hi = (unsigned)(b >> 32), lo = (unsigned)b;
  const int ex = (int)((hi >> 20) & 0x7FFu);
  const int ne = ex + s;
  const unsigned sg = hi & 0x80000000u;
  unsigned nhi = hi + ((unsigned)s << 20), nlo = lo;
  if (ne <= 0) {
    nhi = sg;
    nlo = 0u;
  }
  if (ne >= 0x7FF) {
    nhi = sg | 0x7FF00000u;
    nlo = 0u;
  }
  if (ex == 0 || ex == 0x7FF) {
    nhi = hi;
    nlo = lo;
  }
  return __hiloint2double((int)nhi, (int)nlo);
}
__device__ __forceinline__ double df2d_scaled(df v, int s) {
  return dscale_fast(f2d_fast(v.h) + f2d_fast(v.l), s);
}

// (double-float values carry their vector's power-of-two scale s)
__device__ __forceinline__ void split(df v, double &re, double &im,
                                      int s = 0) {
  re = df2d_scaled(v, s);
  im = 0.;
}
__device__ __forceinline__ void split(dfc v, double &re, double &im,
                                      int s = 0) {
  re = df2d_scaled(v.x, s);
  im = df2d_scaled(v.y, s);
}

__device__ __forceinline__ df from_bits(df raw, int s) {
  return d2df_scaled(*reinterpret_cast<const double *>(&raw), s);
}
__device__ __forceinline__ dfc from_bits(dfc raw, int s) {
  const double2 d = *reinterpret_cast<const double2 *>(&raw);
  return dfc{d2df_scaled(d.x, s), d2df_scaled(d.y, s)};
}
__device__ __forceinline__ df to_bits(df v, int s) {
  const double d = df2d_scaled(v, s);
  return *reinterpret_cast<const df *>(&d);
}
__device__ __forceinline__ dfc to_bits(dfc v, int s) {
  const double2 d = make_double2(df2d_scaled(v.x, s), df2d_scaled(v.y, s));
  return *reinterpret_cast<const dfc *>(&d);
}

// Store v (compute type E) into a buffer of element type `type`, optionally
// adding to what is there.
template <class E>
__device__ __forceinline__ void store_as(void *p, int type, i64 idx, E v,
                                         bool acc, int scale = 0) {
  if (!Emu<E>::v && type == Tr<E>::code) {
    E *q = (E *)p + idx;
    *q = acc ? addv(*q, v) : v;
    return;
  }
  if constexpr (Tr<E>::code == FM_I64) {
    // integer compute narrowed to the output integer type (wraps like
    // fastmat's typed integer loops)
    const i64 iv = v;
    switch (type) {
      case FM_I8: {
        int8_t *q = (int8_t *)p + idx;
        *q = (int8_t)(acc ? (i64)*q + iv : iv);
        return;
      }
      case FM_I16: {
        int16_t *q = (int16_t *)p + idx;
        *q = (int16_t)(acc ? (i64)*q + iv : iv);
        return;
      }
      case FM_I32: {
        int32_t *q = (int32_t *)p + idx;
        *q = (int32_t)(acc ? (i64)*q + iv : iv);
        return;
      }
      default: break;
    }
  }
  double re, im;
  if constexpr (Emu<E>::v) split(v, re, im, scale);
  else split(v, re, im);
  switch (type) {
    case FM_F32: {
      float *q = (float *)p + idx;
      *q = acc ? *q + (float)re : (float)re;
      return;
    }
    case FM_F64: {
      double *q = (double *)p + idx;
      *q = acc ? *q + re : re;
      return;
    }
    case FM_C64: {
      float2 *q = (float2 *)p + idx;
      float2 n = make_float2((float)re, (float)im);
      *q = acc ? *q + n : n;
      return;
    }
    case FM_C128: {
      double2 *q = (double2 *)p + idx;
      double2 n = make_double2(re, im);
      *q = acc ? *q + n : n;
      return;
    }
    case FM_I64: {
      i64 *q = (i64 *)p + idx;
      i64 n = (i64)re;
      *q = acc ? *q + n : n;
      return;
    }
    default: return;
  }
}

// element i of a plan's table (twiddles, spectra, products; dfc in memory
// for the packed form)
template <class E>
__device__ __forceinline__ E tab_get(const void *p, i64 i) {
  if constexpr (sizeof(E) == 16 && Emu<E>::v && Tr<E>::cplx)
    return pack(((const dfc *)p)[i]);
  else
    return ((const E *)p)[i];
}
template <class E>
__device__ __forceinline__ void store_elem(void *p, int type, i64 idx, E v,
                                           bool acc, int scale = 0) {
  if constexpr (Emu<E>::v)
    store_as<dfc>(p, type, idx, unpack(v), acc, scale);
  else
    store_as<float2>(p, type, idx, make_float2(v.x, v.y), acc);
}

// ---- float64 <-> packed double-float in the register kernels.  A vector
// is scaled by 2^-s, s = its largest exponent minus the bias, so its largest
// element sits at 2^0 .. 2^1 and results up to 2^127 of it fit; elements more
// than 2^126 below it flush to zero, the tails of those more than 2^74 below
// it (as the tile conversions, d2df_scaled).
// A vector holding Inf or NaN: with truncated heads s = 896 maps the exponent
// field of Inf / NaN to float's, so those elements stay Inf / NaN; with rounded
// ones (a carry would leave that field) s = kDfNonFinite, and those elements
// enter the transform as NaN (rx_in).
constexpr int kDfNonFinite = 0x7FF - 1023;
// largest (hi & 0x7fffffff) of a vector's words >> 20 -> s
template <bool RN> __device__ __forceinline__ int df_scale(int emax) {
  return !RN && emax >= 0x7FF ? 896 : emax - 1023;
}
// s for which no result can leave the float64 range (results lie within
// 2^-127 .. 2^127 of 2^s)
__device__ __forceinline__ bool df_scale_plain(int s) {
  return s >= -890 && s <= 890;
}
// d 2^-s as h + l.  RN (finite d): h is d rounded to 24 significand bits
// (halves away from zero), l the remainder, at most 2^28 units of d's last
// place, rounded to a float: h + l is within 2^-49 |d|.  Otherwise h is
// truncated, l the other 29 bits, h + l within 2^-48 |d|, with fewer
// operations.  The long-vector transforms take RN, as their loads of
// gathered and converted elements (d2df) always did (Toeplitz(3000, 5001) on
// real data: 1.02e-14 from 64 bits, truncated 1.18e-14; chain adjoint 2^18 x
// 32 491 us, truncated 484); in the Kron modes' kernels, whose loads always
// truncated, it would cost 3 % of the FP64 form (2147 -> 2211 us).
// base = s + 896; thr, thl = the smallest high words (sign cleared) whose
// head and whose tail do not flush.
template <bool RN>
__device__ __forceinline__ void d2hl(double d, int base, int thr, int thl,
                                     float &h, float &l) {
  const unsigned hi = (unsigned)__double2hiint(d),
                 lo = (unsigned)__double2loint(d);
  const unsigned sg = hi & 0x80000000u;
  unsigned t;  // exponent field, rebased, and 23 significand bits
  float r;     // the remainder: its units are 2^(ef - 127 - 52)
  if constexpr (RN) {
    // the next bit is rounded in; a carry moves into the exponent as it
    // should and leaves a negative remainder (ef: the field before it)
    t = (__funnelshift_l(lo, hi, 4) - (((unsigned)base << 24) - 1u)) >> 1;
    const unsigned f =
        (((hi << 3) - ((unsigned)(base + 52) << 23)) & 0x7F800000u) | sg;
    r = (float)((int)(lo << 3) >> 3) * __int_as_float((int)f);
  } else {
    t = __funnelshift_l(lo, hi, 3) - ((unsigned)base << 23);
    r = (float)(lo & 0x1FFFFFFFu) *
        __int_as_float((int)((t & 0x7F800000u) - (52u << 23)));
    r = __int_as_float(__float_as_int(r) | (int)sg);
  }
  const int mag = (int)(hi & 0x7FFFFFFFu);
  h = mag >= thr ? __int_as_float((int)(t | sg)) : 0.f;
  l = mag >= thl ? r : 0.f;
}
// (h + l) 2^s as a float64, rounded to nearest: h's bits widened exactly, l
// converted to units in the last place of that float64 and added to its bit
// pattern (an integer addition: carries move into the exponent as they
// should).  bias = (s + 896) << 20; s plain (df_scale_plain).  A head that is
// Inf or NaN (from the operator's data or an overflow) stays Inf or NaN.
__device__ __forceinline__ double hl2d(float h, float l, int bias) {
  const unsigned u = (unsigned)__float_as_int(h);
  const unsigned eb = u & 0x7F800000u;
  // +-2^(52 - e) in two factors: one unit of the result's last place is
  // 2^(e - 52).  The first is a normal float for every normal h and brings
  // every l, subnormal ones too, to 2^-23 or less (0 for Inf and NaN: n = 0).
  const float w =
      __int_as_float((int)(((255u << 23) - eb) | (u & 0x80000000u)));
  int n = __float2int_rn((l * w) * 2251799813685248.f);
  // below a power of two the spacing halves
  if ((u & 0x007FFFFFu) == 0u && n < 0) n += n;
  unsigned hi = ((unsigned)((int)u >> 3) & 0x8FFFFFFFu) + (unsigned)bias;
  if (eb == 0x7F800000u) hi |= 0x7FF00000u;
  const unsigned lo = u << 29;
  i64 b = (i64)(((unsigned long long)hi << 32) | lo) + (i64)n;
  if (eb == 0u) b = 0;
  return __longlong_as_double(b);
}
// ---- 64-bit fixed point for the register FWHT of float64 data: sums and
// differences only, so points scaled to below 2^(63 - W) take W levels
// without rounding (an addition is 2 integer instructions where an
// unnormalised double-float one is 8, and they issue at the same rate:
// measured 64 int64 additions per clock and SM).  Only the W levels of a
// pass are provided for: the points are rounded to nearest when they are
// converted and again, W bits down, between two passes (rf_pass).  A result
// is off by at most half a unit of each rounding, summed over the points the
// levels after it add up: 3 2^-48 of the vector's largest element at 4096
// points if every rounding agrees (6e-17 of the largest result measured on
// random data), and the final rounding.  (Providing for all K levels at the
// conversion, as sums without any rounding would need, leaves 2^(K - 62) of
// the largest element for each of 2^K points of one sign: one element of 1 on
// a background of 1e-6 then came out 2e-12 off.)
struct fx {
  i64 v;
};
__device__ __forceinline__ fx addv(fx a, fx b) { return fx{a.v + b.v}; }
__device__ __forceinline__ fx subv(fx a, fx b) { return fx{a.v - b.v}; }
// d as fixed point: emax the largest exponent field of the vector, W the
// levels of the first pass
__device__ __forceinline__ fx d2fx(double d, int emax, int W) {
  const unsigned hi = (unsigned)__double2hiint(d),
                 lo = (unsigned)__double2loint(d);
  const int ex = (int)((hi >> 20) & 0x7FFu);
  // significand with its leading bit at bit 63, then down to weight
  // 2^(63 - W) for the largest exponent, the last bit shifted out rounded in;
  // zeros and subnormals vanish
  const unsigned mh = __funnelshift_l(lo, hi, 11) | 0x80000000u;
  const unsigned long long u =
      ((unsigned long long)mh << 32) | (unsigned)(lo << 11);
  const unsigned n = ex ? (unsigned)(emax - ex + W) : 64u;
  unsigned long long w;  // (a shift by 64 or more gives 0)
  asm("shr.u64 %0, %1, %2;" : "=l"(w) : "l"(u), "r"(n));
  const i64 s = (i64)((int)hi >> 31);
  return fx{(((i64)w ^ s) + (i64)(1u + (hi >> 31))) >> 1};
}
// fixed point to float64 after K levels, rounded to nearest; plain: no
// result can leave the float64 range (emax between 80 and 2020)
__device__ __forceinline__ double fx2d(fx a, int emax, int K, bool plain) {
  const i64 s = a.v >> 63;
  const unsigned long long u = (unsigned long long)((a.v ^ s) - s);
  const unsigned uh = (unsigned)(u >> 32), ul = (unsigned)u;
  const int lz = uh ? __clz((int)uh) : 32 + __clz((int)ul);
  const unsigned long long n = u << (lz & 63);  // leading bit at bit 63
  const int e = emax + K + 1 - lz;              // exponent field
  // 53 bits, the implicit one adding 1 to the exponent; rounding carries
  unsigned long long b = (n >> 11) + ((n >> 10) & 1ull);
  unsigned bh = (unsigned)(b >> 32) + ((unsigned)(e - 1) << 20);
  unsigned bl = (unsigned)b;
  if (!plain) {
    if (e <= 0) bh = bl = 0u;
    if (e >= 0x7FF) {
      bh = 0x7FF00000u;
      bl = 0u;
    }
  }
  if (u == 0) bh = bl = 0u;
  bh |= (unsigned)(int)s & 0x80000000u;
  return __hiloint2double((int)bh, (int)bl);
}

// the largest exponent word of raw points
__device__ __forceinline__ int raw_hi(double d) {
  return __double2hiint(d) & 0x7FFFFFFF;
}

}  // namespace fmk
