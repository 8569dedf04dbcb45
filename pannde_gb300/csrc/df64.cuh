// df64.cuh -- double-float ("float-float") arithmetic on the FP32 pipes.
//
// A value is the unevaluated sum hi + lo of two floats with |lo| <= ulp(hi)/2,
// a 48-bit significand.  The operations restate published error-free
// transformations:
//   two_sum        Knuth, TAOCP vol. 2, 4.2.2 (6 flops, exact a+b = s+e)
//   quick_two_sum  Dekker 1971 (3 flops, exact when |a| >= |b|)
//   two_prod       with a fused multiply-add (2 flops, exact a*b = p+e)
//   add            the "sloppy" double-double add of Hida, Li & Bailey,
//                  "Algorithms for quad-double precision floating point
//                  arithmetic" (2001): two_sum of the high words, add the low
//                  words, renormalise (11 flops)
//   mul            two_prod of the high words plus the cross terms, renormalised
//   madd           a*b + c with one renormalisation
// Every step uses the _rn intrinsics so the compiler can neither contract a
// product into a following add nor reorder the sums the algorithms rely on.
// Values must stay inside the float exponent range (about 1e-38..3e38).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace pn {

// Two floats worked on by one instruction (Blackwell's packed add, multiply
// and fused multiply-add): the pipe does the same number of operations a
// second as with single ones (measured 3.8e13 elements/s for both) but the
// pair takes one issue slot instead of two.  Each half is rounded as the
// scalar operation rounds it.
struct f32x2 {
  unsigned long long v;
  __device__ __forceinline__ f32x2() : v(0ull) {}
  __device__ __forceinline__ f32x2(float a, float b) { asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b)); }
  __device__ __forceinline__ float half(int h) const {
    float a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
    return h ? b : a;
  }
};

// the operations the algorithms below are written in: one float, or two
__device__ __forceinline__ float fadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float fmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float ffma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float fneg(float a) { return -a; }
__device__ __forceinline__ f32x2 fadd(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f32x2 fsub(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f32x2 fmul(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f32x2 ffma(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ f32x2 fneg(f32x2 a) {
  a.v ^= 0x8000000080000000ull;
  return a;
}
__device__ __forceinline__ f32x2 operator+(f32x2 a, f32x2 b) { return fadd(a, b); }
__device__ __forceinline__ f32x2 operator-(f32x2 a, f32x2 b) { return fsub(a, b); }
__device__ __forceinline__ f32x2 operator*(f32x2 a, f32x2 b) { return fmul(a, b); }
__device__ __forceinline__ f32x2 operator-(f32x2 a) { return fneg(a); }
__device__ __forceinline__ f32x2 madd(f32x2 a, f32x2 b, f32x2 c) { return ffma(a, b, c); }

// native types: the compiler contracts a*b + c into one FMA
__device__ __forceinline__ float madd(float a, float b, float c) { return a * b + c; }
__device__ __forceinline__ double madd(double a, double b, double c) { return a * b + c; }

// two doubles (no packed instructions: each half on its own)
struct f64x2 {
  double a, b;
  __device__ __forceinline__ f64x2() : a(0.), b(0.) {}
  __device__ __forceinline__ f64x2(double x, double y) : a(x), b(y) {}
};
__device__ __forceinline__ f64x2 operator+(f64x2 x, f64x2 y) { return f64x2(x.a + y.a, x.b + y.b); }
__device__ __forceinline__ f64x2 operator-(f64x2 x, f64x2 y) { return f64x2(x.a - y.a, x.b - y.b); }
__device__ __forceinline__ f64x2 operator*(f64x2 x, f64x2 y) { return f64x2(x.a * y.a, x.b * y.b); }
__device__ __forceinline__ f64x2 operator-(f64x2 x) { return f64x2(-x.a, -x.b); }
__device__ __forceinline__ f64x2 madd(f64x2 x, f64x2 y, f64x2 z) { return f64x2(x.a * y.a + z.a, x.b * y.b + z.b); }

// a double-float (F = float), or two side by side (F = f32x2)
template <typename F> struct ddf {
  F hi, lo;
  __device__ __forceinline__ ddf() : hi(), lo() {}
  __device__ __forceinline__ ddf(F h, F l) : hi(h), lo(l) {}
};
using df64 = ddf<float>;
using df64x2 = ddf<f32x2>;

template <typename F> __device__ __forceinline__ ddf<F> two_sum(F a, F b) {
  const F s = fadd(a, b);
  const F bb = fsub(s, a);
  const F e = fadd(fsub(a, fsub(s, bb)), fsub(b, bb));
  return ddf<F>(s, e);
}
// two_sum(a, -b) without forming -b
template <typename F> __device__ __forceinline__ ddf<F> two_diff(F a, F b) {
  const F s = fsub(a, b);
  const F bb = fsub(s, a);
  const F e = fsub(fsub(a, fsub(s, bb)), fadd(b, bb));
  return ddf<F>(s, e);
}

template <typename F> __device__ __forceinline__ ddf<F> quick_two_sum(F a, F b) {
  const F s = fadd(a, b);
  return ddf<F>(s, fsub(b, fsub(s, a)));
}

template <typename F> __device__ __forceinline__ ddf<F> operator+(ddf<F> a, ddf<F> b) {
  ddf<F> s = two_sum(a.hi, b.hi);
  s.lo = fadd(s.lo, fadd(a.lo, b.lo));
  return quick_two_sum(s.hi, s.lo);
}

template <typename F> __device__ __forceinline__ ddf<F> operator-(ddf<F> a) { return ddf<F>(fneg(a.hi), fneg(a.lo)); }

template <typename F> __device__ __forceinline__ ddf<F> operator-(ddf<F> a, ddf<F> b) {
  ddf<F> s = two_diff(a.hi, b.hi);
  s.lo = fadd(s.lo, fsub(a.lo, b.lo));
  return quick_two_sum(s.hi, s.lo);
}

template <typename F> __device__ __forceinline__ ddf<F> operator*(ddf<F> a, ddf<F> b) {
  const F p = fmul(a.hi, b.hi);
  F e = ffma(a.hi, b.hi, fneg(p));
  e = ffma(a.hi, b.lo, e);
  e = ffma(a.lo, b.hi, e);
  return quick_two_sum(p, e);
}

// a*b + c without renormalising the product first: the two_prod error terms
// join c's low word before the one renormalisation (15 flops against 18 for
// a separate mul and add; the same "sloppy" error bound)
template <typename F> __device__ __forceinline__ ddf<F> madd(ddf<F> a, ddf<F> b, ddf<F> c) {
  const F p = fmul(a.hi, b.hi);
  F e = ffma(a.hi, b.hi, fneg(p));
  e = ffma(a.hi, b.lo, e);
  e = ffma(a.lo, b.hi, e);
  ddf<F> s = two_sum(p, c.hi);
  s.lo = fadd(s.lo, fadd(e, c.lo));
  return quick_two_sum(s.hi, s.lo);
}
// Four-term sums of the stencil with one renormalisation at the end: the
// high words go through error-free two_sums, the low words and the errors
// are summed as floats ("lazy" double-float accumulation; 27 flops for
// (b+c)-(a+d) against 33 for three renormalised adds).  The sums stay
// unnormalised (lo not yet bounded by ulp(hi) / 2) until the add that consumes
// them renormalises anyway (3 flops fewer per value); Lazy<T> is T itself for
// the native types.
template <typename F> struct ddf_unnorm {
  F hi, lo;  // hi + lo, |lo| not yet bounded by ulp(hi)/2
};
template <typename T> struct Lazy { using type = T; };
template <typename F> struct Lazy<ddf<F>> { using type = ddf_unnorm<F>; };
template <typename F> __device__ __forceinline__ ddf_unnorm<F> add_lazy(ddf<F> a, ddf<F> b) {
  const ddf<F> s = two_sum(a.hi, b.hi);
  return {s.hi, fadd(s.lo, fadd(a.lo, b.lo))};
}
template <typename F> __device__ __forceinline__ ddf_unnorm<F> sub_lazy(ddf<F> a, ddf<F> b) {
  const ddf<F> s = two_diff(a.hi, b.hi);
  return {s.hi, fadd(s.lo, fsub(a.lo, b.lo))};
}
template <typename F> __device__ __forceinline__ ddf_unnorm<F> add_unnorm(ddf_unnorm<F> a, ddf_unnorm<F> b) {
  const ddf<F> s = two_sum(a.hi, b.hi);
  return {s.hi, fadd(s.lo, fadd(a.lo, b.lo))};
}
template <typename F> __device__ __forceinline__ ddf_unnorm<F> sub_unnorm(ddf_unnorm<F> a, ddf_unnorm<F> b) {
  const ddf<F> s = two_diff(a.hi, b.hi);
  return {s.hi, fadd(s.lo, fsub(a.lo, b.lo))};
}
template <typename F> __device__ __forceinline__ ddf<F> add_uu(ddf_unnorm<F> a, ddf_unnorm<F> b) {
  const ddf<F> s = two_sum(a.hi, b.hi);
  return quick_two_sum(s.hi, fadd(s.lo, fadd(a.lo, b.lo)));
}
template <typename F> __device__ __forceinline__ ddf<F> sub_uu(ddf_unnorm<F> a, ddf_unnorm<F> b) {
  const ddf<F> s = two_diff(a.hi, b.hi);
  return quick_two_sum(s.hi, fadd(s.lo, fsub(a.lo, b.lo)));
}
template <typename F> __device__ __forceinline__ ddf_unnorm<F> to_u(ddf<F> a) { return {a.hi, a.lo}; }
template <typename F> __device__ __forceinline__ ddf<F> norm_u(ddf_unnorm<F> a) { return quick_two_sum(a.hi, a.lo); }
// (b + c) - (a + d)
template <typename F>
__device__ __forceinline__ ddf_unnorm<F> diff22_u(ddf<F> b, ddf<F> c, ddf<F> a, ddf<F> d) {
  return sub_unnorm(add_lazy(b, c), add_lazy(a, d));
}
// (a + b) + (c + d)
template <typename F>
__device__ __forceinline__ ddf_unnorm<F> sum22_u(ddf<F> a, ddf<F> b, ddf<F> c, ddf<F> d) {
  return add_unnorm(add_lazy(a, b), add_lazy(c, d));
}
// (c + d) - (a + b) and (a + b) + (c + d) sharing the pair sums
template <typename F>
__device__ __forceinline__ void diffsum22_u(ddf<F> a, ddf<F> b, ddf<F> c, ddf<F> d, ddf_unnorm<F> &diff,
                                            ddf_unnorm<F> &sum) {
  const ddf_unnorm<F> ab = add_lazy(a, b), cd = add_lazy(c, d);
  diff = sub_unnorm(cd, ab);
  sum = add_unnorm(ab, cd);
}
// (b + c) - (a + d) and (c + d) - (a + b) as (c - a) + (b - d) and
// (c - a) - (b - d): two pair differences shared (38 flops against 54)
template <typename F>
__device__ __forceinline__ void diffdiff22_u(ddf<F> a, ddf<F> b, ddf<F> c, ddf<F> d, ddf_unnorm<F> &dx,
                                             ddf_unnorm<F> &dy) {
  const ddf_unnorm<F> u = sub_lazy(c, a), w = sub_lazy(b, d);
  dx = add_unnorm(u, w);
  dy = sub_unnorm(u, w);
}
// the same for the native types
template <typename T> __device__ __forceinline__ T diff22_u(T b, T c, T a, T d) { return (b + c) - (a + d); }
template <typename T> __device__ __forceinline__ T sum22_u(T a, T b, T c, T d) { return (a + b) + (c + d); }
template <typename T> __device__ __forceinline__ void diffsum22_u(T a, T b, T c, T d, T &diff, T &sum) {
  const T ab = a + b, cd = c + d;
  diff = cd - ab;
  sum = ab + cd;
}
template <typename T> __device__ __forceinline__ void diffdiff22_u(T a, T b, T c, T d, T &dx, T &dy) {
  const T u = c - a, w = b - d;
  dx = u + w;
  dy = u - w;
}
template <typename T> __device__ __forceinline__ T add_unnorm(T a, T b) { return a + b; }
template <typename T> __device__ __forceinline__ T sub_unnorm(T a, T b) { return a - b; }
template <typename T> __device__ __forceinline__ T add_uu(T a, T b) { return a + b; }
template <typename T> __device__ __forceinline__ T sub_uu(T a, T b) { return a - b; }
template <typename T> __device__ __forceinline__ T to_u(T a) { return a; }
template <typename T> __device__ __forceinline__ T norm_u(T a) { return a; }

// c + sum_j a_j * b_j with one renormalisation at the end (the rows of the
// stiffness product): each product's high part joins the running sum through
// an error-free two_sum, its error terms and the low words are summed as
// floats (12 flops per term against madd's 15, the same "sloppy" bound)
template <typename F> __device__ __forceinline__ ddf_unnorm<F> acc_start(ddf<F> c) { return {c.hi, c.lo}; }
template <typename F> __device__ __forceinline__ void acc_madd(ddf_unnorm<F> &s, ddf<F> a, ddf<F> b) {
  const F p = fmul(a.hi, b.hi);
  F e = ffma(a.hi, b.hi, fneg(p));
  e = ffma(a.hi, b.lo, e);
  e = ffma(a.lo, b.hi, e);
  const ddf<F> t = two_sum(s.hi, p);
  s.hi = t.hi;
  s.lo = fadd(s.lo, fadd(t.lo, e));
}
template <typename F> __device__ __forceinline__ ddf<F> acc_end(ddf_unnorm<F> s) { return quick_two_sum(s.hi, s.lo); }
// ... and for the native types: one FMA per term
template <typename T> __device__ __forceinline__ T acc_start(T c) { return c; }
template <typename T> __device__ __forceinline__ void acc_madd(T &s, T a, T b) { s = madd(a, b, s); }
template <typename T> __device__ __forceinline__ T acc_end(T s) { return s; }

__device__ __forceinline__ bool operator==(df64 a, df64 b) { return a.hi == b.hi && a.lo == b.lo; }

// ---- between IEEE double and double-float ---------------------------------
// GB300 converts double <-> float on its FP64 unit, at the FP64 FMA rate; these
// conversions run on the integer and FP32 pipes instead (loads) or keep to
// two conversions and one FP64 add (stores).
//
// split_double: d = hi + lo exactly up to the first 47 significant bits (the
// rest truncated: |d - (hi + lo)| < 2^-46 |d|).  hi keeps d's sign, exponent
// and top 23 fraction bits: the double's exponent field, rebiased from 1023
// to 127, is (e11 - 896) mod 256 = (e11 mod 256) ^ 0x80 whenever the result
// is a normal float, so a funnel shift of the high and low words by 3 and a
// flip of bit 30 give hi's bits.  lo holds the next 23 fraction bits m as
// (P | m) - P with P = sign | hi's exponent - 23, exact by Sterbenz.
// Exact (to those 47 bits) for 2^-102 <= |d| < 2^128 (biased exponents
// 921..1150); d == +-0 and every value outside that range give 0 -- the
// double-float path takes only values its range check admitted (see
// in_df64_range), so this only keeps a stray value from becoming garbage.
__device__ __forceinline__ df64 split_double(double d) {
  const uint32_t hw = (uint32_t)__double2hiint(d), lw = (uint32_t)__double2loint(d);
  const uint32_t f = __funnelshift_l(lw, hw, 3) ^ 0x40000000u;
  const uint32_t hib = (f & 0x7fffffffu) | (hw & 0x80000000u);
  const uint32_t pb = (hib & 0xff800000u) - (23u << 23);
  const float lo = __fsub_rn(__uint_as_float(pb | ((lw >> 6) & 0x7fffffu)), __uint_as_float(pb));
  const bool zero = (((hw >> 20) & 0x7ffu) - 921u) > (1150u - 921u);
  return df64(zero ? 0.f : __uint_as_float(hib), zero ? 0.f : lo);
}

// join_double: hi + lo rounded once to the nearest double (both convert
// exactly; the FP64 add rounds the exact sum)
__device__ __forceinline__ double join_double(df64 v) { return __dadd_rn((double)v.hi, (double)v.lo); }

// join_double_int: hi + lo to a double within one unit in the last place,
// on the integer and FP32 pipes (the FP64 unit converts at its FMA rate).
// For a normalised pair (|lo| <= ulp(hi) / 2) the double of hi is its bits
// rebiased (exponent + 896, fraction moved 29 bits down), and lo adds
// k = lo * 2^(52 - E) units of that double's last place (|k| <= 2^28, the 29
// zero bits below hi's fraction: no carry into the exponent).  When hi is a
// power of two and lo of the other sign the sum falls into the binade below,
// whose unit is half as large: k is counted in those units.  k is formed at
// 2^(53 - E) and halved (rounding half up) otherwise.  Zero gives +0; hi below
// 2^-74 (where the scale factor would leave float's range) takes join_double.
__device__ __forceinline__ double join_double_int(df64 v) {
  const uint32_t hb = __float_as_uint(v.hi), lb = __float_as_uint(v.lo);
  const uint32_t u = hb & 0x7fffffffu;
  if (u == 0u) return 0.0;
  const uint32_t e8 = u >> 23;
  if (e8 < 53u) return join_double(v);
  const uint32_t hw = ((u >> 3) + 0x38000000u) | (hb & 0x80000000u);
  const uint32_t lw = hb << 29;
  const int kk = __float2int_rn(__fmul_rn(v.lo, __uint_as_float((307u - e8) << 23)));
  const bool opposite = ((hb ^ lb) & 0x80000000u) != 0u;
  const int mag = abs(kk);
  const int step = ((u & 0x7fffffu) == 0u && opposite) ? mag : (mag + 1) >> 1;
  const long long bits = (long long)(((unsigned long long)hw << 32) | lw) + (opposite ? -step : step);
  return __longlong_as_double(bits);
}

// float_bits_to_double: a normal float's exact double by its bits (exponent
// rebiased by +896, fraction moved 29 bits down); 0 for +-0.  A subnormal
// float (below 2^-126, outside every range the double-float path admits)
// comes out wrong by at most 2^-126.
__device__ __forceinline__ double float_bits_to_double(float f) {
  const uint32_t b = __float_as_uint(f), u = b & 0x7fffffffu;
  const uint32_t hw = u ? (((u >> 3) + 0x38000000u) | (b & 0x80000000u)) : 0u;
  return __hiloint2double((int)hw, (int)(b << 29));
}

// base + (hi + lo): the pair added to a double by two FP64 adds of its exact
// halves (within one unit in the last place of the sum)
__device__ __forceinline__ double add_pair(double base, df64 inc) {
  return __dadd_rn(__dadd_rn(base, float_bits_to_double(inc.hi)), float_bits_to_double(inc.lo));
}

// whether d is 0 or its biased exponent lies in [e_lo, e_hi]: the values the
// double-float path of the FP64 form takes (bounds chosen by the host so that
// every product with the step's coefficients stays within 2^+-100)
__device__ __forceinline__ bool in_df64_range(double d, uint32_t e_lo, uint32_t e_hi) {
  const uint32_t hw = (uint32_t)__double2hiint(d);
  const uint32_t e = (hw >> 20) & 0x7ffu;
  const bool zero = (hw & 0x7fffffffu) == 0u && __double2loint(d) == 0;
  return zero || (e - e_lo) <= (e_hi - e_lo);
}

}  // namespace pn
