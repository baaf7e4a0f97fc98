// Double-float ("float-float") arithmetic for FP64-accurate products on the
// FP32 pipes.
//
// A value is hi + lo with |lo| <= ulp(hi)/2 (about 48 significant bits).
// Addition uses Knuth's TwoSum, multiplication the FMA-based TwoProduct,
// each followed by a fast renormalisation (Dekker 1971; Knuth, TAOCP vol. 2,
// sec. 4.2.2).  On GB300 the FP32 pipes are roughly 64x faster than FP64,
// so a double-float butterfly (about 20 FP32 operations per output) beats a
// native FP64 one several times over, at relative error ~1e-14 per sweep.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <cmath>

namespace ltm {

struct __align__(8) dfloat {
  float hi, lo;
  __host__ __device__ dfloat() {}
  __host__ __device__ dfloat(int v) : hi((float)v), lo(0.f) {}
  __host__ __device__ dfloat(float h, float l) : hi(h), lo(l) {}
  __host__ __device__ dfloat(double v) {
    hi = (float)v;
    lo = (float)(v - (double)hi);
  }
  __host__ __device__ explicit operator double() const { return (double)hi + (double)lo; }
};

__device__ __forceinline__ dfloat df_renorm(float s, float e) {
  float h = s + e;
  return dfloat(h, e - (h - s));
}

__device__ __forceinline__ dfloat operator+(dfloat a, dfloat b) {
  float s = a.hi + b.hi;
  float bb = s - a.hi;
  float e = (a.hi - (s - bb)) + (b.hi - bb);
  e += a.lo + b.lo;
  return df_renorm(s, e);
}

__device__ __forceinline__ dfloat operator*(dfloat a, dfloat b) {
  float p = a.hi * b.hi;
  float e = fmaf(a.hi, b.hi, -p);
  e = fmaf(a.hi, b.lo, e);
  e = fmaf(a.lo, b.hi, e);
  return df_renorm(p, e);
}

// a * b + c with one renormalisation (TwoProduct by FMA, then TwoSum)
__device__ __forceinline__ dfloat df_fma(dfloat a, dfloat b, dfloat c) {
  float p = a.hi * b.hi;
  float pe = fmaf(a.hi, b.hi, -p);
  pe = fmaf(a.hi, b.lo, pe);
  pe = fmaf(a.lo, b.hi, pe);
  float s = p + c.hi;
  float bb = s - p;
  float se = (p - (s - bb)) + (c.hi - bb);
  se += pe + c.lo;
  return df_renorm(s, se);
}

// df_fma without the final renormalisation: hi + lo still carries the exact
// TwoSum error, but |lo| may exceed ulp(hi)/2 by a few ulps.  For chains of
// a few such steps (the butterfly levels of one round) followed by df_norm;
// the operands' lo enter only as correction terms, so accuracy is unchanged
// up to a few units of 2^-48.
__device__ __forceinline__ dfloat df_fma_unnorm(dfloat a, dfloat b, dfloat c) {
  float p = a.hi * b.hi;
  float pe = fmaf(a.hi, b.hi, -p);
  pe = fmaf(a.hi, b.lo, pe);
  pe = fmaf(a.lo, b.hi, pe);
  float s = p + c.hi;
  float bb = s - p;
  float se = (p - (s - bb)) + (c.hi - bb);
  se += pe + c.lo;
  return dfloat(s, se);
}

__device__ __forceinline__ dfloat df_norm(dfloat a) { return df_renorm(a.hi, a.lo); }

__device__ __forceinline__ dfloat& operator+=(dfloat& a, dfloat b) {
  a = a + b;
  return a;
}
__device__ __forceinline__ dfloat& operator*=(dfloat& a, dfloat b) {
  a = a * b;
  return a;
}

// Double-float values two to a lane pair: hi words in one float2, lo words in
// another.  df2_fma_unnorm is df_fma_unnorm on both lanes with the
// same operation sequence (so the same results), on the packed FP32 pipes;
// differences are taken as fma(b, -1, a), and -p comes from -r.hi, so no
// operand needs a separate negation.
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
__device__ __forceinline__ void df2_fma_unnorm(float2 rh, float2 rl, float2 rhn, float2 xh, float2 xl, float2 yh,
                                               float2 yl, float2& oh, float2& ol) {
  const float2 np = __fmul2_rn(rhn, xh);  // -p, p = r.hi x.hi
  float2 pe = __ffma2_rn(rh, xh, np);     // r.hi x.hi - p (exact)
  pe = __ffma2_rn(rh, xl, pe);
  pe = __ffma2_rn(rl, xh, pe);
  const float2 sm = sub2(yh, np);            // p + y.hi
  const float2 bb = __fadd2_rn(sm, np);      // s - p
  const float2 t = sub2(sm, bb);             // s - bb
  const float2 e2 = sub2(yh, bb);            // y.hi - bb
  const float2 se = sub2(e2, __fadd2_rn(np, t));  // (p - (s - bb)) + (y.hi - bb)
  oh = sm;
  ol = __fadd2_rn(se, __fadd2_rn(pe, yl));
}

// x * w on both lanes (operator*, renormalised), w = (wh, wl)
__device__ __forceinline__ void df2_mul(float2 xh, float2 xl, float2 wh, float2 wl, float2& oh, float2& ol) {
  const float2 np = __fmul2_rn(xh, make_float2(-wh.x, -wh.y));  // -p
  float2 e = __ffma2_rn(xh, wh, np);
  e = __ffma2_rn(xh, wl, e);
  e = __ffma2_rn(xl, wh, e);
  oh = sub2(e, np);                  // p + e
  ol = sub2(e, __fadd2_rn(oh, np));  // e - (h - p)
}

// A constant factor of a result rounded to FP32 once (scale_round): f64, and
// the same as two * hl with `two` a power of two near its square root, so
// that partial products stay near the result's exponent range.  A factor that
// does not fit (zero, negative or not finite ones too) has a NaN for `two`,
// which no range check passes: every value then takes the FP64 form.
struct ScaleF {
  double f64;
  float two;
  dfloat hl;
};
inline bool scale_fits(double S) {
  int e = 0;
  std::frexp(S, &e);
  return std::isfinite(S) && S > 0 && e > -120 && e < 120;
}
inline ScaleF scale_factor(double S) {
  ScaleF p{S, std::nanf(""), dfloat(1.0)};
  if (scale_fits(S)) {
    int e = 0;
    std::frexp(S, &e);
    p.two = std::ldexp(1.f, e / 2);
    p.hl = dfloat(S / (double)p.two);
  }
  return p;
}

// The FP64 form of scale_round.  Not inlined: as part of the caller it would be
// predicated, and a predicated FP64 instruction takes its slot on the pipe.
static __device__ __noinline__ float scale_round_f64(float vh, float vl, double t, double f) {
  return (float)(((double)vh + (double)vl) * t * f);
}
static __device__ __noinline__ float scale_round_f64(float vh, float vl, float th, float tl, double f) {
  return (float)(((double)vh + (double)vl) * ((double)th + (double)tl) * f);
}
__device__ __forceinline__ float hi_of(float v) { return v; }
__device__ __forceinline__ float hi_of(dfloat v) { return v.hi; }
__device__ __forceinline__ float lo_of(float) { return 0.f; }
__device__ __forceinline__ float lo_of(dfloat v) { return v.lo; }

// Whether the two-word products a = v * two, p = a * sc and q = p * post hold
// all of a result: a has to be exact, the error terms of p representable, and q
// neither infinite (also: p infinite or NaN) nor where its own error terms
// would be lost.
__device__ __forceinline__ bool scale_in_range(float a, float p, float q) {
  return fabsf(a) > 1e-35f && fabsf(p) > 1e-24f && fabsf(q) > 1e-33f && fabsf(q) < 1e38f;
}

// (v * sc) * post rounded to FP32 once: the products' rounding errors are
// carried along (TwoProduct by FMA), so the result is that of FP64 arithmetic
// to within the last rounding, without the FP64 pipe (two lanes per clock and
// SM, conversions included).  Infinities, NaN and products near the ends of
// the exponent range take the FP64 form.
__device__ __forceinline__ float scale_round(float v, dfloat sc, const ScaleF& post) {
  const float a = v * post.two;
  const float p = a * sc.hi;
  if (v == 0.f && p == 0.f) return p;
  const float q = p * post.hl.hi;
  if (!scale_in_range(a, p, q)) return scale_round_f64(hi_of(v), lo_of(v), sc.hi, sc.lo, post.f64);
  const float e = fmaf(a, sc.lo, fmaf(a, sc.hi, -p));
  return q + fmaf(e, post.hl.hi, fmaf(p, post.hl.lo, fmaf(p, post.hl.hi, -q)));
}

// the same for a double-float value
__device__ __forceinline__ float scale_round(dfloat v, dfloat sc, const ScaleF& post) {
  const float a = v.hi * post.two;
  const float p = a * sc.hi;
  if (v.hi == 0.f && p == 0.f) return p;
  const float q = p * post.hl.hi;
  if (!scale_in_range(a, p, q)) return scale_round_f64(hi_of(v), lo_of(v), sc.hi, sc.lo, post.f64);
  const float e = fmaf(v.lo * post.two, sc.hi, fmaf(a, sc.lo, fmaf(a, sc.hi, -p)));
  return q + fmaf(e, post.hl.hi, fmaf(p, post.hl.lo, fmaf(p, post.hl.hi, -q)));
}

// An FP64 weight as a double-float, by integer operations (the hi word
// truncated to 24 bits, the lo word the 29 bits below), so that nothing runs
// on the FP64 pipe but the rare cases; false where it does not fit.
__device__ __forceinline__ bool weight_df(double t, dfloat& w) {
  const uint32_t up = (uint32_t)__double2hiint(t), dn = (uint32_t)__double2loint(t);
  const int e = (int)((up >> 20) & 0x7ffu) - 1023;
  const uint32_t sign = up & 0x80000000u;
  const uint32_t m23 = ((up & 0xfffffu) << 3) | (dn >> 29);
  w.hi = __uint_as_float(sign | ((uint32_t)(e + 127) << 23) | m23);
  w.lo = __uint2float_rn(dn & 0x1fffffffu) * __uint_as_float(sign | ((uint32_t)(e - 52 + 127) << 23));
  return e >= -70 && e <= 90;
}

// v * t * post for an FP64 weight t
template <class V>
__device__ __forceinline__ float scale_round(V v, double t, const ScaleF& post) {
  dfloat w;
  if (!weight_df(t, w)) return scale_round_f64(hi_of(v), lo_of(v), t, post.f64);
  return scale_round(v, w, post);
}

// v * t rounded to FP32 once
__device__ __forceinline__ float scale_round(float v, double t) {
  dfloat w;
  const bool fits = weight_df(t, w);
  const float p = v * w.hi;
  if (!fits || !((fabsf(p) > 1e-24f && fabsf(p) < 1e38f) || v == 0.f)) return scale_round_f64(v, 0.f, t, 1.0);
  return p + fmaf(v, w.lo, fmaf(v, w.hi, -p));
}

// Forward-mode tangent pair (value, derivative with respect to one
// parameter): the adjoint's tangent products of the aux-bit chains run the
// chain steps in this type, d(a b) = da b + a db, d(a + b) = da + db.  Both
// parts are double-float, so the products run on the FP32 pipes at
// FP64-level accuracy (~1e-14), in the FP32 exponent range (the chains
// normalise their steps as the other double-float products do).
struct __align__(16) tangent {
  dfloat v, d;
  __host__ __device__ tangent() {}
  __host__ __device__ tangent(double x) : v(x), d(0.0) {}
  __host__ __device__ tangent(double x, double dx) : v(x), d(dx) {}
  __host__ __device__ tangent(dfloat x, dfloat dx) : v(x), d(dx) {}
};

__device__ __forceinline__ tangent operator+(tangent a, tangent b) { return tangent(a.v + b.v, a.d + b.d); }
__device__ __forceinline__ tangent operator*(tangent a, tangent b) {
  return tangent(a.v * b.v, df_fma(a.d, b.v, a.v * b.d));
}
__device__ __forceinline__ tangent& operator+=(tangent& a, tangent b) {
  a = a + b;
  return a;
}
__device__ __forceinline__ tangent& operator*=(tangent& a, tangent b) {
  a = a * b;
  return a;
}

}  // namespace ltm
