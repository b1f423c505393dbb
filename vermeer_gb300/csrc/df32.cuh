// df32.cuh - float32 results of float64 functions without the float64 pipe.
//
// The reference mode evaluates its transcendentals as math/sincos.go does, in
// float64, and rounds to float32.  GB300 retires about two float64 operations
// a clock and SM against 128 float32 ones, and k_shade spent 80% of its cycles
// with that pipe busy.  Here a value is a pair of float32 (double-float, Dekker
// 1971: an unevaluated sum of about 48 bits), computed to a relative error
// below 2^-40, and Ziv's rounding test (1991) decides: if the value less and
// plus its error bound round to the same float32, that is the float32 of the
// exact result and of float64's, whose own error is far inside the bound;
// otherwise (about one value in 2^12) the float64 function is called.  So every
// result is the one the float64 path gives, bit for bit
// (tests/test_reference_functions.py).
//
// sin and cos: Cody-Waite reduction by pi/2 in four parts, then their Taylor
// series, the leading coefficients as pairs.  acos and atan: CUDA's float32
// value y0, corrected by one Newton step on cos y = x and tan y = x with sin y0
// and cos y0 as pairs (the step's own error is y0's squared, about 2^-45).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace vmr {
namespace {

struct DF {
  float h, l;
};
// Sums and products with their rounding errors.  df_fast: |a| >= |b| or a = 0.
__device__ __forceinline__ DF df_fast(float a, float b) {
  const float s = a + b;
  return DF{s, b - (s - a)};
}
__device__ __forceinline__ DF df_sum(float a, float b) {
  const float s = a + b, t = s - a;
  return DF{s, (a - (s - t)) + (b - t)};
}
__device__ __forceinline__ DF df_prod(float a, float b) {
  const float p = a * b;
  return DF{p, __fmaf_rn(a, b, -p)};
}
__device__ __forceinline__ DF df_add(DF a, DF b) {
  const DF s = df_sum(a.h, b.h);
  return df_fast(s.h, s.l + (a.l + b.l));
}
__device__ __forceinline__ DF df_mul(DF a, DF b) {
  const DF p = df_prod(a.h, b.h);
  return df_fast(p.h, __fmaf_rn(a.h, b.l, __fmaf_rn(a.l, b.h, p.l)));
}
__device__ __forceinline__ DF df_neg(DF a) { return DF{-a.h, -a.l}; }
__device__ __forceinline__ DF df_sqrt(DF v) {
  if (v.h == 0.0f) return DF{0.0f, 0.0f};
  const float s = sqrtf(v.h);
  return df_fast(s, (__fmaf_rn(-s, s, v.h) + v.l) / (s + s));
}
// Ziv's test: out is the float32 of every value within err of v, or false.
__device__ __forceinline__ bool df_round(DF v, float err, float& out) {
  out = v.h + (v.l - err);
  return out == v.h + (v.l + err);
}

// Series on |r| <= pi/4 (truncated below 2^-45 of the result).
__device__ __forceinline__ DF df_sin_series(DF r) {
  const DF z = df_mul(r, r);
  const float t = z.h;
  const float tail = t * __fmaf_rn(t, __fmaf_rn(t, 0x1.612462p-33f, -0x1.ae6456p-26f), 0x1.71de3ap-19f);  // 1/13!, -1/11!, 1/9!
  DF q = df_add(DF{-0x1.a01a02p-13f, 0x1.7f97fap-39f}, DF{tail, 0.0f});          // -1/7!
  q = df_add(DF{0x1.111112p-7f, -0x1.dddddep-32f}, df_mul(z, q));                // 1/5!
  q = df_add(DF{-0x1.555556p-3f, 0x1.555556p-28f}, df_mul(z, q));               // -1/3!
  return df_add(r, df_mul(df_mul(r, z), q));
}
__device__ __forceinline__ DF df_cos_series(DF r) {
  const DF z = df_mul(r, r);
  const float t = z.h;
  const float tail = t * __fmaf_rn(t, __fmaf_rn(t, -0x1.93974ap-37f, 0x1.1eed8ep-29f), -0x1.27e4fcp-22f);  // -1/14!, 1/12!, -1/10!
  DF q = df_add(DF{0x1.a01a02p-16f, -0x1.7f97fap-42f}, DF{tail, 0.0f});         // 1/8!
  q = df_add(DF{-0x1.6c16c2p-10f, 0x1.27d27ep-35f}, df_mul(z, q));              // -1/6!
  q = df_add(DF{0x1.555556p-5f, -0x1.555556p-30f}, df_mul(z, q));               // 1/4!
  return df_add(df_add(DF{1.0f, 0.0f}, DF{-0.5f * z.h, -0.5f * z.l}), df_mul(df_mul(z, z), q));
}
// x = n pi/2 + r for |x| < 12.  pi/2 as 20 + 20 + 20 bits and a rest: n times
// each of the first three is exact.
__device__ __forceinline__ DF df_reduce(float x, int& n) {
  const float k = rintf(x * 0.636619772f);
  n = (int)k;
  const DF a = df_sum(x, -k * 0x1.921fap+0f);
  const DF b = df_sum(a.h, -k * 0x1.54442p-20f);
  const DF c = df_sum(b.h, -k * 0x1.a308cp-41f);
  return df_fast(c.h, (a.l + b.l) + (c.l - k * 0x1.313198p-61f));
}
__device__ __forceinline__ void df_sincos(float x, DF& s, DF& c) {
  int n;
  const DF r = df_reduce(x, n);
  const DF a = df_sin_series(r), b = df_cos_series(r);
  s = (n & 1) ? b : a;
  c = (n & 1) ? a : b;
  if (n & 2) s = df_neg(s);
  if ((n + 1) & 2) c = df_neg(c);
}
constexpr float kDfErr = 0x1p-38f;  // relative bound taken; measured below 2^-42

// The float64 functions, out of line: they are the rare path.
__device__ __noinline__ float sin64(float x) { return (float)sin((double)x); }
__device__ __noinline__ float cos64(float x) { return (float)cos((double)x); }
__device__ __noinline__ float acos64(float x) { return (float)acos((double)x); }
__device__ __noinline__ float atan64(float x) { return (float)atan((double)x); }

// (float)sin((double)x) and (float)cos((double)x).
__device__ __forceinline__ void sincos_rn(float x, float& s, float& c) {
  if (fabsf(x) < 12.0f && fabsf(x) > 1e-15f) {
    DF a, b;
    df_sincos(x, a, b);
    const bool oks = df_round(a, kDfErr * fabsf(a.h), s), okc = df_round(b, kDfErr * fabsf(b.h), c);
    if (oks && okc) return;
  }
  s = sin64(x);
  c = cos64(x);
}
__device__ __forceinline__ float sin_rn(float x) {
  if (fabsf(x) < 12.0f && fabsf(x) > 1e-15f) {
    int n;
    const DF r = df_reduce(x, n);
    const DF a = (n & 1) ? df_cos_series(r) : df_sin_series(r);
    float f;
    if (df_round(a, kDfErr * fabsf(a.h), f)) return (n & 2) ? -f : f;
  }
  return sin64(x);
}
__device__ __forceinline__ float cos_rn(float x) {
  if (fabsf(x) < 12.0f) {
    int n;
    const DF r = df_reduce(x, n);
    const DF a = (n & 1) ? df_sin_series(r) : df_cos_series(r);
    float f;
    if (df_round(a, kDfErr * fabsf(a.h), f)) return ((n + 1) & 2) ? -f : f;
  }
  return cos64(x);
}
// (float)acos((double)x), x in [-1, 1] or NaN.  With y0 near acos |x|:
// |x| >= 1/2: 1 - cos y0 = 2 sin^2(y0/2), against the exact 1 - |x|; below,
// cos y0 against |x|.
__device__ __forceinline__ float acos_rn(float x) {
  const float a = fabsf(x);
  if (a < 1.0f) {
    const float y0 = acosf(a), u = 1.0f - a;
    float num;
    if (a >= 0.5f) {
      const DF s = df_sin_series(DF{0.5f * y0, 0.0f});
      const DF v = df_mul(s, s);
      num = (u - 2.0f * v.h) - 2.0f * v.l;
    } else {
      int n;
      const DF r = df_reduce(y0, n);  // n = 1: cos y0 = -sin r
      const DF s = df_sin_series(r);
      num = -((s.h + a) + s.l);
      if (n != 1) num = __int_as_float(0x7fc00000);
    }
    DF y = df_fast(y0, num / sqrtf(u * (1.0f + a)));
    if (x < 0.0f) y = df_add(DF{0x1.921fb6p+1f, -0x1.777a5cp-24f}, df_neg(y));  // pi - y
    float f;
    if (df_round(y, kDfErr * fabsf(y.h), f)) return f;
  }
  return acos64(x);
}
// (float)atan((double)x): tan(y - y0) = (x cos y0 - sin y0) / (cos y0 + x sin y0).
__device__ __forceinline__ float atan_rn(float x) {
  if (fabsf(x) < 1e6f && fabsf(x) > 1e-6f) {
    const float y0 = atanf(x);
    DF s, c;
    df_sincos(y0, s, c);
    const DF p = df_prod(x, c.h);
    const float num = (p.h - s.h) + (__fmaf_rn(x, c.l, p.l) - s.l);
    const DF y = df_fast(y0, num / __fmaf_rn(x, s.h, c.h));
    float f;
    if (df_round(y, kDfErr * fabsf(y.h), f)) return f;
  }
  return atan64(x);
}

// ---- the QMC sequences' fractions k / 2^52 (k <= 2^52)
__device__ __forceinline__ float frac52(uint64_t k) { return __ull2float_rn(k) * 0x1p-52f; }
__device__ __forceinline__ double frac52d(uint64_t k) { return (double)k / 4503599627370496.0; }
__device__ __forceinline__ DF df_int(int64_t k) {  // |k| <= 2^52
  const float h = __ll2float_rn(k);
  return DF{h, __ll2float_rn(k - __float2ll_rn(h))};
}
__device__ __forceinline__ DF df_frac52(uint64_t k) {
  const DF v = df_int((int64_t)k);
  return DF{v.h * 0x1p-52f, v.l * 0x1p-52f};
}
constexpr uint64_t kOne52 = 1ull << 52;

// CosineHemisphere (math/sample/sample.go:18-27) of r0 = k0 / 2^52, r1 =
// k1 / 2^52 in float64, rounded: (float)(sqrt(1-r0) cos(2 pi r1)), the same
// with sin, (float)sqrt(r0).
__device__ __noinline__ void cosine_hemisphere64(uint64_t k0, uint64_t k1, float& x, float& y, float& z) {
  const double r0 = frac52d(k0), r1 = frac52d(k1);
  const double r = sqrt(1 - r0), th = 2 * 3.14159265358979323846 * r1;
  x = (float)(r * cos(th));
  y = (float)(r * sin(th));
  z = (float)sqrt(r0);
}
__device__ __forceinline__ void cosine_hemisphere(uint64_t k0, uint64_t k1, float& x, float& y, float& z) {
  const DF r = df_sqrt(df_frac52(kOne52 - k0)), w = df_sqrt(df_frac52(k0));
  // 4 r1 = n + f, |f| <= 1/2, both exact
  const int n = (int)((k1 + (1ull << 49)) >> 50);
  const int64_t f = (int64_t)k1 - ((int64_t)n << 50);
  const DF v = df_int(f);
  const DF a = df_mul(DF{v.h * 0x1p-50f, v.l * 0x1p-50f}, DF{0x1.921fb6p+0f, -0x1.777a5cp-25f});
  const DF s0 = df_sin_series(a), c0 = df_cos_series(a);
  DF s = (n & 1) ? c0 : s0, c = (n & 1) ? s0 : c0;
  if (n & 2) s = df_neg(s);
  if ((n + 1) & 2) c = df_neg(c);
  s = df_mul(r, s);
  c = df_mul(r, c);
  // float64's angle is rounded, so near a zero its error is absolute
  const float e = 0x1p-44f * r.h;
  const bool okx = df_round(c, __fmaf_rn(kDfErr, fabsf(c.h), e), x), oky = df_round(s, __fmaf_rn(kDfErr, fabsf(s.h), e), y);
  const bool okz = df_round(w, kDfErr * w.h, z);
  if (!(okx && oky && okz)) cosine_hemisphere64(k0, k1, x, y, z);
}

// (float)((double)z / pi) for z >= 0.
__device__ __noinline__ float over_pi64(float z) { return (float)((double)z / 3.14159265358979323846); }
__device__ __forceinline__ float over_pi(float z) {
  if (z == 0.0f) return z;
  const DF p = df_prod(z, 0x1.45f306p-2f);
  float f;
  if (z > 1e-30f && df_round(DF{p.h, __fmaf_rn(z, 0x1.b93910p-27f, p.l)}, kDfErr * p.h, f)) return f;
  return over_pi64(z);
}

// Uniform over a triangle (builtin/light/triangle.go:248-250):
// (float)(r1 sqrt(1-r0)) and (float)(1 - sqrt(1-r0)).
__device__ __noinline__ void triangle_uv64(uint64_t k0, uint64_t k1, float& a, float& b) {
  const double r0 = frac52d(k0), r1 = frac52d(k1);
  a = (float)(r1 * sqrt(1 - r0));
  b = (float)(1 - sqrt(1 - r0));
}
__device__ __forceinline__ void triangle_uv(uint64_t k0, uint64_t k1, float& a, float& b) {
  const DF r = df_sqrt(df_frac52(kOne52 - k0));
  const DF p = df_mul(df_frac52(k1), r);
  const DF d = df_sum(1.0f, -r.h);
  const DF q = df_fast(d.h, d.l - r.l);
  const bool oka = df_round(p, __fmaf_rn(kDfErr, p.h, 0x1p-50f * r.h), a), okb = df_round(q, 0x1p-44f, b);
  if (!(oka && okb)) triangle_uv64(k0, k1, a, b);
}

// The camera sample's float64 expressions (core/render.go), rounded.
// (float)(-1 + 2 r / w), r = k / 2^40: 2 k - 2^40 w is exact, and float64's
// errors are below 2^-51 of 2 r / w + 1.
__device__ __noinline__ float raster_ndc64(uint64_t k, uint32_t w) {
  return (float)(-1.0 + 2.0 * ((double)k / 1099511627776.0 / (double)w));
}
__device__ __forceinline__ float raster_ndc(uint64_t k, uint32_t w) {
  if (w < (1u << 22)) {
    const DF n = df_int((int64_t)(2 * k) - ((int64_t)w << 40));
    const float fw = (float)w, rw = 1.0f / fw, q = n.h * rw;
    const DF v = df_fast(q * 0x1p-40f, (__fmaf_rn(-q, fw, n.h) + n.l) * rw * 0x1p-40f);
    float f;
    if (df_round(v, __fmaf_rn(kDfErr, fabsf(v.h), 0x1p-49f), f)) return f;
  }
  return raster_ndc64(k, w);
}
// (float)(270 v + 450), v = k / 2^52: the exact sum over 2^52; float64's two
// roundings move it by less than 2^-52 * 512.
__device__ __noinline__ float wavelength64(uint64_t k) { return (float)((720.0 - 450.0) * frac52d(k) + 450.0); }
__device__ __forceinline__ float wavelength52(uint64_t k) {
  const int64_t n = 270 * (int64_t)k + (450ll << 52);
  const float a = __ll2float_rn(n - 512), b = __ll2float_rn(n + 512);
  return a == b ? a * 0x1p-52f : wavelength64(k);
}

}  // namespace
}  // namespace vmr
