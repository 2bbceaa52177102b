// FP64 scalar arithmetic off GB300's slow paths: one FP64 instruction takes 64
// clocks of an SM quadrant, a quotient or square root ~600, a conversion ~95.
#pragma once

namespace tnad {

// FP64 ↔ FP32 by integer operations: the conversion instructions take ~95
// clocks of the FP64 pipe each, these about 20 and 11 (truncation; values below
// the FP32 normal range become 0, above it are not expected: everything is
// scaled to [2^-60, 2^100])
__device__ __forceinline__ float d2f(double d) {
  const unsigned hi = (unsigned)__double2hiint(d), lo = (unsigned)__double2loint(d), a = hi & 0x7fffffffu;
  const unsigned r = a < (897u << 20) ? 0u : (((a - (896u << 20)) << 3) | (lo >> 29));
  return __uint_as_float(r | (hi & 0x80000000u));
}

__device__ __forceinline__ double f2d(float f) {
  const unsigned b = __float_as_uint(f), a = b & 0x7fffffffu;
  const unsigned hi = a ? (a >> 3) + (896u << 20) : 0u;
  return __hiloint2double((int)(hi | (b & 0x80000000u)), (int)(b << 29));
}

// The same with the conversion instructions' results for every argument: round
// to nearest even (d2f_rn: the instruction itself where either side is not a
// normal number or zero); about 25 and 14 clocks.
__device__ __forceinline__ float d2f_rn(double d) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(d);
  const unsigned a = (unsigned)(b >> 32) & 0x7fffffffu, sg = (unsigned)(b >> 32) & 0x80000000u;
  if (a - (897u << 20) >= (253u << 20)) return (b << 1) == 0 ? __uint_as_float(sg) : (float)d;
  const unsigned long long r = b + 0x0fffffffull + ((b >> 29) & 1ull);  // a carry moves on into the exponent
  return __uint_as_float((((((unsigned)(r >> 32) & 0x7fffffffu) - (896u << 20)) << 3) | ((unsigned)r >> 29)) | sg);
}

// (no branch: loads of a sum's next terms move above it)
__device__ __forceinline__ double f2d_any(float f) {
  const unsigned sg = __float_as_uint(f) & 0x80000000u;
  const bool small = (__float_as_uint(f) & 0x7fffffffu) < (1u << 23);  // subnormal or zero
  const unsigned a = __float_as_uint(small ? f * 4294967296.f : f) & 0x7fffffffu;
  const unsigned bias = a >= (255u << 23) ? 1792u << 20 : small ? 864u << 20 : 896u << 20;
  return __hiloint2double((int)((a ? (a >> 3) + bias : 0u) | sg), (int)(a << 29));
}

// z·2^e rounded to nearest even, for results in the normal range
__device__ __forceinline__ double ll2d_scaled(long long z, int e) {
  const unsigned long long u0 = z < 0 ? 0ull - (unsigned long long)z : (unsigned long long)z;
  const int lz = __clzll((long long)(u0 | 1ull));
  const unsigned long long u = u0 << lz;
  unsigned long long q = u >> 11;
  const unsigned rem = (unsigned)u & 0x7ffu;
  q += rem + ((unsigned)q & 1u) > 0x400u ? 1ull : 0ull;
  q += (unsigned long long)(1023 + 62 - lz + e) << 52;  // q's leading one adds the last step of the exponent
  q |= z < 0 ? 1ull << 63 : 0ull;
  return __longlong_as_double((long long)(z != 0 ? q : 0ull));
}

// FP32 quotient and square root to 1-2 ulp (they start Newton steps or only
// decide angles): ~30 clocks instead of ~150 for the rounded ones
__device__ __forceinline__ float fsqrt_ap(float x) {
  float r;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// tan of the rotation that diagonalises [[a, g], [g, b]] with df = b − a, g2 = 2g (FP32)
__device__ __forceinline__ float jacobi_tan(float df, float g2) {
  if (fabsf(df) >= fabsf(g2)) {
    const float w = __fdividef(g2, df);
    return __fdividef(w, 1.f + fsqrt_ap(fmaf(w, w, 1.f)));
  }
  const float w = __fdividef(df, g2);
  return __fdividef(copysignf(1.f, w), fabsf(w) + fsqrt_ap(fmaf(w, w, 1.f)));
}

// 1/√x by one cubic Newton (Halley) step from the FP32 value: relative error
// (5/16)·e³ with e ~ 2e-7.  x inside the FP32 normal range.  Six FP64
// instructions; sqrt() and a division take about 1300 clocks of the FP64 pipe.
__device__ __forceinline__ double rsqrt_fast(double x) {
  const double y = f2d(rsqrtf(d2f(x)));
  const double e = fma(-(x * y), y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}

// 1/√x of any positive x: the same on x scaled by an even power of two
__device__ __forceinline__ double rsqrt_any(double x) {
  const int hi = __double2hiint(x);
  if (hi < (1 << 20)) return 1.0 / sqrt(x);  // subnormal
  const int e = ((hi >> 20) - 1023) & ~1;
  const double r = rsqrt_fast(__hiloint2double(hi - (e << 20), __double2loint(x)));
  return __hiloint2double(__double2hiint(r) - ((e >> 1) << 20), __double2loint(r));
}

// 1/x by two Newton steps from the FP32 value
__device__ __forceinline__ double rcp_fast(double x) {
  double y = f2d(__fdividef(1.f, d2f(x)));
  y = fma(fma(-x, y, 1.0), y, y);
  return fma(fma(-x, y, 1.0), y, y);
}

}  // namespace tnad
