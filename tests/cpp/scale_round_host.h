// Host forms of the device intrinsics that tm_df.cuh uses, so that its
// arithmetic can be compiled and checked without a GPU.
#pragma once
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>

#ifndef __noinline__
#define __noinline__ __attribute__((noinline))
#endif

inline float2 __ffma2_rn(float2 a, float2 b, float2 c) {
  return make_float2(std::fmaf(a.x, b.x, c.x), std::fmaf(a.y, b.y, c.y));
}
inline float2 __fadd2_rn(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
inline float2 __fmul2_rn(float2 a, float2 b) { return make_float2(a.x * b.x, a.y * b.y); }
inline int __double2hiint(double v) {
  long long b;
  std::memcpy(&b, &v, 8);
  return (int)(b >> 32);
}
inline int __double2loint(double v) {
  long long b;
  std::memcpy(&b, &v, 8);
  return (int)b;
}
inline float __uint_as_float(unsigned u) {
  float f;
  std::memcpy(&f, &u, 4);
  return f;
}
inline float __uint2float_rn(unsigned u) { return (float)u; }
