// The few CUDA names that mpm_math.cuh and mpm_svd.cuh use, for a host compiler: the
// device functions run on the CPU.  The approximate reciprocal and inverse square root
// are exact here, so errors of theirs are not part of what the host tests see.
#pragma once
#include <math.h>
#include <stdint.h>
#include <string.h>

#define __device__
#define __host__
#define __forceinline__ inline
#define __noinline__

template <typename To, typename From>
inline To bits_of(From x) {
  To y;
  memcpy(&y, &x, sizeof(y));
  return y;
}
inline float __uint_as_float(unsigned u) { return bits_of<float>(u); }
inline unsigned __float_as_uint(float x) { return bits_of<unsigned>(x); }
inline int __double2hiint(double x) { return (int)(bits_of<uint64_t>(x) >> 32); }
inline int __double2loint(double x) { return (int)bits_of<uint64_t>(x); }
inline double __hiloint2double(int hi, int lo) {
  return bits_of<double>(((uint64_t)(unsigned)hi << 32) | (unsigned)lo);
}
inline unsigned __funnelshift_l(unsigned lo, unsigned hi, unsigned s) {
  return s ? (hi << s) | (lo >> (32 - s)) : hi;
}
inline float __fdividef(float a, float b) { return a / b; }
inline float rsqrtf(float x) { return 1.0f / sqrtf(x); }
inline double rsqrt(double x) { return 1.0 / sqrt(x); }
inline float __expf(float x) { return expf(x); }
