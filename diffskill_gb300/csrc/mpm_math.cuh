// Device math for the MPM substep: small vectors, 3x3 matrices, quaternions
// and their vector-Jacobian products, templated on the scalar type.
//
// Quaternion conventions follow plb/engine/primitive/utils.py:9-54
// (w, x, y, z); autodiff conventions follow the reference's taichi source
// transform: branch decisions frozen, max(a,b) sends the gradient to a iff
// b < a, min(a,b) to a iff a < b, abs' = sgn with sgn(0) = 0.
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#define MPM_DI __device__ __forceinline__
#define MPM_HD __host__ __device__

namespace mpm {

MPM_DI float msqrt(float x) { return sqrtf(x); }
MPM_DI double msqrt(double x) { return sqrt(x); }
// log(1 + x) and exp(x) - 1 for the FP32 strains (x = s - 1 of a singular
// value, or a projected log-strain), accurate to the result's own precision:
// for |x| < 1/64 by their Taylor series (truncation below 3e-12 and 2e-13
// relative), otherwise by the library's log1pf / expm1f.
MPM_DI float log1p_strain(float x) {
  if (fabsf(x) < 0.015625f)
    return x * fmaf(x, fmaf(x, fmaf(x, fmaf(x, fmaf(x, -1.f / 6.f, 0.2f), -0.25f), 1.f / 3.f), -0.5f), 1.f);
  return log1pf(x);
}
MPM_DI float expm1_strain(float x) {
  if (fabsf(x) < 0.015625f)
    return x * fmaf(x, fmaf(x, fmaf(x, fmaf(x, fmaf(x, 1.f / 720.f, 1.f / 120.f), 1.f / 24.f), 1.f / 6.f), 0.5f), 1.f);
  return expm1f(x);
}
// exp of the contact softness exp(-dist * softness) (primive_base.py:99), FP32
// by the hardware approximation: its relative error (a few ulp over the
// influence range exp(x) > 0.1) stays below the substep's rounding noise
MPM_DI float mexp_fast(float x) { return __expf(x); }
MPM_DI double mexp_fast(double x) { return exp(x); }
MPM_DI float msin(float x) { return sinf(x); }
MPM_DI double msin(double x) { return sin(x); }
MPM_DI float mcos(float x) { return cosf(x); }
MPM_DI double mcos(double x) { return cos(x); }
MPM_DI float mabs(float x) { return fabsf(x); }
MPM_DI double mabs(double x) { return fabs(x); }
template <typename T>
MPM_DI T sgn(T x) {
  return x > T(0) ? T(1) : (x < T(0) ? T(-1) : T(0));
}
template <typename T>
MPM_DI bool finite(T x) {
  return isfinite(x);
}

// a[i] for a runtime i in 0..2 without local memory
template <typename T>
MPM_DI T sel3(T a0, T a1, T a2, int i) {
  return i == 0 ? a0 : (i == 1 ? a1 : a2);
}
template <typename T>
MPM_DI T dot3(const T* a, const T* b) {
  return a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
}
template <typename T>
MPM_DI void cross3(const T* a, const T* b, T* c) {
  c[0] = a[1] * b[2] - a[2] * b[1];
  c[1] = a[2] * b[0] - a[0] * b[2];
  c[2] = a[0] * b[1] - a[1] * b[0];
}
template <typename T>
MPM_DI void add_cross3(const T* a, const T* b, T* c) {
  c[0] += a[1] * b[2] - a[2] * b[1];
  c[1] += a[2] * b[0] - a[0] * b[2];
  c[2] += a[0] * b[1] - a[1] * b[0];
}
// C = A B
template <typename T>
MPM_DI void mm(const T* A, const T* B, T* C) {
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) C[i * 3 + j] = A[i * 3] * B[j] + A[i * 3 + 1] * B[3 + j] + A[i * 3 + 2] * B[6 + j];
}
// C = A B^T
template <typename T>
MPM_DI void mmT(const T* A, const T* B, T* C) {
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j)
      C[i * 3 + j] = A[i * 3] * B[j * 3] + A[i * 3 + 1] * B[j * 3 + 1] + A[i * 3 + 2] * B[j * 3 + 2];
}
// C = A^T B
template <typename T>
MPM_DI void mTm(const T* A, const T* B, T* C) {
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) C[i * 3 + j] = A[i] * B[j] + A[3 + i] * B[3 + j] + A[6 + i] * B[6 + j];
}
template <typename T>
MPM_DI T det3(const T* A) {
  return A[0] * (A[4] * A[8] - A[5] * A[7]) - A[1] * (A[3] * A[8] - A[5] * A[6]) +
         A[2] * (A[3] * A[7] - A[4] * A[6]);
}

// FP64 arithmetic from FP32 starting values.  GB300 issues one FP64
// instruction per SM every 16 cycles or more (measured: 19 cycles of the SM per
// FP64 instruction of a warp in p2g, against a quarter of a cycle for an FP32
// one), so what can start from an FP32 value does: the reciprocal, the inverse
// square root and the singular vectors (mpm_svd.cuh).
//
// cut_f32 drops the low mantissa bits of x (0 outside FP32's normal range, NaN
// and infinity included); widen is exact for a normal or zero x.  Both are
// integer operations: the conversion instructions occupy the FP64 pipe.
MPM_DI float cut_f32(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const unsigned mag = hi & 0x7fffffffu;
  const unsigned b = __funnelshift_l(lo, mag, 3) - (896u << 23);  // exponent bias 1023 -> 127
  const bool in = mag - (897u << 20) < (254u << 20);              // exponents 1 .. 254 of FP32
  return __uint_as_float((hi & 0x80000000u) | (in ? b & 0x7fffffffu : 0u));
}
MPM_DI double widen(float x) {
  const unsigned b = __float_as_uint(x), mag = b & 0x7fffffffu;
  const unsigned hi = mag >= (1u << 23) ? (mag >> 3) + (896u << 20) : 0u;
  return __hiloint2double((int)((b & 0x80000000u) | hi), (int)(b << 29));
}
// float <-> double as the conversion instructions of a -ftz build give them
// (subnormals to zero, infinities and NaN kept, nearest-even), in integer
// operations: for the FP64 particle math on FP32 state
MPM_DI double exact_f64(float x) {
  const unsigned b = __float_as_uint(x), mag = b & 0x7fffffffu;
  const unsigned bias = mag >= 0x7f800000u ? 1792u << 20 : 896u << 20;  // infinity, NaN: exponent 2047
  const unsigned hi = mag >= (1u << 23) ? (mag >> 3) + bias : 0u;
  return __hiloint2double((int)((b & 0x80000000u) | hi), (int)(mag >= (1u << 23) ? b << 29 : 0u));
}
MPM_DI float round_f32(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const unsigned mag = hi & 0x7fffffffu, sign = hi & 0x80000000u;
  unsigned b = __funnelshift_l(lo, mag, 3) - (896u << 23);
  const unsigned rest = lo & 0x1fffffffu;
  b += (rest > 0x10000000u || (rest == 0x10000000u && (b & 1u))) ? 1u : 0u;
  const bool normal = mag - (897u << 20) < (254u << 20);
  const bool nan = mag > 0x7ff00000u || (mag == 0x7ff00000u && lo != 0u);
  const unsigned big = nan ? 0x7fffffffu : 0x7f800000u;
  // an exponent of 0 (2^-127 .. 2^-126) may still round up to 2^-126
  const bool edge = (mag >> 20) == 896u && b >= (1u << 23) && b < (1u << 24);
  const unsigned r = normal ? b & 0x7fffffffu : (mag >= (1151u << 20) ? big : (edge ? b : 0u));
  return __uint_as_float(sign | r);
}
// x in the precision T
template <typename T, typename X>
MPM_DI T to_prec(X x) {
  if constexpr (sizeof(T) == sizeof(X))
    return x;
  else if constexpr (sizeof(T) == 8)
    return exact_f64(x);
  else
    return round_f32(x);
}
// 1 / x for |x| in FP32's normal range, less its last two octaves: with y0 = 1/x (1 + e),
// |e| < 1e-6, from FP32, 1/x = y0 (1 + e + e^2) up to e^3 (Newton's iteration and its
// next term)
MPM_DI double rcp64_mid(double x) {
  const double y = widen(__fdividef(1.f, cut_f32(x)));
  const double e = fma(-x, y, 1.0);
  return fma(y, fma(e, e, e), y);
}
// 1 / sqrt(x) for x > 0 in FP32's normal range: y0 from FP32, e = 1 - x y0^2,
// 1/sqrt(x) = y0 (1 - e)^(-1/2) = y0 (1 + e/2 + 3 e^2 / 8) up to 5 e^3 / 16
MPM_DI double rsqrt64_mid(double x) {
  const double y = widen(rsqrtf(cut_f32(x)));
  const double e = fma(-x, y * y, 1.0);
  return fma(y, e * fma(e, 0.375, 0.5), y);
}
// The FP32 starting value of a number whose high word is `hi`, of an exponent near 0
MPM_DI float near_one_f32(unsigned hi, unsigned lo) {
  return __uint_as_float(__funnelshift_l(lo, hi, 3) - (896u << 23));  // exponent bias 1023 -> 127
}
// widen of a positive normal x
MPM_DI double widen_normal(float x) {
  const unsigned b = __float_as_uint(x);
  return __hiloint2double((int)((b >> 3) + (896u << 20)), (int)(b << 29));
}
// 1 / x of a normal |x| < 2^1022: of x = m 2^k, 1 <= m < 2, by the above, and k taken off
// the exponent.  (Its integer operations are in the chain of each value: in the SVD and
// the return map, whose values are near 1, it would make an iteration of 10,000 FP64
// particles 0.4 % slower than rcp64_mid; in the tools and the grid it costs 0.6 %.)
MPM_DI double rcp64_normal(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const unsigned ex = hi & 0x7ff00000u, mh = (hi & 0x000fffffu) | 0x3ff00000u;
  const double m = __hiloint2double((int)mh, (int)lo);
  const double y = widen_normal(__fdividef(1.f, near_one_f32(mh, lo)));
  const double e = fma(-m, y, 1.0), r = fma(y, fma(e, e, e), y);
  const unsigned rh = (unsigned)__double2hiint(r) + (0x3ff00000u - ex);
  return __hiloint2double((int)(rh | (hi & 0x80000000u)), __double2loint(r));
}
// 1 / x.  0 and subnormals give infinity; infinity and |x| >= 2^1022 (a subnormal
// reciprocal) 0.
MPM_DI double rcp64(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), ex = hi & 0x7ff00000u;
  const double r = rcp64_normal(x);
  if (ex - (1u << 20) < (2044u << 20)) return r;
  const bool nan = ex == 0x7ff00000u && ((hi & 0x000fffffu) | (unsigned)__double2loint(x)) != 0u;
  const unsigned rh = nan ? 0x7ff80000u : (ex == 0u ? 0x7ff00000u : 0u);
  return __hiloint2double((int)(rh | (hi & 0x80000000u)), 0);
}
// 1 / sqrt(x) of a normal x > 0: of x = m 4^k, 1 <= m < 4, and k taken off the exponent
MPM_DI double rsqrt64_normal(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const unsigned ex = hi & 0x7ff00000u, base = 0x3ff00000u + (~hi & 0x00100000u);
  const unsigned mh = (hi & 0x000fffffu) | base;
  const double m = __hiloint2double((int)mh, (int)lo);
  const double y = widen_normal(rsqrtf(near_one_f32(mh, lo)));
  const double e = fma(-m, y * y, 1.0), r = fma(y, e * fma(e, 0.375, 0.5), y);
  return __hiloint2double(__double2hiint(r) - ((int)(ex - base) >> 1), __double2loint(r));
}
// 1 / sqrt(x).  0 and subnormals give infinity, infinity 0, a negative x NaN.
MPM_DI double rsqrt64(double x) {
  const unsigned hi = (unsigned)__double2hiint(x);
  const double r = rsqrt64_normal(x);
  if (hi - (1u << 20) < (2046u << 20)) return r;
  const bool zero = (hi & 0x7ff00000u) == 0u, inf = hi == 0x7ff00000u && __double2loint(x) == 0;
  return __hiloint2double((int)(zero ? 0x7ff00000u : (inf ? 0u : 0x7ff80000u)), 0);
}
// sqrt(x) of a normal x > 0, infinity or NaN
MPM_DI float sqrt_pos(float x) { return msqrt(x); }
MPM_DI double sqrt_pos(double x) {
  const double r = x * rsqrt64_normal(x);
  return ((unsigned)__double2hiint(x) & 0x7ff00000u) == 0x7ff00000u ? x : r;
}

// length() with the eps of plb/engine/primitive/primitives.py:13-15
template <typename T>
MPM_DI T len14(const T* a) {
  return sqrt_pos(dot3(a, a) + T(1e-14));
}
// its reciprocal
template <typename T>
MPM_DI T inv_len14(const T* a) {
  if constexpr (sizeof(T) == 8)
    return rsqrt64_normal(dot3(a, a) + T(1e-14));
  else
    return T(1) / len14(a);
}
// length() with the eps of plb/engine/primitive/utils.py:4-6
template <typename T>
MPM_DI T len8(const T* a) {
  return sqrt_pos(dot3(a, a) + T(1e-8));
}
// a / b (FP64: |b| < 2^1022)
MPM_DI float quot(float a, float b) { return a / b; }
MPM_DI double quot(double a, double b) { return a * rcp64(b); }
// the same where b is normal (a length with its eps, a time step)
MPM_DI float quot_normal(float a, float b) { return a / b; }
MPM_DI double quot_normal(double a, double b) { return a * rcp64_normal(b); }
// d(u/len14(u))^T g
template <typename T>
MPM_DI void unit14_vjp(const T* u, const T* g, T* gu) {
  T ug = dot3(u, g);
  T iL = inv_len14(u);
  T c = ug * iL * iL * iL;
#pragma unroll
  for (int k = 0; k < 3; ++k) gu[k] = g[k] * iL - u[k] * c;
}

// ---------------------------------------------------------------------------
// quaternions
// ---------------------------------------------------------------------------
// qrot (utils.py:9-15)
template <typename T>
MPM_DI void qrot(const T* q, const T* v, T* out) {
  const T qv[3] = {q[1], q[2], q[3]};
  T uv[3], uuv[3];
  cross3(qv, v, uv);
  cross3(qv, uv, uuv);
#pragma unroll
  for (int d = 0; d < 3; ++d) out[d] = v[d] + T(2) * (q[0] * uv[d] + uuv[d]);
}
// accumulates gq (may be null) and gv (may be null)
template <typename T>
MPM_DI void qrot_vjp(const T* q, const T* v, const T* g, T* gq, T* gv) {
  const T qv[3] = {q[1], q[2], q[3]};
  T uv[3];
  cross3(qv, v, uv);
  T g_uv[3], g_uuv[3], g_qv[3] = {T(0), T(0), T(0)};
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    g_uv[d] = T(2) * q[0] * g[d];
    g_uuv[d] = T(2) * g[d];
  }
  add_cross3(uv, g_uuv, g_qv);
  add_cross3(g_uuv, qv, g_uv);
  add_cross3(v, g_uv, g_qv);
  if (gv) {
#pragma unroll
    for (int d = 0; d < 3; ++d) gv[d] += g[d];
    add_cross3(g_uv, qv, gv);
  }
  if (gq) {
    gq[0] += T(2) * dot3(g, uv);
    gq[1] += g_qv[0];
    gq[2] += g_qv[1];
    gq[3] += g_qv[2];
  }
}
// normalized() of the conjugate (utils.py:53, primive_base.py:89-90)
template <typename T>
MPM_DI void conj_unit(const T* r, T* iq) {
  T L = msqrt(r[0] * r[0] + r[1] * r[1] + r[2] * r[2] + r[3] * r[3]);
  T inv = T(1) / L;
  iq[0] = r[0] * inv;
  iq[1] = -r[1] * inv;
  iq[2] = -r[2] * inv;
  iq[3] = -r[3] * inv;
}
template <typename T>
MPM_DI void conj_unit_vjp(const T* r, const T* g_iq, T* g_r) {
  const T c[4] = {r[0], -r[1], -r[2], -r[3]};
  T L = msqrt(c[0] * c[0] + c[1] * c[1] + c[2] * c[2] + c[3] * c[3]);
  T inv = T(1) / L;
  T ng = (c[0] * g_iq[0] + c[1] * g_iq[1] + c[2] * g_iq[2] + c[3] * g_iq[3]) * inv;
  T gc[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) gc[i] = (g_iq[i] - c[i] * inv * ng) * inv;
  g_r[0] += gc[0];
  g_r[1] -= gc[1];
  g_r[2] -= gc[2];
  g_r[3] -= gc[3];
}
// inv_trans (utils.py:50-54)
template <typename T>
MPM_DI void inv_trans(const T* p, const T* pos, const T* rot, T* out) {
  T iq[4];
  conj_unit(rot, iq);
  const T d[3] = {p[0] - pos[0], p[1] - pos[1], p[2] - pos[2]};
  qrot(iq, d, out);
}
template <typename T>
MPM_DI void inv_trans_vjp(const T* p, const T* pos, const T* rot, const T* g, T* g_p, T* g_pos, T* g_rot) {
  T iq[4];
  conj_unit(rot, iq);
  const T d[3] = {p[0] - pos[0], p[1] - pos[1], p[2] - pos[2]};
  T g_iq[4] = {T(0), T(0), T(0), T(0)}, g_d[3] = {T(0), T(0), T(0)};
  qrot_vjp(iq, d, g, g_iq, g_d);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    if (g_p) g_p[k] += g_d[k];
    g_pos[k] -= g_d[k];
  }
  conj_unit_vjp(rot, g_iq, g_rot);
}
// qmul (utils.py:23-31): Hamilton product q*r, normalised
template <typename T>
MPM_DI void qmul_raw(const T* q, const T* r, T* o) {
  o[0] = r[0] * q[0] - r[1] * q[1] - r[2] * q[2] - r[3] * q[3];
  o[1] = r[0] * q[1] + r[1] * q[0] - r[2] * q[3] + r[3] * q[2];
  o[2] = r[0] * q[2] + r[1] * q[3] + r[2] * q[0] - r[3] * q[1];
  o[3] = r[0] * q[3] - r[1] * q[2] + r[2] * q[1] + r[3] * q[0];
}
// 1 / sqrt(L2) through rsqrt: FP64 within 1 ulp (FP64 divide and square root
// are long instruction sequences on GB300's FP64 pipe), FP32 by the hardware
// approximation
MPM_DI double inv_len(double L2) { return rsqrt(L2); }
MPM_DI float inv_len(float L2) { return rsqrtf(L2); }
template <typename T>
MPM_DI void qmul(const T* q, const T* r, T* out) {
  T o[4];
  qmul_raw(q, r, o);
  T inv = inv_len(o[0] * o[0] + o[1] * o[1] + o[2] * o[2] + o[3] * o[3]);
#pragma unroll
  for (int i = 0; i < 4; ++i) out[i] = o[i] * inv;
}
template <typename T>
MPM_DI void qmul_vjp(const T* q, const T* r, const T* g, T* gq, T* gr) {
  T o[4];
  qmul_raw(q, r, o);
  T iL = inv_len(o[0] * o[0] + o[1] * o[1] + o[2] * o[2] + o[3] * o[3]);
  T on = (o[0] * g[0] + o[1] * g[1] + o[2] * g[2] + o[3] * g[3]) * iL * iL;
  T go[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) go[i] = (g[i] - o[i] * on) * iL;
  gq[0] += go[0] * r[0] + go[1] * r[1] + go[2] * r[2] + go[3] * r[3];
  gq[1] += -go[0] * r[1] + go[1] * r[0] - go[2] * r[3] + go[3] * r[2];
  gq[2] += -go[0] * r[2] + go[1] * r[3] + go[2] * r[0] - go[3] * r[1];
  gq[3] += -go[0] * r[3] - go[1] * r[2] + go[2] * r[1] + go[3] * r[0];
  gr[0] += go[0] * q[0] + go[1] * q[1] + go[2] * q[2] + go[3] * q[3];
  gr[1] += -go[0] * q[1] + go[1] * q[0] + go[2] * q[3] - go[3] * q[2];
  gr[2] += -go[0] * q[2] - go[1] * q[3] + go[2] * q[0] + go[3] * q[1];
  gr[3] += -go[0] * q[3] + go[1] * q[2] - go[2] * q[1] + go[3] * q[0];
}
// w2quat (utils.py:34-47)
template <typename T>
MPM_DI void w2quat(const T* aa, T* out) {
  T w = msqrt(dot3(aa, aa) + T(1e-16));
  out[0] = T(1);
  out[1] = out[2] = out[3] = T(0);
  if (w > T(1e-9)) {
    T s = msin(w / T(2));
    out[0] = mcos(w / T(2));
#pragma unroll
    for (int k = 0; k < 3; ++k) out[k + 1] = (aa[k] / w) * s;
  }
}
template <typename T>
MPM_DI void w2quat_vjp(const T* aa, const T* g, T* gaa) {
  T w = msqrt(dot3(aa, aa) + T(1e-16));
  if (!(w > T(1e-9))) return;
  T s = msin(w / T(2)), c = mcos(w / T(2));
  T gw = T(-0.5) * s * g[0];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    gaa[k] += g[k + 1] * s / w;
    gw += g[k + 1] * aa[k] * (-s / (w * w) + T(0.5) * c / w);
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) gaa[k] += gw * aa[k] / w;
}

}  // namespace mpm
