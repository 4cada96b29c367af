// 3x3 SVD and its clamped backward on the device.
//
// Forward: A = U diag(s) V^T with det U = det V = +1 and the sign of det A on the last
// value, as ti.svd (plb/engine/mpm_simulator.py:127-129), from the left: a cyclic Jacobi
// eigen-decomposition of A A^T with symmetric Schur rotations (Golub & Van Loan,
// "Matrix Computations", Sec. 8.5.2) gives U and s^2, then V = A^T U / s.  The values
// come in no particular order (nothing depends on it) but where V is taken by
// Gram-Schmidt: s0 >= s1 >= |s2| there.  FP32 rotates A A^T - I (svd3_left32), FP64
// refines an FP32 decomposition (svd3_left64).
//
// Backward: backward_svd of plb/engine/mpm_simulator.py:137-156 with the
// +-1e-6 clamp of clamp() (184-192) on s_j^2 - s_i^2.
#pragma once
#include "mpm_math.cuh"

namespace mpm {

template <typename T>
struct SvdIters;
template <>
struct SvdIters<float> {
  static constexpr int max_sweeps = 6;
  static constexpr float tol = 1e-14f;  // on off^2 / diag^2
};
template <>
struct SvdIters<double> {
  static constexpr int max_sweeps = 12;
  static constexpr double tol = 1e-32;
};

// rotation tangent t = sgn(theta) / (|theta| + sqrt(theta^2 + 1)) and cosine c;
// FP32 uses the approximate reciprocal, square root and rsqrt: the error only
// moves the rotation angle, and c and s = t c come from the same rsqrt, so the
// rotation stays orthogonal to rounding
MPM_DI void rot_tc(double theta, double& t, double& c) {
  t = (theta >= 0.0 ? 1.0 : -1.0) / (fabs(theta) + sqrt(theta * theta + 1.0));
  c = 1.0 / sqrt(t * t + 1.0);
}
MPM_DI void rot_tc(float theta, float& t, float& c) {
  const float at = fabsf(theta);
  // for huge |theta|, t ~ 1/(2 theta) (avoids theta^2 overflow)
  const float y = fmaf(theta, theta, 1.0f);
  const float den = at < 1e18f ? at + y * rsqrtf(y) : 2.0f * at;
  t = copysignf(__fdividef(1.0f, den), theta);
  c = rsqrtf(fmaf(t, t, 1.0f));
}

// a / b; FP32 by the approximate reciprocal (|b| < 2^126 here), FP64 by rcp64_normal.
// Used for the return map, for the Jacobi angle (angle_div: FP64 divides as such there),
// and for the SVD backward's 1 / (s_j^2 - s_i^2), whose divisor is clamped to |b| >= 1e-6.  The substep kernels are built with -ftz=true, so
// a subnormal s_pq compares equal to 0 and is never a divisor.
MPM_DI double fast_div(double a, double b) { return a * rcp64_normal(b); }
MPM_DI float fast_div(float a, float b) { return __fdividef(a, b); }
MPM_DI double angle_div(double a, double b) { return a / b; }  // any quotient
MPM_DI float angle_div(float a, float b) { return __fdividef(a, b); }

// log(s) of a singular value from sm1 = s - 1: 2 atanh(z) with
// z = (s - 1) / (s + 1), by the series of atanh to z^13 for |s - 1| < 1/8
// (|z| < 1/15: truncation below 3e-18 of the result)
MPM_DI double log_strain64(double s, double sm1) {
  if (fabs(sm1) < 0.125) {
    const double z = 2.0 * sm1 * rcp64_mid(s + 1.0);  // 2 z
    const double w = 0.25 * z * z;
    const double p = fma(w, fma(w, fma(w, fma(w, fma(w, 1.0 / 13.0, 1.0 / 11.0), 1.0 / 9.0), 1.0 / 7.0), 1.0 / 5.0),
                         1.0 / 3.0);
    return fma(z * w, p, z);
  }
  return log(s);
}
// exp(x) - 1 by its Taylor series to x^11 for |x| < 1/8 (truncation below 2e-20)
MPM_DI double expm1_strain64(double x) {
  if (fabs(x) < 0.125) {
    double p = fma(x, 1.0 / 39916800.0, 1.0 / 3628800.0);
    p = fma(x, p, 1.0 / 362880.0);
    p = fma(x, p, 1.0 / 40320.0);
    p = fma(x, p, 1.0 / 5040.0);
    p = fma(x, p, 1.0 / 720.0);
    p = fma(x, p, 1.0 / 120.0);
    p = fma(x, p, 1.0 / 24.0);
    p = fma(x, p, 1.0 / 6.0);
    p = fma(x, p, 0.5);
    return fma(x * x, p, x);
  }
  return expm1(x);
}
MPM_DI float third(float x) { return fast_div(x, 3.f); }
MPM_DI double third(double x) { return x * (1.0 / 3.0); }

// one Jacobi rotation zeroing s_pq of the symmetric matrix held as
// (s_pp, s_qq, s_pq, s_rp, s_rq); V columns p, q rotated alongside
template <typename T>
MPM_DI void jacobi_rot(T& app, T& aqq, T& apq, T& arp, T& arq, T* V, int p, int q) {
  if (apq == T(0)) return;
  T theta = angle_div(aqq - app, T(2) * apq);
  T t, c;
  rot_tc(theta, t, c);
  T s = t * c;
  app = app - t * apq;
  aqq = aqq + t * apq;
  apq = T(0);
  T rp = c * arp - s * arq;
  T rq = s * arp + c * arq;
  arp = rp;
  arq = rq;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    T vp = V[k * 3 + p], vq = V[k * 3 + q];
    V[k * 3 + p] = c * vp - s * vq;
    V[k * 3 + q] = s * vp + c * vq;
  }
}

// The rest of an SVD from the left, for any matrix: U's columns are eigenvectors of
// A A^T with eigenvalues ev (any common offset), B = A^T U.  Orders the columns by
// eigenvalue, keeping det U = 1, and takes V from Gram-Schmidt on B's columns, longest
// first, so that the short singular vectors are as exact as the long ones.  Returns
// |b0|, v1 . b1 and v2 . b2 in n (the singular values, the last one signed).
template <typename T>
MPM_DI void left_gram_schmidt(T* U, T* ev, T* B, T* n, T* V) {
  const auto order = [&](int a, int b) {
    if (ev[a] < ev[b]) {
      const T t = ev[a];
      ev[a] = ev[b];
      ev[b] = t;
#pragma unroll
      for (int k = 0; k < 3; ++k) {  // a swap, and one column negated: det U is kept
        const T u = U[k * 3 + a], w = B[k * 3 + a];
        U[k * 3 + a] = U[k * 3 + b];
        B[k * 3 + a] = B[k * 3 + b];
        U[k * 3 + b] = -u;
        B[k * 3 + b] = -w;
      }
    }
  };
  order(0, 1);
  order(0, 2);
  order(1, 2);
  const T b0[3] = {B[0], B[3], B[6]}, b1[3] = {B[1], B[4], B[7]}, b2[3] = {B[2], B[5], B[8]};
  T v0[3] = {T(1), T(0), T(0)}, v1[3], v2[3];
  n[0] = T(0);
  const T d0 = dot3(b0, b0);
  if (d0 != T(0)) {  // (NaN too)
    const T inv = inv_len(d0);
    n[0] = d0 * inv;
#pragma unroll
    for (int k = 0; k < 3; ++k) v0[k] = b0[k] * inv;
  }
  T r[3] = {b1[0], b1[1], b1[2]};
#pragma unroll
  for (int pass = 0; pass < 2; ++pass) {  // twice: b1 may be nothing but its part along v0
    const T pr = dot3(v0, r);
#pragma unroll
    for (int k = 0; k < 3; ++k) r[k] -= pr * v0[k];
  }
  T d1 = dot3(r, r);
  if (d1 == T(0)) {  // A of rank <= 1: any unit vector orthogonal to v0
    int m = (mabs(v0[0]) < mabs(v0[1])) ? 0 : 1;
    if (mabs(v0[2]) < mabs(sel3(v0[0], v0[1], v0[2], m))) m = 2;
    const T pe = sel3(v0[0], v0[1], v0[2], m);
#pragma unroll
    for (int k = 0; k < 3; ++k) r[k] = (k == m ? T(1) : T(0)) - pe * v0[k];
    d1 = dot3(r, r);
  }
  const T inv = inv_len(d1);
#pragma unroll
  for (int k = 0; k < 3; ++k) v1[k] = r[k] * inv;
  cross3(v0, v1, v2);
  n[1] = dot3(v1, b1);
  n[2] = dot3(v2, b2);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    V[k * 3] = v0[k];
    V[k * 3 + 1] = v1[k];
    V[k * 3 + 2] = v2[k];
  }
}

// convergence of the shifted sweeps: off-diagonal^2 <= kShiftedTol * diagonal^2
constexpr float kShiftedTol = 1e-14f;
// FP32 SVD of A = I + D = U diag(s) V^T from the left, given the displacement D = A - I
// (not A itself), so that the strain information (of size |D|, typically 1e-4 .. 1e-2)
// keeps FP32's relative precision instead of the absolute precision of numbers near
// 1: Jacobi rotations on A A^T - I = D + D^T + D D^T, converged relative to that
// matrix, give U and s^2 - 1, and s - 1 = (s^2 - 1) / (1 + s) is exact as s -> 1.  The
// forward pass, which needs no V, then has neither a product A V nor a Gram-Schmidt,
// and V = A^T U diag(1/s) takes their place in the adjoint.  The values are in no
// particular order (nothing depends on it).  A rotation scales its two columns by
// sqrt(c^2 + s^2) = 1 + O(1e-7), so each column is normalised once at the end
// (unit_column).  So is each column of V, whose length has the error of the approximate
// is, mostly of one sign: the adjoint takes an elastic particle's gradient of F through
// U (U^T g V) V^T in every substep, and 2e-8 to 7e-8 each time made the action gradients
// of 5,000 substeps 1e-4 to 2e-4 too small.  detA = det(I + D).  V is written when WithV; is = 1/s.
//
// U carries a rounding error of 1e-7, and A^T U / s that error times the ratio of A's
// longest to its shortest axis.  So an inverted or strongly deformed matrix,
// |A A^T - I|^2 (Frobenius) of kLeftNorm2 or more, takes V from Gram-Schmidt: then
// true (plain) is returned, V is written, is = 0, and s[2] may be negative.  Median
// relative error, without and with it, of newF at a smallest s of 0.2 .. 0.25: 3.4e-7,
// 2.0e-7; at 0.5 .. 0.7: 1.0e-7, 8.9e-8; of the gradient of C at a largest s of
// 3 .. 10: 1.8e-6, 6.0e-7 (an SVD by Gram-Schmidt throughout: 2.2e-7, 9.2e-8 and
// 6.7e-7).  Below kLeftNorm2 the two agree to 3 %; dough, which yields at strains near
// 0.01, is far below it.
constexpr float kLeftNorm2 = 0.5f;
// the column u of a 3x3 matrix, of length 1 + O(1e-7), normalised: u + u (1 - |u|^2) / 2.
// (The factor 3/2 - |u|^2 / 2 itself, rounded above and below 1 to different spacings,
// leaves columns 1e-8 short on average.)
MPM_DI void unit_column(float* u) {
  const float e = 0.5f * fmaf(-u[6], u[6], fmaf(-u[3], u[3], fmaf(-u[0], u[0], 1.f)));
  u[0] = fmaf(u[0], e, u[0]);
  u[3] = fmaf(u[3], e, u[3]);
  u[6] = fmaf(u[6], e, u[6]);
}
template <bool WithV>
MPM_DI bool svd3_left32(const float* D, float detA, float* U, float* s, float* sm1, float* is, float* V) {
  float ev[3], norm2;
  {
    float a00 = 2.f * D[0] + dot3(D, D), a11 = 2.f * D[4] + dot3(D + 3, D + 3), a22 = 2.f * D[8] + dot3(D + 6, D + 6);
    float a01 = D[1] + D[3] + dot3(D, D + 3), a02 = D[2] + D[6] + dot3(D, D + 6), a12 = D[5] + D[7] + dot3(D + 3, D + 6);
#pragma unroll
    for (int k = 0; k < 9; ++k) U[k] = (k % 4 == 0) ? 1.f : 0.f;
    for (int sweep = 0; sweep < SvdIters<float>::max_sweeps; ++sweep) {
      const float off = a01 * a01 + a02 * a02 + a12 * a12;
      const float dg = a00 * a00 + a11 * a11 + a22 * a22;
      // relative to the matrix; the absolute floor stops sweeps on rounding noise (rigid rotations)
      if (off <= kShiftedTol * dg + 1e-30f) break;
      jacobi_rot(a00, a11, a01, a02, a12, U, 0, 1);
      jacobi_rot(a00, a22, a02, a01, a12, U, 0, 2);
      jacobi_rot(a11, a22, a12, a01, a02, U, 1, 2);
    }
    ev[0] = a00;
    ev[1] = a11;
    ev[2] = a22;
    norm2 = a00 * a00 + a11 * a11 + a22 * a22;
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) unit_column(U + k);
  if (!(norm2 < kLeftNorm2 && detA > 0.f)) {
    float B[9], n[3];
    mTm(D, U, B);
#pragma unroll
    for (int k = 0; k < 9; ++k) B[k] += U[k];
    left_gram_schmidt(U, ev, B, n, V);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      s[k] = sqrtf(fmaxf(1.f + ev[k], 0.f));
      sm1[k] = ev[k] / (1.f + s[k]);  // (s^2 - 1) / (s + 1)
    }
    if (n[2] < 0.f) {
      s[2] = -s[2];
      sm1[2] = s[2] - 1.f;
    }
    is[0] = is[1] = is[2] = 0.f;
    return true;
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float q = 1.f + ev[k];
    is[k] = rsqrtf(q);
    s[k] = q * is[k];
    sm1[k] = fast_div(ev[k], 1.f + s[k]);  // (s^2 - 1) / (s + 1)
  }
  if constexpr (WithV) {
    mTm(D, U, V);
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int k = 0; k < 3; ++k) V[r * 3 + k] = (V[r * 3 + k] + U[r * 3 + k]) * is[k];
#pragma unroll
    for (int k = 0; k < 3; ++k) unit_column(V + k);
  }
  return false;
}

// Two parts of svd3_left64 that few particles reach, out of line so that the kernels do
// not carry their registers (inline, the second one made the adjoint of 37,001 FP64
// particles 3 % slower): Jacobi sweeps in FP64 on a matrix whose eigenvalues nearly
// coincide (S = s00, s11, s22, s01, s02, s12 and U, both updated), and V by
// Gram-Schmidt.
__device__ __noinline__ inline void jacobi64_finish(double* S, double* U) {
  double a00 = S[0], a11 = S[1], a22 = S[2], a01 = S[3], a02 = S[4], a12 = S[5];
  for (int sweep = 0; sweep < SvdIters<double>::max_sweeps; ++sweep) {
    const double off = a01 * a01 + a02 * a02 + a12 * a12;
    const double dg = a00 * a00 + a11 * a11 + a22 * a22;
    if (off <= SvdIters<double>::tol * dg) break;
    jacobi_rot(a00, a11, a01, a02, a12, U, 0, 1);
    jacobi_rot(a00, a22, a02, a01, a12, U, 0, 2);
    jacobi_rot(a11, a22, a12, a01, a02, U, 1, 2);
  }
  S[0] = a00;
  S[1] = a11;
  S[2] = a22;
}
__device__ __noinline__ inline void left_gram_schmidt64(const double* A, double* U, double* S, double* s, double* V) {
  double B[9];
  mTm(A, U, B);
  left_gram_schmidt(U, S, B, s, V);
}

// FP64 SVD A = U diag(s) V^T from the left: U and s^2 are the eigenvectors and
// eigenvalues of A A^T, V = A^T U diag(1/s), the values in no particular order, unless
// `plain` is returned: then the matrix was inverted, strongly deformed (an s below 0.2
// or above 3) or not finite, V comes from Gram-Schmidt, and s[2] is perhaps negative.
// V is written when plain or WithV; is = 1/s (plain: 0 for s at or below the return
// map's 0.05).
//
// An FP64 Jacobi rotation costs about 68 FP64 instructions, and four to five sweeps
// of three were about 900 of the 1,245 FP64 instructions that p2g spent on a
// particle.  Here the sweeps run in FP32 on the shifted matrix
// A A^T - I (relative to the strain, as svd3_left32), and FP64 only refines:
// - U is orthonormalised by Gram-Schmidt (a unit vector's norm is 1 + O(1e-6),
//   so 1/|u| is a two-term series);
// - S = U^T A A^T U is then diagonal but for E of at most 1e-6 of the strain;
//   Q = exp(X) with the antisymmetric X = X1 + X2 of second-order perturbation
//   theory, X1_pq = E_pq / (S_qq - S_pp), X2_pq = 1/2 [E, X1]_pq / (S_qq - S_pp),
//   diagonalises it to E X^2;
// - where that is above FP64's rounding of S, or X above 2e-4 (eigenvalues nearly
//   equal, but not within rounding), FP64 sweeps finish it instead (jacobi64_finish):
//   under one matrix in 20,000 at strains up to 0.3, one in 250 at singular values of
//   0.2 .. 3.  With |X| <= 2e-4 alone E X^2 reached 600 times the rounding: newF, worst
//   of 20,000 at 0.2 .. 3, 2.0e-14, now 2.8e-15, by FP64 sweeps 4.3e-15; with
//   |X| <= 2e-5 alone, as exact, 1 % of an iteration went into sweeps.
// About 180 FP64 instructions, and 100 more for a plain matrix.  p2g of 0.76M particles
// (FP32 state, FP64 SVD): 1469 -> 494 us; its adjoint: 2096 -> 997 us.
template <bool WithV>
MPM_DI bool svd3_left64(const double* A, double* U, double* s, double* is, double* V) {
  double S[6];  // 00, 11, 22, 01, 02, 12
  {
    const double* a = A;
    S[0] = dot3(a, a);
    S[1] = dot3(a + 3, a + 3);
    S[2] = dot3(a + 6, a + 6);
    S[3] = dot3(a, a + 3);
    S[4] = dot3(a, a + 6);
    S[5] = dot3(a + 3, a + 6);
  }
  {
    float W[9];
    float a00 = cut_f32(S[0] - 1.0), a11 = cut_f32(S[1] - 1.0), a22 = cut_f32(S[2] - 1.0);
    float a01 = cut_f32(S[3]), a02 = cut_f32(S[4]), a12 = cut_f32(S[5]);
#pragma unroll
    for (int k = 0; k < 9; ++k) W[k] = (k % 4 == 0) ? 1.f : 0.f;
    for (int sweep = 0; sweep < SvdIters<float>::max_sweeps; ++sweep) {
      const float off = a01 * a01 + a02 * a02 + a12 * a12;
      const float dg = a00 * a00 + a11 * a11 + a22 * a22;
      if (off <= kShiftedTol * dg + 1e-30f) break;
      jacobi_rot(a00, a11, a01, a02, a12, W, 0, 1);
      jacobi_rot(a00, a22, a02, a01, a12, W, 0, 2);
      jacobi_rot(a11, a22, a12, a01, a02, W, 1, 2);
    }
    double u0[3], u1[3], u2[3];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      u0[r] = widen(W[r * 3]);
      u1[r] = widen(W[r * 3 + 1]);
    }
    double e = 1.0 - dot3(u0, u0);
    double f = fma(e, fma(e, 0.375, 0.5), 1.0);
#pragma unroll
    for (int r = 0; r < 3; ++r) u0[r] *= f;
    const double d = dot3(u0, u1);
#pragma unroll
    for (int r = 0; r < 3; ++r) u1[r] = fma(-d, u0[r], u1[r]);
    e = 1.0 - dot3(u1, u1);
    f = fma(e, fma(e, 0.375, 0.5), 1.0);
#pragma unroll
    for (int r = 0; r < 3; ++r) u1[r] *= f;
    cross3(u0, u1, u2);
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      U[r * 3] = u0[r];
      U[r * 3 + 1] = u1[r];
      U[r * 3 + 2] = u2[r];
    }
  }
  {
    double B[9];
    mTm(A, U, B);  // columns b_i = A^T u_i
    const double b0[3] = {B[0], B[3], B[6]}, b1[3] = {B[1], B[4], B[7]}, b2[3] = {B[2], B[5], B[8]};
    S[0] = dot3(b0, b0);
    S[1] = dot3(b1, b1);
    S[2] = dot3(b2, b2);
    S[3] = dot3(b0, b1);
    S[4] = dot3(b0, b2);
    S[5] = dot3(b1, b2);
  }
  const float round = 4e-17f * (cut_f32(S[0]) + cut_f32(S[1]) + cut_f32(S[2]));
  float x32[3], r32[3], e32[3];
  double x[3];
  bool far = false;
#pragma unroll
  for (int q = 0; q < 3; ++q) {  // pairs (0, 1), (0, 2), (1, 2)
    const double gap = S[q == 0 ? 1 : 2] - S[q == 2 ? 1 : 0], E = S[3 + q];
    e32[q] = cut_f32(E);
    const float g = cut_f32(gap);
    const bool none = fabsf(e32[q]) <= round;
    far = far || !(none || fabsf(e32[q]) <= 2e-4f * fabsf(g));
    r32[q] = none || g == 0.f ? 0.f : __fdividef(1.f, g);
    const double r = widen(r32[q]);
    x[q] = E * r;
    x[q] = fma(fma(-x[q], gap, E), r, x[q]);
    x32[q] = e32[q] * r32[q];
  }
  const float me = fmaxf(fmaxf(fabsf(e32[0]), fabsf(e32[1])), fabsf(e32[2]));
  const float mx = fmaxf(fmaxf(fabsf(x32[0]), fabsf(x32[1])), fabsf(x32[2]));
  far = far || !(me * mx * mx <= round);
  if (far) {
    double Sl[6], Ul[9];
#pragma unroll
    for (int k = 0; k < 6; ++k) Sl[k] = S[k];
#pragma unroll
    for (int k = 0; k < 9; ++k) Ul[k] = U[k];
    jacobi64_finish(Sl, Ul);
#pragma unroll
    for (int k = 0; k < 3; ++k) S[k] = Sl[k];
#pragma unroll
    for (int k = 0; k < 9; ++k) U[k] = Ul[k];
  } else {
    x[0] += widen(0.5f * r32[0] * (-e32[1] * x32[2] - x32[1] * e32[2]));
    x[1] += widen(0.5f * r32[1] * (e32[0] * x32[2] - x32[0] * e32[2]));
    x[2] += widen(0.5f * r32[2] * (e32[0] * x32[1] + x32[0] * e32[1]));
    S[0] -= fma(S[3], x[0], S[4] * x[1]);
    S[1] += fma(S[3], x[0], -S[5] * x[2]);
    S[2] += fma(S[4], x[1], S[5] * x[2]);
    const double a = x[0], b = x[1], c = x[2];
    const double ha = 0.5 * a, hb = 0.5 * b, hc = 0.5 * c;
    double Q[9], T1[9];  // I + X + X^2 / 2
    Q[0] = 1.0 - fma(ha, a, hb * b);
    Q[1] = fma(-hb, c, a);
    Q[2] = fma(ha, c, b);
    Q[3] = fma(-hb, c, -a);
    Q[4] = 1.0 - fma(ha, a, hc * c);
    Q[5] = fma(-ha, b, c);
    Q[6] = fma(ha, c, -b);
    Q[7] = fma(-ha, b, -c);
    Q[8] = 1.0 - fma(hb, b, hc * c);
    mm(U, Q, T1);
#pragma unroll
    for (int k = 0; k < 9; ++k) U[k] = T1[k];
  }
  if (!(S[0] > 0.04 && S[1] > 0.04 && S[2] > 0.04 && S[0] < 9.0 && S[1] < 9.0 && S[2] < 9.0 && det3(A) > 0.0)) {
    double Al[9], Ul[9], Sl[3], sl[3], Vl[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      Al[k] = A[k];
      Ul[k] = U[k];
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) Sl[k] = S[k];
    left_gram_schmidt64(Al, Ul, Sl, sl, Vl);
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      U[k] = Ul[k];
      V[k] = Vl[k];
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      s[k] = sl[k];
      is[k] = 0.05 < sl[k] ? rcp64(sl[k]) : 0.0;
    }
    return true;
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    is[k] = rsqrt64_mid(S[k]);
    s[k] = S[k] * is[k];
  }
  if constexpr (WithV) {
    mTm(A, U, V);
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int k = 0; k < 3; ++k) V[r * 3 + k] *= is[k];
  }
  return false;
}

template <typename T>
MPM_DI T svd_clamp(T a) {
  return a >= T(0) ? (a > T(1e-6) ? a : T(1e-6)) : (a < T(-1e-6) ? a : T(-1e-6));
}

// Divided difference D = (e_j - e_i) / (s_j - s_i) of the return map's new
// singular values e = exp((1 - k) log s + k mean(log s)) (mpm_simulator.py:
// 172-180; k = delta_gamma / |eps_hat|, a = 1 - k), exact as s_j -> s_i:
//   e_j / e_i = (s_j / s_i)^a, so D = e_i a / s_i * E1(a L) * L / u
// with u = (s_j - s_i) / s_i, L = log1p(u) and E1(z) = expm1(z) / z.  For
// |u| < 1/64 both factors come from their Taylor series (L / u = 1 - u/2 +
// u^2/3 - u^3/4 + u^4/5, E1 = 1 + z/2 + z^2/6 + z^3/24 + z^4/120; truncation
// below 3e-11 and 2e-11); otherwise |s_j - s_i| is well above the rounding
// of s and the plain quotient is exact enough, as it is when a singular value
// sits at the return map's 0.05 floor.  ds = s_j - s_i and e_j - e_i are
// formed from s - 1 and e - 1.
MPM_DI float ret_map_dd(float si, float, float sj, float ds, float ei, float em1i, float em1j, float a) {
  if (si > 0.05f && sj > 0.05f) {
    const float u = ds / si;
    if (fabsf(u) < 0.015625f) {
      const float lg = fmaf(u, fmaf(u, fmaf(u, fmaf(u, 0.2f, -0.25f), 1.f / 3.f), -0.5f), 1.f);
      const float z = a * u * lg;
      const float e1 = fmaf(z, fmaf(z, fmaf(z, fmaf(z, 1.f / 120.f, 1.f / 24.f), 1.f / 6.f), 0.5f), 1.f);
      return ei * a / si * e1 * lg;
    }
  }
  return ds != 0.f ? (em1j - em1i) / ds : 0.f;
}
// FP64: the series below |u| < 2^-10 (L / u to u^5, E1 to z^5; truncation below
// 2e-19), above it the quotient keeps 1e-13
MPM_DI double ret_map_dd(double si, double ri, double sj, double ds, double ei, double em1i, double em1j, double a) {
  if (si > 0.05 && sj > 0.05) {
    const double u = ds * ri;
    if (fabs(u) < 0.0009765625) {
      const double lg =
          fma(u, fma(u, fma(u, fma(u, fma(u, -1.0 / 6.0, 0.2), -0.25), 1.0 / 3.0), -0.5), 1.0);
      const double z = a * u * lg;
      const double e1 =
          fma(z, fma(z, fma(z, fma(z, fma(z, 1.0 / 720.0, 1.0 / 120.0), 1.0 / 24.0), 1.0 / 6.0), 0.5), 1.0);
      return ei * a * ri * e1 * lg;
    }
  }
  return fabs(ds) > 1e-30 ? fast_div(em1j - em1i, ds) : 0.0;
}

// backward_svd (mpm_simulator.py:137-156, clamp 184-192) of the two functions
// p2g takes of the trial F's SVD, in a form without cancellation:
// the rotation R = U V^T (gradient gR) and, when the return map yields,
// newF = U diag(e) V^T (gradient gN).  Then gU = gR V + gN V diag(e),
// gV = gR^T U + gN^T U diag(e), and with M_R = U^T gR V, M_N = U^T gN V the
// reference's off-diagonal term
//   X_ij = (au_ij s_j + s_i av_ij) / clamp(s_j^2 - s_i^2)
// (au = U^T gU - gU^T U, av = V^T gV - gV^T V) is, identically,
//   X_ij = K_ij (s_j - s_i) / clamp((s_j - s_i)(s_j + s_i)),
//   K_ij = (M_R,ij - M_R,ji) + 1/2 [M_N,ij (D S + E) + M_N,ji (D S - E)]
// with S = s_i + s_j, E = e_i + e_j and D the divided difference of e
// (ret_map_dd; is = 1/s, read in FP64 only); s_j - s_i is taken from sm1 = s - 1.  The reference's numerator is a difference of terms of size
// |g| that leaves a value of size |g| (s_j - s_i), so in FP32 its rounding
// error is amplified by 1 / (s_j^2 - s_i^2), up to 1e6 at the clamp, whenever
// two singular values nearly coincide (near-isotropic deformation); K has no
// such cancellation.  The diagonal X_ii = gs_i (sigma_term) is unchanged.
// Returns X, the gradient of the SVD's input in the bases U, V (gA =
// U X V^T).  M_N, e and e - 1 (em1) are read only when `yield`.
template <typename T>
MPM_DI void svd3_bwd_factored_basis(const T* s, const T* is, const T* sm1, const T* MR, const T* MN, const T* e,
                                    const T* em1, T a, bool yield, const T* gs, T* X) {
#pragma unroll
  for (int i = 0; i < 3; ++i) X[i * 4] = gs[i];
  // each unordered pair (i, j) once: D and the clamped factor are symmetric in i, j
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const int i = q == 2 ? 1 : 0, j = q == 0 ? 1 : 2;
    const T ds = sm1[j] - sm1[i], sm = s[j] + s[i];  // s_j - s_i from s - 1: exact as s_j -> s_i
    const T f = fast_div(ds, svd_clamp(ds * sm));    // ds / clamp(s_j^2 - s_i^2); swapping i, j keeps it
    T Kij = MR[i * 3 + j] - MR[j * 3 + i];
    T Kji = -Kij;
    if (yield) {
      const T D = ret_map_dd(s[i], is[i], s[j], ds, e[i], em1[i], em1[j], a);
      const T se = e[i] + e[j];
      const T p = T(0.5) * (D * sm + se), m = T(0.5) * (D * sm - se);
      Kij += MN[i * 3 + j] * p + MN[j * 3 + i] * m;
      Kji += MN[j * 3 + i] * p + MN[i * 3 + j] * m;
    }
    X[i * 3 + j] = Kij * f;
    X[j * 3 + i] = Kji * f;
  }
}

}  // namespace mpm
