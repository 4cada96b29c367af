// Device math of mpm_math.cuh and mpm_svd.cuh, compiled for the host and called on arrays.
#include "cuda_runtime.h"

#include "math_calls.h"

namespace {
// U, s, V and 1/s of n matrices, and whether the plain form was taken
template <typename T, typename F>
void each(long n, const T* A, T* U, T* s, T* V, int* plain, F&& svd) {
  for (long i = 0; i < n; ++i) plain[i] = svd(A + 9 * i, U + 9 * i, s + 3 * i, V + 9 * i);
}
// Jacobi sweeps on the symmetric m00, m11, m22, m01, m02, m12
template <typename T>
void sweeps(T* m, T* u) {
  for (int k = 0; k < 9; ++k) u[k] = k % 4 == 0;
  for (int sweep = 0; sweep < 12; ++sweep) {
    mpm::jacobi_rot(m[0], m[1], m[3], m[4], m[5], u, 0, 1);
    mpm::jacobi_rot(m[0], m[2], m[4], m[3], m[5], u, 0, 2);
    mpm::jacobi_rot(m[1], m[2], m[5], m[3], m[4], u, 1, 2);
  }
}
}  // namespace

extern "C" {
int scalar(int what, int n, const double* x, double* y) {
  for (int i = 0; i < n; ++i) y[i] = calls::call(what, x[i]);
  return 0;
}
// of I + D
void left32(long n, const float* D, float* U, float* s, float* V, int* plain) {
  each(n, D, U, s, V, plain, [](const float* d, float* u, float* sv, float* v) {
    float sm1[3], is[3], t = d[0] + d[4] + d[8], d2 = 0.f;
    for (int i = 0; i < 3; ++i)
      for (int j = 0; j < 3; ++j) d2 += d[i * 3 + j] * d[j * 3 + i];
    const float det = 1.f + (t + (0.5f * (t * t - d2) + mpm::det3(d)));
    return (int)mpm::svd3_left32<true>(d, det, u, sv, sm1, is, v);
  });
}
void left64(long n, const double* A, double* U, double* s, double* V, int* plain) {
  each(n, A, U, s, V, plain, [](const double* a, double* u, double* sv, double* v) {
    double is[3];
    return (int)mpm::svd3_left64<true>(a, u, sv, is, v);
  });
}
// V by Gram-Schmidt, whatever the deformation: of I + D, and of A
void by_gram_schmidt32(long n, const float* D, float* U, float* s, float* V, int* plain) {
  each(n, D, U, s, V, plain, [](const float* d, float* u, float* sv, float* v) {
    float m[6], B[9], norms[3];
    for (int i = 0; i < 3; ++i) m[i] = 2.f * d[4 * i] + mpm::dot3(d + 3 * i, d + 3 * i);
    m[3] = d[1] + d[3] + mpm::dot3(d, d + 3);
    m[4] = d[2] + d[6] + mpm::dot3(d, d + 6);
    m[5] = d[5] + d[7] + mpm::dot3(d + 3, d + 6);
    sweeps(m, u);
    mpm::mTm(d, u, B);
    for (int k = 0; k < 9; ++k) B[k] += u[k];
    mpm::left_gram_schmidt(u, m, B, norms, v);
    for (int k = 0; k < 3; ++k) sv[k] = norms[2] < 0.f && k == 2 ? -sqrtf(1.f + m[k]) : sqrtf(1.f + m[k]);
    return 1;
  });
}
void by_gram_schmidt64(long n, const double* A, double* U, double* s, double* V, int* plain) {
  each(n, A, U, s, V, plain, [](const double* a, double* u, double* sv, double* v) {
    double m[6] = {mpm::dot3(a, a),     mpm::dot3(a + 3, a + 3), mpm::dot3(a + 6, a + 6),
                   mpm::dot3(a, a + 3), mpm::dot3(a, a + 6),     mpm::dot3(a + 3, a + 6)};
    double B[9];
    sweeps(m, u);
    mpm::mTm(a, u, B);
    mpm::left_gram_schmidt(u, m, B, sv, v);
    return 1;
  });
}
}
