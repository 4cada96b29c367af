// The scalar helpers of mpm_math.cuh and mpm_svd.cuh by number, for the host and the
// device tests (value in and out as FP64; FP32 ones go through a float).
#pragma once
#include "mpm_svd.cuh"

namespace calls {
MPM_DI double call(int what, double x) {
  switch (what) {
    case 0: return mpm::rcp64(x);
    case 1: return mpm::rsqrt64(x);
    case 2: return mpm::sqrt_pos(x);
    case 3: return mpm::log_strain64(1.0 + x, (1.0 + x) - 1.0);
    case 4: return mpm::expm1_strain64(x);
    case 5: return mpm::cut_f32(x);
    case 6: return mpm::widen((float)x);
    case 7: return mpm::exact_f64((float)x);
    case 8: return mpm::round_f32(x);
    case 9: return mpm::quot(3.0, x);
    case 10: return mpm::rcp64_mid(x);
    default: return mpm::rsqrt64_mid(x);
  }
}
}  // namespace calls
