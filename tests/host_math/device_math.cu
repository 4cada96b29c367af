// The same helpers on the device, one value per thread.
#include <cuda_runtime.h>

#include "math_calls.h"

__global__ void k_call(int what, int n, const double* x, double* y) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = calls::call(what, x[i]);
}
// x, y: device arrays of n values; 0 or a CUDA error code
extern "C" int scalar(int what, int n, const double* x, double* y) {
  if (n > 0) k_call<<<(n + 127) / 128, 128>>>(what, n, x, y);
  const cudaError_t e = cudaGetLastError();
  return (int)(e != cudaSuccess ? e : cudaDeviceSynchronize());
}
