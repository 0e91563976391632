// The FP64 building blocks of amuse_gb300/csrc beside CUDA's own operators,
// element by element (tests/test_gpu_fp64_ops.py).
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "fp64_approx.cuh"
#include "g6_dev.h"

// got: the building block; want: CUDA's operator (rsqrt: 1/sqrt, two roundings).
__global__ void ops(int op, int n, const double *a, const double *b, double *got, double *want) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double x = a[i], y = b[i];
  switch (op) {
    case 0: got[i] = fp64::rcp64(x), want[i] = __drcp_rn(x); break;
    case 1: got[i] = fp64::rsqrt64(x), want[i] = 1.0 / __dsqrt_rn(x); break;
    case 2: got[i] = fp64::sqrt64(x), want[i] = __dsqrt_rn(x); break;
    case 3: got[i] = fp64::div64(x, y), want[i] = __ddiv_rn(x, y); break;
    case 4:
      got[i] = fp64::div_by(x, y, __drcp_rn(y), fp64::mid_range(y)), want[i] = __ddiv_rn(x, y);
      break;
    case 5: got[i] = fp64::Div(x).inv(), want[i] = __drcp_rn(x); break;
    case 6: got[i] = g6_div_const(x, 3.0, 1.0 / 3.0), want[i] = __ddiv_rn(x, 3.0); break;
    case 7: got[i] = g6_div_const(x, 12.0, 1.0 / 12.0), want[i] = __ddiv_rn(x, 12.0); break;
    case 8: got[i] = g6_div_const(x, 20.0, 1.0 / 20.0), want[i] = __ddiv_rn(x, 20.0); break;
  }
}

extern "C" int fp64_ops(int op, int n, const double *a, const double *b, double *got,
                        double *want) {
  double *d = nullptr;
  const size_t bytes = sizeof(double) * (size_t)n;
  if (cudaMalloc(&d, 4 * bytes) != cudaSuccess) return -1;
  cudaMemcpy(d, a, bytes, cudaMemcpyHostToDevice);
  cudaMemcpy(d + n, b, bytes, cudaMemcpyHostToDevice);
  ops<<<(n + 255) / 256, 256>>>(op, n, d, d + n, d + 2 * (size_t)n, d + 3 * (size_t)n);
  cudaMemcpy(got, d + 2 * (size_t)n, bytes, cudaMemcpyDeviceToHost);
  cudaMemcpy(want, d + 3 * (size_t)n, bytes, cudaMemcpyDeviceToHost);
  const int rc = cudaGetLastError() == cudaSuccess ? 0 : -2;
  cudaFree(d);
  return rc;
}
