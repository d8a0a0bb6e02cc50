// The library's FP32 spreading weights (bspline_weights) at given offsets, for
// tests/test_kernel_edges.py: w[P][n] for u[n] in [0, 1], host buffers.
#include <cuda_runtime.h>

#include "common.cuh"

template <int P>
__global__ void weights_kernel(const float *u, int n, float *w) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float a[P], d[P];
  npme::bspline_weights<float, P, false>(u[i], a, d);
  for (int t = 0; t < P; t++) w[t * n + i] = a[t];
}

extern "C" int spline_weights(int order, int n, const float *u, float *w) {
  float *du = nullptr, *dw = nullptr;
  cudaError_t e = cudaMalloc(&du, sizeof(float) * n);
  if (e == cudaSuccess) e = cudaMalloc(&dw, sizeof(float) * n * order);
  if (e == cudaSuccess) e = cudaMemcpy(du, u, sizeof(float) * n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    const int b = (n + 255) / 256;
    switch (order) {
      case 4: weights_kernel<4><<<b, 256>>>(du, n, dw); break;
      case 6: weights_kernel<6><<<b, 256>>>(du, n, dw); break;
      case 8: weights_kernel<8><<<b, 256>>>(du, n, dw); break;
      case 10: weights_kernel<10><<<b, 256>>>(du, n, dw); break;
      case 12: weights_kernel<12><<<b, 256>>>(du, n, dw); break;
      case 14: weights_kernel<14><<<b, 256>>>(du, n, dw); break;
      case 16: weights_kernel<16><<<b, 256>>>(du, n, dw); break;
      default: e = cudaErrorInvalidValue;
    }
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e == cudaSuccess)
      e = cudaMemcpy(w, dw, sizeof(float) * n * order, cudaMemcpyDeviceToHost);
  }
  cudaFree(du);
  cudaFree(dw);
  return (int)e;
}
