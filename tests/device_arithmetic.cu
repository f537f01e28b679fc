// The kernels' own arithmetic, one thread per value, for test_device_arithmetic.py
#include <cuda_runtime.h>

#include "dg_kernels.cuh"

namespace {

__global__ void k_split_value(int n, const int *d, const int *ex, double *out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int q[dg::kSplit];
  for (int s = 0; s < dg::kSplit; s++) q[s] = d[dg::kSplit * i + s];
  out[i] = dg::split_value(q, ex[i]);
}

template <typename T>
T *to_device(const T *h, size_t n) {
  T *d = nullptr;
  if (cudaMalloc(&d, n * sizeof(T)) != cudaSuccess) return nullptr;
  cudaMemcpy(d, h, n * sizeof(T), cudaMemcpyHostToDevice);
  return d;
}
template <typename T>
int finish(T *h, T *d, size_t n) {
  cudaMemcpy(h, d, n * sizeof(T), cudaMemcpyDeviceToHost);
  cudaFree(d);
  return (int)cudaGetLastError();
}

}  // namespace

extern "C" int split_value(int n, const int *d, const int *ex, double *out) {
  int *dd = to_device(d, (size_t)n * dg::kSplit), *de = to_device(ex, (size_t)n);
  double *o = to_device(out, (size_t)n);
  if (!dd || !de || !o) return -1;
  k_split_value<<<(n + 127) / 128, 128>>>(n, dd, de, o);
  cudaFree(dd);
  cudaFree(de);
  return finish(out, o, (size_t)n);
}
