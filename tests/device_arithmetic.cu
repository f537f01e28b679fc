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
__global__ void k_pivot(int n, const T *c, const T *d, T *inv, T *quot, T *root) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  inv[i] = dg::pivot_inverse(d[i]);
  const dg::KeptPivot<T> p(dg::KeptPivot<T>::keep(d[i]));
  quot[i] = p.divide(c[i]);
  root[i] = p.inverse_root();
}
__global__ void k_widen(int n, const float *x, double *y) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = dg::to_f64(x[i]);
}
__global__ void k_narrow(int n, const double *x, float *y) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = dg::from_f64<float>(x[i]);
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

template <typename T>
static int pivot(int n, const T *c, const T *d, T *inv, T *quot, T *root) {
  T *dc = to_device(c, (size_t)n), *dd = to_device(d, (size_t)n), *o = to_device(inv, (size_t)n);
  T *q = to_device(quot, (size_t)n), *r = to_device(root, (size_t)n);
  if (!dc || !dd || !o || !q || !r) return -1;
  k_pivot<T><<<(n + 127) / 128, 128>>>(n, dc, dd, o, q, r);
  cudaFree(dc);
  cudaFree(dd);
  return finish(inv, o, (size_t)n) | finish(quot, q, (size_t)n) | finish(root, r, (size_t)n);
}
extern "C" int pivot_f64(int n, const double *c, const double *d, double *inv, double *quot, double *root) {
  return pivot(n, c, d, inv, quot, root);
}
extern "C" int pivot_f32(int n, const float *c, const float *d, float *inv, float *quot, float *root) {
  return pivot(n, c, d, inv, quot, root);
}
extern "C" int widen(int n, const float *x, double *y) {
  float *dx = to_device(x, (size_t)n);
  double *dy = to_device(y, (size_t)n);
  if (!dx || !dy) return -1;
  k_widen<<<(n + 127) / 128, 128>>>(n, dx, dy);
  cudaFree(dx);
  return finish(y, dy, (size_t)n);
}
extern "C" int narrow(int n, const double *x, float *y) {
  double *dx = to_device(x, (size_t)n);
  float *dy = to_device(y, (size_t)n);
  if (!dx || !dy) return -1;
  k_narrow<<<(n + 127) / 128, 128>>>(n, dx, dy);
  cudaFree(dx);
  return finish(y, dy, (size_t)n);
}
