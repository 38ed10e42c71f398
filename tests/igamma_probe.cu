// The device's incomplete gamma functions over arrays, for test_gpu_igamma.py.
#include "igamma.cuh"

namespace {
__global__ void k_probe(const double *lf, int n, const int *a, const double *x, double *up, double *lo, int *st)
{
  const int i = blockIdx.x * 128 + threadIdx.x;
  if (i >= n) return;
  IgBase u{lf, 0}, l{lf, 0};
  up[i] = u.upper(a[i], x[i]);
  lo[i] = l.lower(a[i], x[i]);
  st[2 * i] = u.st;
  st[2 * i + 1] = l.st;
}
}  // namespace

extern "C" int probe_table() { return TW_LF_N; }

// host arrays: lf [TW_LF_N], the others [n] (st [2 n]); 0 or a CUDA error
extern "C" int probe(const double *lf, int n, const int *a, const double *x, double *up, double *lo, int *st)
{
  double *d = nullptr;
  int *k = nullptr;
  if (cudaMalloc(&d, (TW_LF_N + 3ul * n) * 8) != cudaSuccess || cudaMalloc(&k, 3ul * n * 4) != cudaSuccess) return -1;
  cudaMemcpy(d, lf, TW_LF_N * 8ul, cudaMemcpyHostToDevice);
  cudaMemcpy(d + TW_LF_N, x, n * 8ul, cudaMemcpyHostToDevice);
  cudaMemcpy(k, a, n * 4ul, cudaMemcpyHostToDevice);
  double *du = d + TW_LF_N + n, *dl = du + n;
  k_probe<<<(n + 127) / 128, 128>>>(d, n, k, d + TW_LF_N, du, dl, k + n);
  cudaMemcpy(up, du, n * 8ul, cudaMemcpyDeviceToHost);
  cudaMemcpy(lo, dl, n * 8ul, cudaMemcpyDeviceToHost);
  cudaMemcpy(st, k + n, 2ul * n * 4, cudaMemcpyDeviceToHost);
  const int r = (int)cudaGetLastError();
  cudaFree(d);
  cudaFree(k);
  return r;
}
