// ff_round (ff.cuh) over an array, for test_gpu_band.py.
#include "ff.cuh"

__global__ void k_round(int n, const double *z, float2 *out)
{
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i < n) out[i] = ff_round(z[i]);
}

// host arrays z [n], out [n][2]; 0 or a CUDA error
extern "C" int probe_round(int n, const double *z, float *out)
{
  double *d = nullptr;
  float2 *o = nullptr;
  if (cudaMalloc(&d, n * 8ul) != cudaSuccess || cudaMalloc(&o, n * 8ul) != cudaSuccess) return -1;
  cudaMemcpy(d, z, n * 8ul, cudaMemcpyHostToDevice);
  k_round<<<(n + 255) / 256, 256>>>(n, d, o);
  cudaMemcpy(out, o, n * 8ul, cudaMemcpyDeviceToHost);
  const int r = (int)cudaGetLastError();
  cudaFree(d);
  cudaFree(o);
  return r;
}
