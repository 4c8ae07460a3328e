// fix_mad (chorus-mhd_gb300/csrc/fixdot.cuh) on the device where a factor is the accumulator's own
// low or high word: mad_run(n, a, b, out) fills out[4 n] on the host.
#include <cuda_runtime.h>

#include "fixdot.cuh"

__global__ void mad_kernel(int n, const int* a, const int* b, long long* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int x = a[i], y = b[i];
  const int64_t xy = (int64_t)(((uint64_t)(uint32_t)y << 32) | (uint32_t)x);
  out[4 * i] = chorus::fix_mad(x, y, xy);  // low word x, high word y
  out[4 * i + 1] = chorus::fix_mad(y, x, xy);
  out[4 * i + 2] = chorus::fix_mad(x, x, (int64_t)(uint32_t)x);
  out[4 * i + 3] = chorus::fix_mad(x, y, (int64_t)x);
}

extern "C" int mad_run(int n, const int* a, const int* b, long long* out) {
  int *da = nullptr, *db = nullptr;
  long long* dout = nullptr;
  cudaError_t e = cudaMalloc(&da, sizeof(int) * n);
  if (e == cudaSuccess) e = cudaMalloc(&db, sizeof(int) * n);
  if (e == cudaSuccess) e = cudaMalloc(&dout, sizeof(long long) * 4 * n);
  if (e == cudaSuccess) e = cudaMemcpy(da, a, sizeof(int) * n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(db, b, sizeof(int) * n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    mad_kernel<<<(n + 127) / 128, 128>>>(n, da, db, dout);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(out, dout, sizeof(long long) * 4 * n, cudaMemcpyDeviceToHost);
  cudaFree(da);
  cudaFree(db);
  cudaFree(dout);
  return (int)e;
}
