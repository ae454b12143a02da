// block_loading of exact_dot.cuh on its own (test_gpu_pls_loading.py): out[j] = the
// loading of column j of z (rows x zp) with the scores sc, by one block.
#include "exact_dot.cuh"

namespace {

__global__ void __launch_bounds__(kgb::kEvalThreads) loading_kernel(const float* z, int zp, int p, const int* rows, int n,
                                                                    const float* sc, const int* zexp, float* out) {
  __shared__ float scratch[4 * kgb::kEvalThreads + 2 * kgb::kLoadChunk + 16];
  __shared__ float ld[1024];
  kgb::block_loading(z, zp, p, rows, n, sc, zexp, ld, scratch, threadIdx.x & 31, threadIdx.x >> 5);
  __syncthreads();
  for (int j = threadIdx.x; j < p; j += kgb::kEvalThreads) out[j] = ld[j];
}

}  // namespace

// z, sc, out: host memory; the rows are taken in order; p <= 1024
extern "C" int loading_probe(const float* z, int zp, int p, int n, const float* sc, const int* zexp, float* out) {
  float *dz = nullptr, *ds = nullptr, *dout = nullptr;
  int *de = nullptr, *dr = nullptr;
  int* rows = new int[n];
  for (int i = 0; i < n; ++i) rows[i] = i;
  const size_t zb = sizeof(float) * static_cast<size_t>(n) * zp;
  cudaError_t e = cudaMalloc(&dz, zb);
  if (e == cudaSuccess) e = cudaMalloc(&ds, sizeof(float) * n);
  if (e == cudaSuccess) e = cudaMalloc(&dout, sizeof(float) * p);
  if (e == cudaSuccess) e = cudaMalloc(&de, sizeof(int) * p);
  if (e == cudaSuccess) e = cudaMalloc(&dr, sizeof(int) * n);
  if (e == cudaSuccess) e = cudaMemcpy(dz, z, zb, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(ds, sc, sizeof(float) * n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(de, zexp, sizeof(int) * p, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(dr, rows, sizeof(int) * n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    loading_kernel<<<1, kgb::kEvalThreads>>>(dz, zp, p, dr, n, ds, de, dout);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(out, dout, sizeof(float) * p, cudaMemcpyDeviceToHost);
  cudaFree(dz);
  cudaFree(ds);
  cudaFree(dout);
  cudaFree(de);
  cudaFree(dr);
  delete[] rows;
  return static_cast<int>(e);
}
