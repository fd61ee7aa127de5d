// The products, quotients and square roots of wf_int64.cuh on arrays, for
// test_34_gpu_int_arith.py.
#include <cuda_runtime.h>

#include "../weldformgpu_gb300/csrc/wf_int64.cuh"

__global__ void k_eval(int op, long n, const double* a, const double* b, double* out) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  out[i] = op == 0 ? mul_int(a[i], b[i]) : op == 1 ? div_int(a[i], b[i]) : sqrt_int(a[i]);
}

// op 0: a b, 1: a / b, 2: sqrt(a); host arrays of n; returns the CUDA error
extern "C" int int_arith(int op, long n, const double* a, const double* b, double* out) {
  double *da = nullptr, *db = nullptr, *dout = nullptr;
  const size_t bytes = sizeof(double) * (size_t)n;
  cudaError_t e = cudaMalloc(&da, bytes);
  if (e == cudaSuccess) e = cudaMalloc(&db, bytes);
  if (e == cudaSuccess) e = cudaMalloc(&dout, bytes);
  if (e == cudaSuccess) e = cudaMemcpy(da, a, bytes, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(db, b, bytes, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    k_eval<<<(unsigned)((n + 255) / 256), 256>>>(op, n, da, db, dout);
    e = cudaMemcpy(out, dout, bytes, cudaMemcpyDeviceToHost);
  }
  cudaFree(da);
  cudaFree(db);
  cudaFree(dout);
  return (int)e;
}
