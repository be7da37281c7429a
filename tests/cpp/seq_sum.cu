// k_seq_sum over a host array, for tests/test_gpu_ic_sum.py.
#include "vh_seq_sum.cuh"

extern "C" int seq_sum(const double* t, long n, double* sum) {
  double *d = nullptr, *o = nullptr;
  cudaError_t e = cudaMalloc(&d, sizeof(double) * (n + 1));
  if (e == cudaSuccess) e = cudaMalloc(&o, sizeof(double));
  if (e == cudaSuccess) e = cudaMemcpy(d, t, sizeof(double) * n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    vh::icr::k_seq_sum<<<1, vh::icr::kSumThreads>>>(d, n, o);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(sum, o, sizeof(double), cudaMemcpyDeviceToHost);
  cudaFree(d);
  cudaFree(o);
  return (int)e;
}
