// pd_check.cu -- the elementary FP64 functions of the kernels off the serial order (pd_bond64.cuh) and
// CUDA's own on arrays, so that their errors can be measured.
#include "pd_bond64.cuh"
#include "pd_handle.h"

namespace pd {

__global__ void k_eval64(int op, long long n, const double* x, const double* y, double* out) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double a = x[i], b = y[i];
  double r = 0.0;
  switch (op) {
    case PD_EVAL_RSQRT: r = rsqrt3(a); break;
    case PD_EVAL_RCP: r = rcp3(a); break;
    case PD_EVAL_SQRT: r = sqrt_of(a, rsqrt3(a)); break;
    case PD_EVAL_LENGTH: r = sqrt_of(a, rsqrt3(a * (b * b)) * b); break;
    case PD_EVAL_QUOTIENT: r = quotient(a, b, 1.0 / b); break;
    case PD_EVAL_CUDA_RSQRT: r = rsqrt(a); break;
    case PD_EVAL_CUDA_SQRT: r = sqrt(a); break;
    case PD_EVAL_CUDA_QUOTIENT: r = a / b; break;
  }
  out[i] = r;
}

}  // namespace pd

extern "C" pd_status pd_eval64(int32_t op, int64_t n, const double* x, const double* y, double* out,
                               int32_t device) {
  if (op < PD_EVAL_RSQRT || op > PD_EVAL_CUDA_QUOTIENT) return pd_fail(PD_ERR_ARG, "unknown operation");
  if (n < 0 || (n > 0 && (!x || !y || !out))) return pd_fail(PD_ERR_ARG, "invalid arguments");
  if (n == 0) return PD_OK;
  PD_CUDA(cudaSetDevice(device));
  double* d = nullptr;
  const size_t bytes = sizeof(double) * n;
  PD_CUDA(cudaMalloc(&d, 3 * bytes));
  cudaError_t e = cudaMemcpy(d, x, bytes, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d + n, y, bytes, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    pd::k_eval64<<<(unsigned)((n + 255) / 256), 256>>>(op, n, d, d + n, d + 2 * n);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(out, d + 2 * n, bytes, cudaMemcpyDeviceToHost);
  cudaFree(d);
  if (e != cudaSuccess) return pd_fail(PD_ERR_CUDA, std::string("pd_eval64: ") + cudaGetErrorString(e));
  return PD_OK;
}
