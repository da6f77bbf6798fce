// fp64_shim.cu -- test helper: evp_fp64.cuh's quotient and square root on the
// device, for comparison with the correctly rounded results.
#include "evp_fp64.cuh"

namespace {
__global__ void k_quot(int n, const double *a, const double *b, double *q, int *ok) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  q[i] = evp::fp64_quot(a[i], b[i], evp::fp64_recip(b[i]));
  ok[i] = (evp::fp64_divisor(b[i]) && evp::fp64_mid_abs(a[i])) ||
          (evp::fp64_mid(b[i]) && evp::fp64_dividend(a[i]));
}
__global__ void k_sqrt(int n, const double *x, double *r, int *ok) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  r[i] = evp::fp64_sqrt(x[i]);
  ok[i] = evp::fp64_radicand(x[i]);
}
}  // namespace

extern "C" {
// op 0: out = a / b, op 1: out = sqrt(a).  ok: whether the functions cover the
// operands.  Returns the CUDA error code.
int fp64_run(int op, int n, const double *a, const double *b, double *out, int *ok) {
  double *d = nullptr;
  int *o = nullptr;
  cudaError_t e = cudaMalloc(&d, sizeof(double) * 3 * (size_t)n);
  if (e == cudaSuccess) e = cudaMalloc(&o, sizeof(int) * (size_t)n);
  if (e == cudaSuccess) e = cudaMemcpy(d, a, 8 * (size_t)n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess && op == 0) e = cudaMemcpy(d + n, b, 8 * (size_t)n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    const int g = (n + 255) / 256;
    if (op == 0)
      k_quot<<<g, 256>>>(n, d, d + n, d + 2 * (size_t)n, o);
    else
      k_sqrt<<<g, 256>>>(n, d, d + 2 * (size_t)n, o);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(out, d + 2 * (size_t)n, 8 * (size_t)n, cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemcpy(ok, o, 4 * (size_t)n, cudaMemcpyDeviceToHost);
  cudaFree(d);
  cudaFree(o);
  return (int)e;
}
}
