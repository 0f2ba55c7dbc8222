// The strip walk's reciprocal and exponential (csrc/walk_strip.cuh) over arrays,
// beside the compiler's division and exp().
#include "../../slsimlib_b200/csrc/walk_strip.cuh"

using namespace glb;

namespace {
__global__ void k_math(const double *x, size_t n, const ExpTab *tab, double *rcp, double *div, double *mine,
                       double *cuda) {
  __shared__ ExpTab E;
  strip_exp_table(E, tab);
  __syncthreads();
  const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  rcp[i] = strip_rcp(x[i]);
  div[i] = 1.0 / x[i];
  mine[i] = strip_exp_neg(x[i], E);
  cuda[i] = exp(-x[i]);
}
}  // namespace

// out: 4 n doubles {1/x, CUDA's, exp(-x), CUDA's}; returns the CUDA status.
extern "C" int strip_math(const double *x, size_t n, double *out) {
  static const ExpTab host = make_exp_table();
  double *d = nullptr;
  ExpTab *tab = nullptr;
  cudaError_t e = cudaMalloc((void **)&d, 5 * n * sizeof(double));
  if (e == cudaSuccess) e = cudaMalloc((void **)&tab, sizeof(ExpTab));
  if (e == cudaSuccess) e = cudaMemcpy(tab, &host, sizeof(ExpTab), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d, x, n * sizeof(double), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    k_math<<<(unsigned)((n + 255) / 256), 256>>>(d, n, tab, d + n, d + 2 * n, d + 3 * n, d + 4 * n);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(out, d + n, 4 * n * sizeof(double), cudaMemcpyDeviceToHost);
  cudaFree(d);
  cudaFree(tab);
  return (int)e;
}
