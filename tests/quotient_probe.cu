// Test access to the pair code's shared quotient: out[i] = 1 where div_by differs from x / y.
#include "sc_pair.cuh"

__global__ void compare(const double* x, const double* y, int n, int* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double q = sc::div_by(x[i], y[i], sc::shared_rcp(y[i])), want = x[i] / y[i];
  out[i] = __double_as_longlong(q) != __double_as_longlong(want);
}

extern "C" int probe_quotients(const double* x, const double* y, int n, int* out) {
  double *dx = nullptr, *dy = nullptr;
  int* d = nullptr;
  const size_t b = n * sizeof(double);
  bool ok = cudaMalloc(&dx, b) == cudaSuccess && cudaMalloc(&dy, b) == cudaSuccess &&
            cudaMalloc(&d, n * sizeof(int)) == cudaSuccess &&
            cudaMemcpy(dx, x, b, cudaMemcpyHostToDevice) == cudaSuccess &&
            cudaMemcpy(dy, y, b, cudaMemcpyHostToDevice) == cudaSuccess;
  if (ok) {
    compare<<<(n + 255) / 256, 256>>>(dx, dy, n, d);
    ok = cudaMemcpy(out, d, n * sizeof(int), cudaMemcpyDeviceToHost) == cudaSuccess;
  }
  cudaFree(dx);
  cudaFree(dy);
  cudaFree(d);
  return ok ? 0 : -1;
}
