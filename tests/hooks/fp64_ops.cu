// Device results of the FP64 quotient and half slope (physics.cuh) and of
// the expressions that they stand for, for arrays of operands.  Build with
// -fmad=false, as the FP64 units are.
#include <cuda_runtime.h>

#include "../../vac_gb300/csrc/physics.cuh"

using namespace vacgpu;

// out: 10 x n: div64, a/b, half slope and 0.5*limiter of minmod, the same of
// woodward, RN(1/b) and 1/b - RN(1/b) of rcp64, half_plus and 0.5*a + b
__global__ void k_ops(const double* a, const double* b, double* out, long long n) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double x = a[i], y = b[i];
  const Rcp64 r = rcp64(y);
  out[i] = div64(x, r);
  out[i + n] = x / y;
  out[i + 2 * n] = hlimiter_fn(LIM_MINMOD, x, y);
  out[i + 3 * n] = 0.5 * limiter_fn(LIM_MINMOD, x, y);
  out[i + 4 * n] = hlimiter_fn(LIM_WOODWARD, x, y);
  out[i + 5 * n] = 0.5 * limiter_fn(LIM_WOODWARD, x, y);
  out[i + 6 * n] = r.y;
  out[i + 7 * n] = r.yl;
  out[i + 8 * n] = half_plus(x, y);
  out[i + 9 * n] = 0.5 * x + y;
}

extern "C" int fp64_ops(const double* a, const double* b, double* out, long long n) {
  double *da = nullptr, *db = nullptr, *dout = nullptr;
  cudaError_t e = cudaMalloc(&da, 8 * n);
  if (e == cudaSuccess) e = cudaMalloc(&db, 8 * n);
  if (e == cudaSuccess) e = cudaMalloc(&dout, 80 * n);
  if (e == cudaSuccess) e = cudaMemcpy(da, a, 8 * n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(db, b, 8 * n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    k_ops<<<(unsigned)((n + 255) / 256), 256>>>(da, db, dout, n);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(out, dout, 80 * n, cudaMemcpyDeviceToHost);
  cudaFree(da);
  cudaFree(db);
  cudaFree(dout);
  return e != cudaSuccess;
}
