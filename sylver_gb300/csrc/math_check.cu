// Self-check of the scalar arithmetic of pivot.cuh: out[i] = op(a[i], b[i]).
#include "../../include/sylver_gb300.h"
#include "numeric.hpp"
#include "pivot.cuh"

namespace sylver_gb300 {

namespace {

__global__ void __launch_bounds__(256) k_pivot_math(int op, const double* __restrict__ a,
                                                    const double* __restrict__ b,
                                                    double* __restrict__ out, long n) {
  for (long i = blockIdx.x * 256l + threadIdx.x; i < n; i += gridDim.x * 256l) {
    const double x = a[i];
    const float f = (float)x;
    switch (op) {
      case 0: out[i] = div64(x, b[i]); break;
      case 1: out[i] = pivot_rsqrt(x); break;
      case 2: out[i] = pivot_sqrt(x, pivot_rsqrt(x)); break;
      case 3: out[i] = (double)pivot_rsqrt(f); break;
      default: out[i] = (double)pivot_sqrt(f, pivot_rsqrt(f)); break;
    }
  }
}

}  // namespace

}  // namespace sylver_gb300

using namespace sylver_gb300;

extern "C" int sylver_gb300_pivot_math(int op, long n, double const* a, double const* b,
                                       double* out) {
  if (op < 0 || op > 4 || n < 1 || !a || !b || !out) return SYLVER_ERROR_UNKNOWN;
  Runtime& rt = Runtime::get();
  if (!rt.init()) return SYLVER_ERROR_CUDA_UNKNOWN;
  try {
    DevMem da, db, dout;
    const size_t bytes = (size_t)n * sizeof(double);
    da.ensure(bytes);
    db.ensure(bytes);
    dout.ensure(bytes);
    SG_CUDA(cudaMemcpyAsync(da.p, a, bytes, cudaMemcpyHostToDevice, rt.stream));
    SG_CUDA(cudaMemcpyAsync(db.p, b, bytes, cudaMemcpyHostToDevice, rt.stream));
    k_pivot_math<<<1024, 256, 0, rt.stream>>>(op, da.as<double>(), db.as<double>(),
                                              dout.as<double>(), n);
    SG_CUDA(cudaGetLastError());
    SG_CUDA(cudaMemcpyAsync(out, dout.p, bytes, cudaMemcpyDeviceToHost, rt.stream));
    SG_CUDA(cudaStreamSynchronize(rt.stream));
    return SYLVER_SUCCESS;
  } catch (const std::exception&) {
    return SYLVER_ERROR_CUDA_UNKNOWN;
  }
}
