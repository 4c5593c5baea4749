// Device functions of the kernels, called on arrays from host memory (built
// by tests/device_probe.py).  Every call returns the CUDA error code.
#include <cuda_runtime.h>

#include "hdg_reciprocal.cuh"

namespace
{
  __global__ void
  reciprocal_kernel(const double *x, double *r, int n, bool scaled)
  {
    using namespace ddhdg;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n)
      r[i] = scaled ? reciprocal_scaled(x[i] * ReciprocalScale) * ReciprocalScale :
                      reciprocal(x[i], reciprocal_normal(x[i]));
  }
} // namespace

// scaled: reciprocal_scaled, back in the scale of x
extern "C" int
probe_reciprocal(const double *x, double *r, int n, int scaled)
{
  double       *d = nullptr;
  const size_t  b = (size_t)n * sizeof(double);
  cudaError_t   e = cudaMalloc(reinterpret_cast<void **>(&d), 2 * b);
  if (e != cudaSuccess)
    return (int)e;
  e = cudaMemcpy(d, x, b, cudaMemcpyHostToDevice);
  if (e == cudaSuccess)
    {
      reciprocal_kernel<<<(n + 255) / 256, 256>>>(d, d + n, n, scaled != 0);
      e = cudaGetLastError();
    }
  if (e == cudaSuccess)
    e = cudaMemcpy(r, d + n, b, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return (int)e;
}
