// FP64 tensor-path tile product shared by the kernels (sm_100a).
#pragma once

#include <cuda_runtime.h>

namespace ddhdg
{
  // D += A B for one 8x8x4 FP64 tile on the tensor path (mma.sync m8n8k4):
  // lane l holds A[l/4][l%4], B[l%4][l/4] and D[l/4][2(l%4) + {0,1}]
  __device__ __forceinline__ void
  dmma8x8x4(double &d0, double &d1, double a, double b)
  {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
  }
} // namespace ddhdg
