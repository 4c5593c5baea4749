// Batched condensation and reconstruction kernels of one dimension
// (DDHDG_DIM).
#include <algorithm>
#include <cstring>
#include <mutex>
#include <vector>

#include "hdg_launch.h"

namespace ddhdg
{
  namespace
  {
    // the unit-cell constant tables of every register-kernel degree
    template <int D>
    void
    fill_batch_tabs(BatchTabs<D> &C)
    {
      const double unit[3] = {1., 1., 1.};
      if constexpr (batch_warp<D, 1>)
        fill_ctab(build_tables(D, 1, unit), C.t1);
      if constexpr (batch_warp<D, 2>)
        fill_ctab(build_tables(D, 2, unit), C.t2);
      if constexpr (batch_warp<D, 3>)
        fill_ctab(build_tables(D, 3, unit), C.t3);
    }
  } // namespace

  template <int D>
  const void *
  BatchKernels<D>::condense_fn(int prec)
  {
    switch (prec)
      {
        case BatchFP64: return reinterpret_cast<const void *>(batch_condense_kernel<D, BatchFP64>);
        case BatchMixed: return reinterpret_cast<const void *>(batch_condense_kernel<D, BatchMixed>);
        default: return reinterpret_cast<const void *>(batch_condense_kernel<D, BatchBoth>);
      }
  }

  template <int D>
  const void *
  BatchKernels<D>::reconstruct_fn()
  {
    return reinterpret_cast<const void *>(batch_reconstruct_kernel<D>);
  }

  template <int D>
  void
  BatchKernels<D>::condense(int prec, int grid, size_t smem, const BatchJob *jobs, const BatchTile *tiles, int ntiles,
                            int *counter, cudaStream_t s)
  {
    static BatchTabs<D>   C; // filled once; the tables do not depend on the device
    static std::once_flag once;
    std::call_once(once, [] { fill_batch_tabs<D>(C); });
    if (prec == BatchFP64)
      batch_condense_kernel<D, BatchFP64><<<grid, batch_threads(D), smem, s>>>(jobs, tiles, ntiles, counter, C);
    else if (prec == BatchMixed)
      batch_condense_kernel<D, BatchMixed><<<grid, batch_threads(D), smem, s>>>(jobs, tiles, ntiles, counter, C);
    else
      batch_condense_kernel<D, BatchBoth><<<grid, batch_threads(D), smem, s>>>(jobs, tiles, ntiles, counter, C);
  }

  template <int D>
  void
  BatchKernels<D>::reconstruct(int grid, size_t smem, const BatchJob *jobs, const BatchTile *tiles, int ntiles,
                               int *counter, cudaStream_t s)
  {
    batch_reconstruct_kernel<D><<<grid, BatchRTPB, smem, s>>>(jobs, tiles, ntiles, counter);
  }

  template struct BatchKernels<DDHDG_DIM>;
} // namespace ddhdg
