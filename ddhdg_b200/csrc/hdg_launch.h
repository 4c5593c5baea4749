// The condensation, reconstruction and batched kernels by dimension: their
// addresses (attributes, occupancy) and launchers.  Each dimension is its own
// translation unit (hdg_condense_dim.cu, hdg_batch_dim.cu).
#pragma once

#include <cuda_runtime.h>

#include "hdg_batch.cuh"
#include "hdg_condense3.cuh"
#include "hdg_kernels.cuh"
#include "hdg_tables.h"

namespace ddhdg
{
  // one condense kernel of a (dim, degree)
  struct CondenseKernel
  {
    const void *fn = nullptr;
    // tables, parameters, grid, threads, dynamic shared memory, stream
    void (*launch)(const Tables &, const KParams &, int, int, size_t, cudaStream_t) = nullptr;
  };

  using ReconstructFn = void (*)(KParams, const double *, double *);

  // mixed: the FP32-Jacobian variant of the register kernel; false when the
  // degree has none (the caller rejects mixed precision there).  wide: its
  // wide form, where there is one (condense3_has_wide).
  template <int D>
  bool condense_kernels(int k, CondenseKernel &cf, ReconstructFn &rf, bool mixed, bool wide);

  template <int D>
  struct BatchKernels
  {
    static const void *condense_fn(int prec);
    static const void *reconstruct_fn();
    static void        condense(int prec, int grid, size_t smem, const BatchJob *jobs, const BatchTile *tiles,
                                int ntiles, int *counter, cudaStream_t s);
    static void reconstruct(int grid, size_t smem, const BatchJob *jobs, const BatchTile *tiles, int ntiles,
                            int *counter, cudaStream_t s);
  };

  template <int D, int K>
  inline void
  fill_ctab(const Tables &T, CTab<D, K> &C)
  {
    auto put = [](double *dst, size_t n, const std::vector<double> &src) {
      std::memcpy(dst, src.data(), std::min(n, src.size()) * sizeof(double));
    };
    put(C.phi_c, sizeof(C.phi_c) / sizeof(double), T.phi_c);
    put(C.RTk, sizeof(C.RTk) / sizeof(double), T.RTk);
    put(C.phi_f, sizeof(C.phi_f) / sizeof(double), T.phi_f);
    put(C.RTr, sizeof(C.RTr) / sizeof(double), T.RTr);
    put(C.RQk, sizeof(C.RQk) / sizeof(double), T.RQk);
    put(C.RQr, sizeof(C.RQr) / sizeof(double), T.RQr);
    put(C.xi, sizeof(C.xi) / sizeof(double), T.xi);
  }
} // namespace ddhdg
