// Condensation and reconstruction kernels of one dimension (DDHDG_DIM).
#include <algorithm>
#include <cstring>
#include <vector>

#include "hdg_launch.h"

namespace ddhdg
{
  namespace
  {
    template <int D, int K, typename JT, bool WIDE>
    void
    launch_condense(const Tables &T, const KParams &P, int grid, int threads, size_t smem, cudaStream_t s)
    {
      if constexpr (3 * Dims<D, K>::nb <= 32)
        {
          CTab<D, K> C;
          fill_ctab(T, C);
          condense3_kernel<D, K, JT, WIDE><<<grid, threads, smem, s>>>(P, C);
        }
      else
        condense2_kernel<D, K><<<grid, threads, smem, s>>>(P);
    }

    template <int D, int K>
    bool
    pick(CondenseKernel &cf, ReconstructFn &rf, bool mixed, bool wide)
    {
      // register kernel when one lane can own one row of the scalar system,
      // CTA-per-cell shared-memory kernel otherwise
      rf = reconstruct_kernel<D, K>;
      if constexpr (3 * Dims<D, K>::nb <= 32)
        {
          if (mixed)
            {
              cf.fn     = reinterpret_cast<const void *>(condense3_kernel<D, K, float>);
              cf.launch = launch_condense<D, K, float, false>;
            }
          else if (condense3_has_wide(Dims<D, K>::nb, 8) && wide)
            {
              constexpr bool W = condense3_has_wide(Dims<D, K>::nb, 8);
              cf.fn            = reinterpret_cast<const void *>(condense3_kernel<D, K, double, W>);
              cf.launch        = launch_condense<D, K, double, W>;
            }
          else
            {
              cf.fn     = reinterpret_cast<const void *>(condense3_kernel<D, K, double>);
              cf.launch = launch_condense<D, K, double, false>;
            }
          return true;
        }
      else
        {
          cf.fn     = reinterpret_cast<const void *>(condense2_kernel<D, K>);
          cf.launch = launch_condense<D, K, double, false>;
          return !mixed;
        }
    }
  } // namespace

  template <>
  bool
  condense_kernels<DDHDG_DIM>(int k, CondenseKernel &cf, ReconstructFn &rf, bool mixed, bool wide)
  {
    if (k == 1)
      return pick<DDHDG_DIM, 1>(cf, rf, mixed, wide);
    if (k == 2)
      return pick<DDHDG_DIM, 2>(cf, rf, mixed, wide);
#if DDHDG_DIM < 3
    if (k == 3)
      return pick<DDHDG_DIM, 3>(cf, rf, mixed, wide);
#endif
    return false;
  }
} // namespace ddhdg
