// Global trace solve of the HDG system on a structured mesh (sm_100a, FP64):
// the host interface.  Kernels in hdg_ndkernels.cuh, plan and launch sequence
// in hdg_ndsolve.cu.
//
// The global trace matrix is the sum over cells of the condensed per-cell
// blocks tt (copy_local_to_global, src/np_solver.cpp:1293-1322, with the
// Dirichlet rows replaced by identity rows).  The reference factorises it
// with UMFPACK (src/np_solver.cpp:1326-1354).  Here it is factorised
// directly from the per-cell blocks by nested dissection: the cell grid is
// bisected recursively (longest axis first) and every tree node is a dense
// front over the trace dofs of the faces on its split plane (eliminated
// there) and of the faces on its boundary (kept for the parent).
//
//   leaves    one front per cell: the cell's block tt, with the faces on the
//             physical boundary eliminated (Dirichlet dofs are identity rows);
//             an interior cell's block is read where it is needed
//   upward    LU with partial pivoting of the eliminated block,
//             W = F_EE^-1 [F_EK | r_E], Schur complement F_KK - F_KE W
//   downward  x_E = y_E - W x_K from the root to the leaves
//
// The nodes of one height are processed together, whatever their shapes, in
// classes by the number of eliminated dofs: up to 36, one fused kernel with a
// CTA per front; up to 4096, an LU by panels over all fronts at once, blocked
// triangular solves and tensor-path products; beyond, cuSOLVER's LU in place
// of the panels.  The numeric sequence is captured in a CUDA graph on the
// second call with the same buffers and replayed afterwards.  Before the
// factorisation the rows are equilibrated: row g is scaled by
// 1 / max |row g| over the cells sharing it.
#pragma once

#include <cuda_runtime.h>
#include <cusolverDn.h>

#include <cstdint>
#include <memory>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

#include "../../include/ddhdg_b200.h"

namespace ddhdg
{
  // A kernel's dynamic shared-memory limit is process-wide state.  It is set
  // once per device to the opt-in maximum (minus the kernel's static shared
  // memory) and never lowered, so that contexts launching one kernel with
  // different sizes from several host threads cannot race on it.
  inline cudaError_t
  allow_full_dynamic_smem(const void *fn)
  {
    static std::mutex                                mu;
    static std::vector<std::pair<int, const void *>> done;
    int                                              dev = 0;
    cudaError_t                                      e   = cudaGetDevice(&dev);
    if (e != cudaSuccess)
      return e;
    std::lock_guard<std::mutex> lock(mu);
    for (auto &d : done)
      if (d.first == dev && d.second == fn)
        return cudaSuccess;
    cudaFuncAttributes fa;
    if ((e = cudaFuncGetAttributes(&fa, fn)) != cudaSuccess)
      return e;
    int optin = 0;
    if ((e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev)) != cudaSuccess)
      return e;
    if ((e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  optin - (int)fa.sharedSizeBytes)) != cudaSuccess)
      return e;
    done.push_back({dev, fn});
    return cudaSuccess;
  }

  class NDSolver
  {
  public:
    struct Mesh
    {
      int     dim            = 2;
      int     n[3]           = {1, 1, 1};
      int64_t face_off[3]    = {0, 0, 0};
      int     face_ext[3][3] = {{1, 1, 1}, {1, 1, 1}, {1, 1, 1}};
      int64_t ncells = 0, nfaces = 0;
      int     F  = 4;
      int     nd = 1; // trace dofs per face (enabled components x face nodes)
    };

    NDSolver();
    ~NDSolver();
    NDSolver(const NDSolver &)            = delete;
    NDSolver &operator=(const NDSolver &) = delete;

    // symbolic phase on the host: tree, fronts, maps and batches.  The plan
    // depends on the mesh shape only, so plans are kept in a small process-
    // wide cache: contexts of the same shape (the serving layer's requests,
    // a bias sweep's solvers) share it.
    int plan(const Mesh &M, std::string &err);

    // symbolic phase and the device buffers
    int build(const Mesh &M, std::string &err);

    // device bytes that build() allocates for the planned mesh (each
    // allocation rounded up to the allocator's 2 MiB granularity); plan()
    // must have succeeded
    int64_t planned_device_bytes() const;

    // capture and replay of the numeric sequence on (default) or off
    void set_graphs(bool on);

    // numeric phase: x (global trace dofs) from the per-cell condensed
    // blocks.  check = false: the caller reads the pivot status later
    // (check_info), so that solves on several streams overlap.
    int solve(const double *tt, const double *rhs, const int32_t *dflag, const double *dval, int Nt,
              double *x, cudaStream_t s, int sm_count, std::string &err, bool check = true);

    // singular fronts (outside any graph: a host read)
    int check_info(cudaStream_t s, std::string &err);

    struct Plan; // defined in hdg_ndsolve.cu

  private:
    struct Key
    {
      const void *tt, *rhs, *dflag, *dval, *x;
      int         sm;
      bool
      operator==(const Key &o) const
      {
        return tt == o.tt && rhs == o.rhs && dflag == o.dflag && dval == o.dval && x == o.x && sm == o.sm;
      }
    };
    struct Device; // device buffers

    int  enqueue(const double *tt, const double *rhs, const int32_t *dflag, const double *dval, int Nt, double *x,
                 cudaStream_t s, int sm_count, std::string &err);
    void release();

    std::shared_ptr<const Plan> plan_;
    std::unique_ptr<Device>     dev_;
    bool                        built_ = false;
    cudaStream_t                cap_   = nullptr; // stream the graph is captured on
    cudaGraphExec_t             exec_  = nullptr;
    cusolverDnHandle_t          dn_    = nullptr; // only for fronts beyond the panel kernel
    Key                         key_{};
    bool                        graphs_ok_  = true; // capture works in this build
    bool                        use_graphs_ = true; // the caller wants graphs
  };
} // namespace ddhdg
