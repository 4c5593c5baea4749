// Plan and launch sequence of the nested-dissection trace solve (see
// hdg_ndsolve.h; the kernels are in hdg_ndkernels.cuh).
#include "hdg_ndsolve.h"

#include <algorithm>
#include <array>
#include <map>

#include "hdg_ndkernels.cuh"

namespace ddhdg
{
  namespace
  {
    int
    bad(std::string &err, const char *msg, int code = DDHDG_BAD_ARG)
    {
      err = msg;
      return code;
    }

    // elimination classes of a node
    enum Class
    {
      Small4,
      Small12,
      Small20,
      Small28,
      Small36, // nd_small_kernel, by its register array size
      Panels,  // nd_panel_kernel / nd_update_kernel, triangular solves, GEMM
      Library  // cuSOLVER LU, then as above
    };

    constexpr int    PanelRows  = NDPanelT * NDPanelC; // rows the panel kernel can hold
    constexpr size_t SmallSmem  = 200 * 1024;
    constexpr int    RootRows   = 24576; // rows of a single right-hand side in shared memory (192 KB)
    constexpr int    BatchNodes = 65535; // fronts per launch of the panel kernels (grid y)

    Class
    class_of(int nE, int nK)
    {
      if (nE <= NDSmallE && nd_small_smem(nd_small_class(nE), nK) <= SmallSmem)
        return nE <= 4 ? Small4 : nE <= 12 ? Small12 : nE <= 20 ? Small20 : nE <= 28 ? Small28 : Small36;
      return nE <= PanelRows ? Panels : Library;
    }

    struct Batch
    {
      Class   cls = Small4;
      bool    leaf = false;
      int     node0 = 0, count = 0; // nodes in the device order
      int     maxE = 0, maxK = 0, maxld = 0;
      int64_t esize = 0, lusize = 0, tisize = 0, psize = 0; // scratch (elements)
    };

    struct HostNode
    {
      int                lo[3], hi[3];
      std::array<int, 2> child{{-1, -1}};
      int                height = 0;
      int64_t            cell   = -1;
      unsigned           bmask  = 0; // faces on the physical boundary (bit 2 axis + side)
      int                nE = 0, nK = 0;
      int64_t            koff = 0, doff = 0;
      int                map = 0;
    };
  } // namespace

  struct NDSolver::Plan
  {
    Mesh                 M;
    std::vector<NDNode>  nodes; // in batch order
    std::vector<Batch>   batches; // by height
    std::vector<int32_t> fdofs, maps;
    std::vector<int64_t> cell_faces;
    int64_t              front_total = 0;
    int64_t              e_total = 0, lu_total = 0, ti_total = 0, p_total = 0; // largest batch
    int                  lib_nE = 0;
    std::vector<HostNode> tree; // only while planning

    size_t
    bytes() const
    {
      return nodes.size() * sizeof(NDNode) + (fdofs.size() + maps.size()) * 4 + cell_faces.size() * 8;
    }

    int64_t
    face_at(int a, const int co[3]) const
    {
      int64_t idx = 0, stride = 1;
      for (int b = 0; b < M.dim; ++b)
        {
          idx += co[b] * stride;
          stride *= M.face_ext[a][b];
        }
      return M.face_off[a] + idx;
    }

    int64_t
    face_of_cell(int64_t cell, int f) const
    {
      int       co[3];
      const int n1 = M.dim > 1 ? M.n[1] : 1;
      co[0]        = (int)(cell % M.n[0]);
      co[1]        = (int)((cell / M.n[0]) % n1);
      co[2]        = (int)(cell / ((int64_t)M.n[0] * n1));
      co[f / 2] += f % 2;
      return face_at(f / 2, co);
    }

    // faces of axis a at face coordinate p, over the box's extent in the
    // other axes, in increasing id order
    void
    plane_faces(int a, int p, const int lo[3], const int hi[3], std::vector<int64_t> &out) const
    {
      int co[3], l[3], h[3];
      for (int b = 0; b < 3; ++b)
        {
          l[b] = (b == a) ? p : lo[b];
          h[b] = (b == a) ? p + 1 : hi[b];
        }
      for (co[2] = l[2]; co[2] < h[2]; ++co[2])
        for (co[1] = l[1]; co[1] < h[1]; ++co[1])
          for (co[0] = l[0]; co[0] < h[0]; ++co[0])
            out.push_back(face_at(a, co));
    }

    int
    split_axis(const HostNode &h) const
    {
      int s = 0;
      for (int b = 1; b < M.dim; ++b)
        if (h.hi[b] - h.lo[b] > h.hi[s] - h.lo[s])
          s = b;
      return s;
    }

    int
    make_node(const int lo[3], const int hi[3])
    {
      const int id = (int)tree.size();
      tree.emplace_back();
      int64_t vol = 1, kept = 0;
      for (int b = 0; b < 3; ++b)
        {
          tree[id].lo[b] = lo[b];
          tree[id].hi[b] = hi[b];
          vol *= hi[b] - lo[b];
        }
      unsigned msk = 0;
      for (int a = 0; a < M.dim; ++a)
        {
          const int64_t area = vol / (hi[a] - lo[a]);
          if (lo[a] == 0)
            msk |= 1u << (2 * a);
          else
            kept += area;
          if (hi[a] == M.n[a])
            msk |= 2u << (2 * a);
          else
            kept += area;
        }
      tree[id].bmask = msk;
      tree[id].nK    = (int)kept * M.nd;
      if (vol == 1)
        {
          const int n1     = M.dim > 1 ? M.n[1] : 1;
          tree[id].cell    = lo[0] + (int64_t)M.n[0] * (lo[1] + (int64_t)n1 * lo[2]);
          tree[id].nE      = (M.F - (int)kept) * M.nd;
          return id;
        }
      const int s     = split_axis(tree[id]);
      const int mid   = lo[s] + (hi[s] - lo[s]) / 2;
      int       hl[3] = {hi[0], hi[1], hi[2]}, lh[3] = {lo[0], lo[1], lo[2]};
      hl[s]           = mid;
      lh[s]           = mid;
      tree[id].nE     = (int)(vol / (hi[s] - lo[s])) * M.nd;
      const int c0    = make_node(lo, hl);
      const int c1    = make_node(lh, hi);
      HostNode &h     = tree[id]; // after the recursion: the tree may have grown
      h.child         = {{c0, c1}};
      h.height        = 1 + std::max(tree[c0].height, tree[c1].height);
      return id;
    }

    // dof list [E, K] of a node
    void
    fill_dofs(const HostNode &h, std::vector<int64_t> &E, std::vector<int64_t> &K)
    {
      E.clear();
      K.clear();
      if (h.cell >= 0)
        {
          for (int f = 0; f < M.F; ++f)
            ((h.bmask >> f & 1u) ? E : K).push_back(cell_faces[h.cell * M.F + f]);
        }
      else
        {
          const int s = split_axis(h);
          plane_faces(s, h.lo[s] + (h.hi[s] - h.lo[s]) / 2, h.lo, h.hi, E);
          for (int a = 0; a < M.dim; ++a)
            {
              if (h.lo[a] > 0)
                plane_faces(a, h.lo[a], h.lo, h.hi, K);
              if (h.hi[a] < M.n[a])
                plane_faces(a, h.hi[a], h.lo, h.hi, K);
            }
          std::sort(K.begin(), K.end());
        }
      int32_t *d = fdofs.data() + h.doff;
      for (auto *v : {&E, &K})
        for (int64_t f : *v)
          for (int j = 0; j < M.nd; ++j)
            *d++ = (int32_t)(f * M.nd + j);
    }

    int
    make(const Mesh &mesh, std::string &err)
    {
      M = mesh;
      if (M.F > 6 || M.dim < 1 || M.dim > 3)
        return bad(err, "unsupported mesh for the nested-dissection solve");
      if (M.nfaces * (int64_t)M.nd > INT32_MAX)
        return bad(err, "too many trace dofs for 32-bit dof lists");
      cell_faces.assign(M.ncells * M.F, 0);
      for (int64_t c = 0; c < M.ncells; ++c)
        for (int f = 0; f < M.F; ++f)
          cell_faces[c * M.F + f] = face_of_cell(c, f);
      int lo[3] = {0, 0, 0}, hi[3] = {M.n[0], M.dim > 1 ? M.n[1] : 1, M.dim > 2 ? M.n[2] : 1};
      make_node(lo, hi);
      // device order: by height, class and size; interior cells have nothing
      // to eliminate and no front
      std::vector<int>   ids;
      std::vector<Class> cls(tree.size());
      int64_t            doff = 0;
      for (int i = 0; i < (int)tree.size(); ++i)
        {
          HostNode &h = tree[i];
          if (h.nE == 0)
            continue;
          cls[i] = class_of(h.nE, h.nK);
          h.doff = doff;
          doff += h.nE + h.nK;
          ids.push_back(i);
        }
      std::stable_sort(ids.begin(), ids.end(), [&](int a, int b) {
        const HostNode &A = tree[a], &B = tree[b];
        if (A.height != B.height)
          return A.height < B.height;
        if (cls[a] != cls[b])
          return cls[a] < cls[b];
        if (A.nE != B.nE)
          return A.nE > B.nE;
        return A.nK > B.nK;
      });
      fdofs.assign(doff, 0);
      nodes.clear();
      nodes.reserve(ids.size());
      batches.clear();
      const auto even = [](int64_t v) { return (v + 1) & ~(int64_t)1; };
      int        last_h = -1;
      for (int id : ids)
        {
          HostNode &h = tree[id];
          if (batches.empty() || h.height != last_h || batches.back().cls != cls[id] ||
              (cls[id] >= Panels && batches.back().count == BatchNodes))
            {
              Batch b;
              b.cls   = cls[id];
              b.leaf  = h.height == 0;
              b.node0 = (int)nodes.size();
              batches.push_back(b);
              last_h = h.height;
            }
          Batch &b = batches.back();
          NDNode n{};
          n.nE  = h.nE;
          n.nK  = h.nK;
          n.nEp = (int)even(h.nE);
          n.ld  = n.nEp + (int)even(h.nK);
          h.koff = n.koff = front_total;
          front_total += (int64_t)n.ld * (n.nK + 1);
          n.doff  = h.doff;
          n.cell  = h.cell;
          n.eoff  = b.esize;
          n.luoff = b.lusize;
          n.tioff = b.tisize;
          n.poff  = b.psize;
          if (b.cls >= Panels)
            {
              b.esize += (int64_t)n.ld * n.nE;
              b.lusize += (int64_t)n.nEp * n.nE;
              b.tisize += (int64_t)((n.nE + NDPanel - 1) / NDPanel) * 2 * NDPanel * NDPanel;
              b.psize += n.nE;
            }
          if (b.cls == Library)
            lib_nE = std::max(lib_nE, n.nE);
          b.count += 1;
          b.maxE  = std::max(b.maxE, n.nE);
          b.maxK  = std::max(b.maxK, n.nK);
          b.maxld = std::max(b.maxld, n.ld);
          nodes.push_back(n);
        }
      for (const auto &b : batches)
        {
          e_total  = std::max(e_total, b.esize);
          lu_total = std::max(lu_total, b.lusize);
          ti_total = std::max(ti_total, b.tisize);
          p_total  = std::max(p_total, b.psize);
        }
      // dof lists, and the maps of each node shape (they depend on the box's
      // extents and on which of its sides lie on the physical boundary)
      std::map<std::array<int, 4>, int> shapes;
      std::vector<int32_t>              pos(M.nfaces * (int64_t)M.nd, -1);
      std::vector<int64_t>              E, K;
      for (int q = 0; q < (int)ids.size(); ++q)
        fill_dofs(tree[ids[q]], E, K);
      std::vector<int32_t> kid_dofs;
      for (int q = 0; q < (int)ids.size(); ++q)
        {
          HostNode &h = tree[ids[q]];
          NDNode   &n = nodes[q];
          for (int s = 0; s < 2; ++s)
            {
              n.ccell[s] = -1;
              if (h.cell >= 0)
                continue;
              const HostNode &c = tree[h.child[s]];
              n.cnK[s]          = c.nK;
              if (c.nE == 0)
                n.ccell[s] = c.cell;
              else
                {
                  n.coff[s] = c.koff;
                  n.cEp[s]  = (int)even(c.nE);
                  n.cld[s]  = n.cEp[s] + (int)even(c.nK);
                }
              if (n.ccell[s] >= 0 && class_of(h.nE, h.nK) >= Panels)
                return bad(err, "nested dissection: a large front over an interior cell");
            }
          const std::array<int, 4> key{
            {h.hi[0] - h.lo[0], h.hi[1] - h.lo[1], h.hi[2] - h.lo[2], (int)h.bmask}};
          auto it = shapes.find(key);
          if (it == shapes.end())
            {
              it = shapes.emplace(key, (int)maps.size()).first;
              const int32_t *d = fdofs.data() + h.doff;
              if (h.cell >= 0)
                {
                  // position -> the cell's local dof, faces on the boundary first
                  for (int part = 1; part >= 0; --part)
                    for (int f = 0; f < M.F; ++f)
                      if ((int)(h.bmask >> f & 1u) == part)
                        for (int j = 0; j < M.nd; ++j)
                          maps.push_back(f * M.nd + j);
                }
              else
                {
                  const int nF = h.nE + h.nK;
                  for (int i = 0; i < nF; ++i)
                    pos[d[i]] = i;
                  const size_t m0 = maps.size();
                  maps.resize(m0 + 2 * (size_t)h.nE + h.nK, -1);
                  for (int s = 0; s < 2; ++s)
                    {
                      const HostNode &c  = tree[h.child[s]];
                      const int32_t  *cd = nullptr;
                      if (c.nE > 0)
                        cd = fdofs.data() + c.doff + c.nE;
                      else
                        {
                          kid_dofs.clear();
                          for (int f = 0; f < M.F; ++f)
                            for (int j = 0; j < M.nd; ++j)
                              kid_dofs.push_back((int32_t)(cell_faces[c.cell * M.F + f] * M.nd + j));
                          cd = kid_dofs.data();
                        }
                      for (int k = 0; k < c.nK; ++k)
                        {
                          const int p = pos[cd[k]];
                          if (p < 0)
                            return bad(err, "nested dissection: a kept dof is missing from the parent front");
                          if (p < h.nE)
                            maps[m0 + (size_t)s * h.nE + p] = k;
                          else
                            maps[m0 + h.nE + (size_t)p] = (s << NDKidBit) | k;
                        }
                    }
                  for (size_t e = m0; e < maps.size(); ++e)
                    if (maps[e] < 0)
                      return bad(err, "nested dissection: a front dof belongs to no child");
                  for (int i = 0; i < nF; ++i)
                    pos[d[i]] = -1;
                }
            }
          n.map = it->second;
        }
      tree.clear();
      tree.shrink_to_fit();
      return DDHDG_OK;
    }
  };

  struct NDSolver::Device
  {
    std::vector<void *>  allocs;
    double              *fronts = nullptr, *ecols = nullptr, *luf = nullptr, *tinv = nullptr, *dscale = nullptr,
                        *work   = nullptr;
    NDNode              *nodes  = nullptr;
    int32_t             *fdofs = nullptr, *maps = nullptr, *perm = nullptr, *ul[2] = {nullptr, nullptr};
    int                 *sing = nullptr, *ipiv = nullptr;
    int64_t             *cell_faces = nullptr;
    unsigned long long  *dmax       = nullptr;
    int64_t              work_n     = 0;
    ~Device()
    {
      for (void *p : allocs)
        cudaFree(p);
    }
    template <typename T>
    int
    alloc(T *&p, int64_t count, std::string &err)
    {
      const size_t bytes = std::max<size_t>((size_t)count * sizeof(T), 16);
      if (cudaMalloc(reinterpret_cast<void **>(&p), bytes) != cudaSuccess)
        {
          cudaGetLastError();
          p   = nullptr;
          err = "cudaMalloc of " + std::to_string(bytes) + " bytes for the trace solver failed";
          return DDHDG_OOM;
        }
      allocs.push_back(p);
      return DDHDG_OK;
    }
    template <typename T>
    int
    upload(T *&p, const std::vector<T> &v, std::string &err)
    {
      int r = alloc(p, (int64_t)v.size(), err);
      if (r)
        return r;
      if (!v.empty() && cudaMemcpy(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice) != cudaSuccess)
        return bad(err, "upload failed", DDHDG_CUDA_ERROR);
      return DDHDG_OK;
    }
  };

  NDSolver::NDSolver() = default;
  NDSolver::~NDSolver() { release(); }

  void
  NDSolver::release()
  {
    if (exec_)
      cudaGraphExecDestroy(exec_);
    exec_ = nullptr;
    dev_.reset();
    if (dn_)
      cusolverDnDestroy(dn_);
    dn_ = nullptr;
    if (cap_)
      cudaStreamDestroy(cap_);
    cap_       = nullptr;
    key_       = Key{};
    graphs_ok_ = true;
    built_     = false;
    plan_.reset();
  }

  int
  NDSolver::plan(const Mesh &M, std::string &err)
  {
    static std::mutex                               mu;
    static std::vector<std::shared_ptr<const Plan>> cache;
    release();
    const auto same = [](const Mesh &a, const Mesh &b) {
      bool eq = a.dim == b.dim && a.ncells == b.ncells && a.nfaces == b.nfaces && a.F == b.F && a.nd == b.nd;
      for (int i = 0; i < 3; ++i)
        {
          eq = eq && a.n[i] == b.n[i] && a.face_off[i] == b.face_off[i];
          for (int j = 0; j < 3; ++j)
            eq = eq && a.face_ext[i][j] == b.face_ext[i][j];
        }
      return eq;
    };
    {
      std::lock_guard<std::mutex> lock(mu);
      for (auto &e : cache)
        if (same(e->M, M))
          {
            plan_ = e;
            return DDHDG_OK;
          }
    }
    auto      p = std::make_shared<Plan>();
    const int r = p->make(M, err);
    if (r)
      return r;
    plan_ = p;
    std::lock_guard<std::mutex> lock(mu);
    cache.insert(cache.begin(), plan_);
    // at most 32 plans (two modes of 16 requests in flight), and no more
    // than 4 GB of host copies
    size_t bytes = 0, keep = 0;
    for (; keep < cache.size() && keep < 32; ++keep)
      {
        bytes += cache[keep]->bytes();
        if (bytes > ((size_t)4 << 30) && keep > 0)
          break;
      }
    cache.resize(keep);
    return DDHDG_OK;
  }

  int64_t
  NDSolver::planned_device_bytes() const
  {
    const Plan   &P = *plan_;
    const int64_t g = (int64_t)2 << 20;
    int64_t       b = 0;
    auto          add = [&](int64_t bytes) { b += (std::max<int64_t>(bytes, 16) + g - 1) / g * g; };
    add(P.front_total * 8);
    add(P.e_total * 8);
    add(P.lu_total * 8);
    add(P.ti_total * 8);
    for (int q = 0; q < 3; ++q)
      add(P.p_total * 4);
    add((int64_t)P.nodes.size() * (int64_t)sizeof(NDNode));
    add((int64_t)P.fdofs.size() * 4);
    add((int64_t)P.maps.size() * 4);
    add((int64_t)P.cell_faces.size() * 8);
    const int64_t ndofs = P.M.nfaces * (int64_t)P.M.nd;
    add(ndofs * 8);
    add(ndofs * 8);
    add(16);
    if (P.lib_nE)
      {
        // a bound of the library LU's workspace, its pivots, and its handle
        // (measured on CUDA 12.9: about 300 MB)
        add((int64_t)64 * P.lib_nE * 8);
        add((int64_t)P.lib_nE * 4);
        b += (int64_t)320 << 20;
      }
    return b;
  }

  int
  NDSolver::build(const Mesh &M, std::string &err)
  {
    int r;
    if ((r = plan(M, err)))
      return r;
    const Plan &P = *plan_;
    dev_.reset(new Device);
    Device       &D     = *dev_;
    const int64_t ndofs = M.nfaces * (int64_t)M.nd;
    if ((r = D.alloc(D.fronts, P.front_total, err)) || (r = D.alloc(D.ecols, P.e_total, err)) ||
        (r = D.alloc(D.luf, P.lu_total, err)) || (r = D.alloc(D.tinv, P.ti_total, err)) ||
        (r = D.alloc(D.perm, P.p_total, err)) || (r = D.alloc(D.ul[0], P.p_total, err)) ||
        (r = D.alloc(D.ul[1], P.p_total, err)) || (r = D.upload(D.nodes, P.nodes, err)) ||
        (r = D.upload(D.fdofs, P.fdofs, err)) || (r = D.upload(D.maps, P.maps, err)) ||
        (r = D.upload(D.cell_faces, P.cell_faces, err)) || (r = D.alloc(D.dmax, ndofs, err)) ||
        (r = D.alloc(D.dscale, ndofs, err)) || (r = D.alloc(D.sing, 2, err)))
      return r;
    if (P.lib_nE)
      {
        if (cusolverDnCreate(&dn_) != CUSOLVER_STATUS_SUCCESS)
          return bad(err, "cusolverDnCreate failed", DDHDG_SOLVER_ERROR);
        for (const auto &n : P.nodes)
          if (n.nE > PanelRows)
            {
              int lw = 0;
              if (cusolverDnDgetrf_bufferSize(dn_, n.nE, n.nE, D.ecols, n.ld, &lw) != CUSOLVER_STATUS_SUCCESS)
                return bad(err, "cusolverDnDgetrf_bufferSize failed", DDHDG_SOLVER_ERROR);
              D.work_n = std::max<int64_t>(D.work_n, lw);
            }
        if ((r = D.alloc(D.work, D.work_n, err)) || (r = D.alloc(D.ipiv, P.lib_nE, err)))
          return r;
      }
    if (cudaStreamCreateWithFlags(&cap_, cudaStreamNonBlocking) != cudaSuccess)
      return bad(err, "cudaStreamCreate failed", DDHDG_CUDA_ERROR);
    const void *fns[] = {(const void *)nd_small_kernel<4, false>,  (const void *)nd_small_kernel<12, false>,
                         (const void *)nd_small_kernel<20, false>, (const void *)nd_small_kernel<28, false>,
                         (const void *)nd_small_kernel<36, false>, (const void *)nd_small_kernel<4, true>,
                         (const void *)nd_small_kernel<12, true>,  (const void *)nd_small_kernel<20, true>,
                         (const void *)nd_small_kernel<28, true>,  (const void *)nd_small_kernel<36, true>,
                         (const void *)nd_gather_b_kernel,         (const void *)nd_update_kernel,
                         (const void *)nd_solve_kernel<32>,        (const void *)nd_solve_kernel<64>,
                         (const void *)nd_root_solve_kernel,       (const void *)nd_gemm_kernel<true>,
                         (const void *)nd_gemm_kernel<false>,      (const void *)nd_backsolve_kernel};
    for (const void *f : fns)
      if (allow_full_dynamic_smem(f) != cudaSuccess)
        return bad(err, "cannot raise the shared-memory limit of the trace-solve kernels", DDHDG_CUDA_ERROR);
    built_ = true;
    return DDHDG_OK;
  }

  void
  NDSolver::set_graphs(bool on)
  {
    use_graphs_ = on;
    if (!on && exec_)
      {
        cudaGraphExecDestroy(exec_);
        exec_ = nullptr;
      }
  }

  int
  NDSolver::solve(const double *tt, const double *rhs, const int32_t *dflag, const double *dval, int Nt, double *x,
                  cudaStream_t s, int sm_count, std::string &err, bool check)
  {
    if (!built_)
      return bad(err, "nested-dissection solver not built");
    if (Nt != plan_->M.F * plan_->M.nd)
      return bad(err, "trace block size does not match the solver");
    const Key k{tt, rhs, dflag, dval, x, sm_count};
    int       r = DDHDG_OK;
    if (use_graphs_ && graphs_ok_ && exec_ && k == key_)
      {
        if (cudaGraphLaunch(exec_, s) != cudaSuccess)
          return bad(err, "cudaGraphLaunch failed", DDHDG_CUDA_ERROR);
      }
    else if (use_graphs_ && graphs_ok_ && k == key_ && !exec_)
      {
        // same buffers as the last (eager) call: capture, then launch
        cudaGraph_t gph = nullptr;
        if (cudaStreamBeginCapture(cap_, cudaStreamCaptureModeThreadLocal) != cudaSuccess)
          {
            cudaGetLastError();
            graphs_ok_ = false;
            r          = enqueue(tt, rhs, dflag, dval, Nt, x, s, sm_count, err);
          }
        else
          {
            const int         rc = enqueue(tt, rhs, dflag, dval, Nt, x, cap_, sm_count, err);
            const cudaError_t e  = cudaStreamEndCapture(cap_, &gph);
            if (rc || e != cudaSuccess || !gph || cudaGraphInstantiate(&exec_, gph, 0) != cudaSuccess)
              {
                cudaGetLastError();
                exec_      = nullptr;
                graphs_ok_ = false; // this build cannot capture: stay eager
                r          = enqueue(tt, rhs, dflag, dval, Nt, x, s, sm_count, err);
              }
            else if (cudaGraphLaunch(exec_, s) != cudaSuccess)
              r = bad(err, "cudaGraphLaunch failed", DDHDG_CUDA_ERROR);
            if (gph)
              cudaGraphDestroy(gph);
          }
      }
    else
      {
        if (exec_)
          cudaGraphExecDestroy(exec_);
        exec_ = nullptr;
        key_  = k;
        r     = enqueue(tt, rhs, dflag, dval, Nt, x, s, sm_count, err);
      }
    if (r)
      return r;
    return check ? check_info(s, err) : DDHDG_OK;
  }

  int
  NDSolver::check_info(cudaStream_t s, std::string &err)
  {
    int sing = 0;
    if (cudaMemcpyAsync(&sing, dev_->sing, sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess)
      return bad(err, "nested-dissection solve failed", DDHDG_CUDA_ERROR);
    if (sing)
      return bad(err, "global trace matrix is singular (zero pivot in a front)", DDHDG_SOLVER_ERROR);
    return DDHDG_OK;
  }

  namespace
  {
    template <int NEM>
    void
    launch_small(const Batch &b, const NDNode *nodes, const int32_t *maps, const NDCells &C, int *sing, double *fronts,
                 cudaStream_t s)
    {
      const size_t smem = nd_small_smem(NEM, b.maxK);
      // one or two warps factorise, the others stage; a thread per column
      // solves for W; 16 warps where one CTA fills the SM's shared memory
      const int T = NEM > 28 && smem > 110 * 1024 ? 512 : b.maxK + 1 > 128 ? 256 : 128;
      if (b.leaf)
        nd_small_kernel<NEM, true><<<b.count, T, smem, s>>>(nodes, maps, C, b.maxK, sing, fronts);
      else
        nd_small_kernel<NEM, false><<<b.count, T, smem, s>>>(nodes, maps, C, b.maxK, sing, fronts);
    }

    template <int CL>
    cudaError_t
    launch_panel(int count, int T, const NDNode *nodes, int k0, const int32_t *ul_in, int32_t *ul_out, double *ecols,
                 double *luf, int32_t *perm, double *tinv, int *sing, cudaStream_t s)
    {
      cudaLaunchConfig_t    cfg = {};
      cudaLaunchAttribute   at[1];
      cfg.gridDim               = dim3((unsigned)count * CL);
      cfg.blockDim              = dim3(T);
      cfg.stream                = s;
      at[0].id                  = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x    = CL;
      at[0].val.clusterDim.y    = 1;
      at[0].val.clusterDim.z    = 1;
      cfg.attrs                 = at;
      cfg.numAttrs              = CL > 1 ? 1 : 0;
      return cudaLaunchKernelEx(&cfg, nd_panel_kernel<CL>, nodes, k0, ul_in, ul_out, ecols, luf, perm, tinv, sing);
    }
  } // namespace

  // the numeric phase's launches on stream s (no host synchronisation)
  int
  NDSolver::enqueue(const double *tt, const double *rhs, const int32_t *dflag, const double *dval, int Nt, double *x,
                    cudaStream_t s, int sm_count, std::string &err)
  {
    const Plan   &P     = *plan_;
    Device       &D     = *dev_;
    const Mesh   &M     = P.M;
    const int64_t ndofs = M.nfaces * (int64_t)M.nd;
    const int     grid  = sm_count * 8;
    const NDCells C{tt, rhs, dval, D.dscale, dflag, D.cell_faces, Nt, M.nd, M.F};
    // row equilibration
    if (cudaMemsetAsync(D.dmax, 0, ndofs * sizeof(unsigned long long), s) != cudaSuccess ||
        cudaMemsetAsync(D.sing, 0, 2 * sizeof(int), s) != cudaSuccess)
      return bad(err, "memset failed", DDHDG_CUDA_ERROR);
    nd_rowmax_kernel<<<grid, 256, 0, s>>>(M.ncells, C, D.dmax);
    nd_rowscale_kernel<<<grid, 256, 0, s>>>(ndofs, D.dmax, D.dscale);
    // upward pass
    for (const auto &b : P.batches)
      {
        const NDNode *nodes = D.nodes + b.node0;
        switch (b.cls)
          {
            case Small4:
              launch_small<4>(b, nodes, D.maps, C, D.sing, D.fronts, s);
              continue;
            case Small12:
              launch_small<12>(b, nodes, D.maps, C, D.sing, D.fronts, s);
              continue;
            case Small20:
              launch_small<20>(b, nodes, D.maps, C, D.sing, D.fronts, s);
              continue;
            case Small28:
              launch_small<28>(b, nodes, D.maps, C, D.sing, D.fronts, s);
              continue;
            case Small36:
              launch_small<36>(b, nodes, D.maps, C, D.sing, D.fronts, s);
              continue;
            default:
              break;
          }
        const auto ceil_div = [](int a, int c) { return (a + c - 1) / c; };
        const int  nb       = b.count;
        // E columns: about 4 CTAs per SM over the batch
        {
          const int gx = std::max(1, std::min(b.maxE, ceil_div(sm_count * 8, nb)));
          nd_gather_e_kernel<<<dim3(gx, nb), 256, 0, s>>>(nodes, D.maps, C, D.fronts, D.ecols);
        }
        if (b.cls == Panels)
          {
            for (int k0 = 0, par = 0; k0 < b.maxE; k0 += NDPanel, par ^= 1)
              {
                const int      m = b.maxE - k0;
                const int32_t *in  = D.ul[par];
                int32_t       *out = D.ul[par ^ 1];
                cudaError_t    e;
                const int      T = m <= 128 ? 128 : m <= 256 ? 256 : NDPanelT;
                if (m <= NDPanelT)
                  e = launch_panel<1>(nb, T, nodes, k0, in, out, D.ecols, D.luf, D.perm, D.tinv, D.sing, s);
                else if (m <= 2 * NDPanelT)
                  e = launch_panel<2>(nb, T, nodes, k0, in, out, D.ecols, D.luf, D.perm, D.tinv, D.sing, s);
                else if (m <= 4 * NDPanelT)
                  e = launch_panel<4>(nb, T, nodes, k0, in, out, D.ecols, D.luf, D.perm, D.tinv, D.sing, s);
                else
                  e = launch_panel<8>(nb, T, nodes, k0, in, out, D.ecols, D.luf, D.perm, D.tinv, D.sing, s);
                if (e != cudaSuccess)
                  return bad(err, "panel launch failed", DDHDG_CUDA_ERROR);
                if (m > NDPanel)
                  {
                    const int ct = ceil_div(m - NDPanel, NDUpd);
                    nd_update_kernel<<<dim3(ct * ct, nb), 128, nd_update_smem(), s>>>(nodes, k0, ct, out, D.ecols,
                                                                                     D.luf, D.perm, D.tinv);
                  }
              }
            if (b.maxE > NDPanel)
              {
                const int gx = std::max(1, std::min((b.maxE - 1) / NDPanel * NDPanel, ceil_div(sm_count * 8, nb)));
                nd_lu_finish_kernel<<<dim3(gx, nb), 256, 0, s>>>(nodes, D.ecols, D.perm, D.luf);
              }
          }
        else
          {
            cusolverDnSetStream(dn_, s);
            for (int q = 0; q < nb; ++q)
              {
                const NDNode &n = P.nodes[b.node0 + q];
                if (cusolverDnDgetrf(dn_, n.nE, n.nE, D.ecols + n.eoff, n.ld, D.work, D.ipiv, D.sing + 1) !=
                    CUSOLVER_STATUS_SUCCESS)
                  return bad(err, "cusolverDnDgetrf failed", DDHDG_SOLVER_ERROR);
                nd_lib_perm_kernel<<<1, 256, 0, s>>>(nodes + q, D.ipiv, D.sing + 1, D.perm, D.sing);
                nd_lib_copy_kernel<<<grid, 256, 0, s>>>(nodes + q, D.ecols, D.luf);
                nd_lib_inverse_kernel<<<ceil_div(n.nE, NDPanel), 64, 0, s>>>(nodes + q, D.luf, D.tinv);
              }
          }
        // W = U^-1 L^-1 P [F_EK | r_E]
        {
          const int cb = std::max(1, std::min(16, 2048 / b.maxE));
          nd_gather_b_kernel<<<dim3(ceil_div(b.maxK + 1, cb), nb), 256, (size_t)cb * b.maxE * sizeof(double), s>>>(
            nodes, D.maps, C, D.perm, cb, D.fronts);
        }
        if (b.maxK == 0 && b.maxE <= RootRows)
          nd_root_solve_kernel<<<nb, NDRootT, (size_t)ceil_div(b.maxE, NDPanel) * NDPanel * sizeof(double), s>>>(
            nodes, D.luf, D.tinv, D.fronts);
        else
          {
            const bool wide  = (int64_t)ceil_div(b.maxK + 1, 64) * nb >= sm_count;
            const int  CT    = wide ? 64 : 32, cols = ceil_div(b.maxK + 1, CT);
            const auto sweep = [&](int b0, int bs, int dir) {
              if (wide)
                nd_solve_kernel<64><<<dim3(cols, nb), 256, nd_solve_smem(64, bs), s>>>(nodes, b0, bs, dir, D.luf,
                                                                                      D.tinv, D.fronts);
              else
                nd_solve_kernel<32><<<dim3(cols, nb), 256, nd_solve_smem(32, bs), s>>>(nodes, b0, bs, dir, D.luf,
                                                                                      D.tinv, D.fronts);
            };
            // blocked: block rows whose column tiles fit in shared memory, the
            // rest of the rows updated by products
            const int nblk = ceil_div(b.maxE, nd_solve_rows(CT));
            const int bs   = ceil_div(ceil_div(b.maxE, nblk), NDPanel) * NDPanel;
            const int tn   = ceil_div(b.maxK + 1, NDGN);
            if (nblk == 1)
              sweep(0, bs, 3);
            else
              for (int dir = 1; dir <= 2; ++dir)
                for (int i = 0; i < nblk; ++i)
                  {
                    const int b0 = (dir == 1 ? i : nblk - 1 - i) * bs;
                    sweep(b0, bs, dir);
                    const int r0 = dir == 1 ? b0 + bs : 0, mr = dir == 1 ? b.maxE - r0 : b0;
                    if (mr > 0)
                      {
                        const int tm = ceil_div(mr, NDGM);
                        nd_gemm_kernel<false><<<dim3(tm * tn, nb), 128, nd_gemm_smem(), s>>>(
                          nodes, D.maps, C, tm, r0, mr, b0, bs, D.ecols, D.luf, D.fronts);
                      }
                  }
          }
        if (b.maxK > 0)
          {
            const int tm = ceil_div(b.maxK, NDGM), tn = ceil_div(b.maxK + 1, NDGN);
            nd_gemm_kernel<true><<<dim3(tm * tn, nb), 128, nd_gemm_smem(), s>>>(nodes, D.maps, C, tm, 0, 0, 0, 0,
                                                                               D.ecols, D.luf, D.fronts);
          }
      }
    // downward pass: R rows per CTA, S slices of the kept dofs, about 8 or
    // more terms per thread
    for (auto it = P.batches.rbegin(); it != P.batches.rend(); ++it)
      {
        const Batch &b = *it;
        const int    R = b.maxE < 32 ? b.maxE : 32;
        const int    S = std::max(1, std::min((b.maxK + 7) / 8, 1024 / R));
        nd_backsolve_kernel<<<dim3(b.count, (b.maxE + R - 1) / R), R * S,
                              (size_t)(b.maxK + R * S) * sizeof(double), s>>>(R, D.nodes + b.node0, D.fdofs,
                                                                             D.fronts, x);
      }
    if (cudaGetLastError() != cudaSuccess)
      return bad(err, "nested-dissection kernel launch failed", DDHDG_CUDA_ERROR);
    return DDHDG_OK;
  }
} // namespace ddhdg
