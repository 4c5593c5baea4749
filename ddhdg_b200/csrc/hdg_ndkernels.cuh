// Device kernels of the nested-dissection trace solve (sm_100a, FP64); the
// tree, the batches and the launch sequence are in hdg_ndsolve.cu.
//
// A tree node eliminates its nE dofs (E) against its nK kept dofs (K).  What
// stays of a front in memory is its K columns and the right-hand-side
// column, [E rows | K rows] x (nK + 1), column-major with leading dimension
// ld: W = F_EE^-1 [F_EK | r_E] in the E rows and the Schur complement
// F_KK - F_KE W in the K rows.  The E columns live in scratch while the
// node's batch is eliminated.  Every front entry is the sum of at most two
// entries of the children's Schur complements, read through the maps of the
// node's shape where it is needed (no zeroed front, no extend-add pass):
// an E face touches both children, a K face exactly one.  Children that are
// interior cells are read directly from the condensed blocks.
#pragma once

#include <cooperative_groups.h>
#include <cstdint>
#include <cuda_runtime.h>

#include "hdg_mma.cuh"
#include "hdg_reciprocal.cuh"

namespace ddhdg
{
  struct NDNode
  {
    int64_t koff;     // K columns of the front (doubles)
    int64_t eoff;     // E columns in the batch's scratch
    int64_t luoff;    // LU factors in the batch's scratch
    int64_t tioff;    // inverted diagonal blocks in the batch's scratch
    int64_t coff[2];  // the children's K columns
    int64_t ccell[2]; // cell of a child read from the condensed blocks, or -1
    int64_t cell;     // the node's cell (leaf), or -1
    int64_t doff;     // dof list [E, K]
    int64_t poff;     // pivot order and row lists in the batch's scratch
    int32_t map;      // maps of the node's shape
    int32_t nE, nK;
    int32_t nEp; // nE rounded up to even: first K row
    int32_t ld;  // nEp + nK rounded up to even
    int32_t cEp[2], cld[2], cnK[2];
  };

  // the condensed per-cell blocks and the row scaling
  struct NDCells
  {
    const double  *tt, *rhs, *dval, *dscale;
    const int32_t *dflag;
    const int64_t *cell_faces;
    int            Nt, nd, F;
  };

  constexpr int NDKidBit = 30; // maps of the K rows: child << 30 | kept index

  // rows of the trace matrix: max |tt[a][:]| per global dof (bit pattern of a
  // non-negative double, so that an integer max is the double max)
  __global__ void
  nd_rowmax_kernel(int64_t ncells, NDCells C, unsigned long long *dmax)
  {
    const int64_t tot = ncells * C.Nt;
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < tot;
         idx += (int64_t)gridDim.x * blockDim.x)
      {
        const int64_t cell = idx / C.Nt;
        const int     a    = (int)(idx % C.Nt);
        const double *row  = C.tt + (cell * C.Nt + a) * (int64_t)C.Nt;
        double        m    = 0.;
        for (int b = 0; b < C.Nt; ++b)
          m = fmax(m, fabs(row[b]));
        const int64_t g = C.cell_faces[cell * C.F + a / C.nd] * C.nd + a % C.nd;
        atomicMax(dmax + g, (unsigned long long)__double_as_longlong(m));
      }
  }

  __global__ void
  nd_rowscale_kernel(int64_t n, const unsigned long long *dmax, double *dscale)
  {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
      {
        const double m = __longlong_as_double((long long)dmax[i]);
        dscale[i]      = (m > 0.) ? 1. / m : 1.;
      }
  }

  __device__ __forceinline__ double
  nd_cell_scale(const NDCells &C, int64_t cell, int a)
  {
    return C.dscale[C.cell_faces[cell * C.F + a / C.nd] * C.nd + a % C.nd];
  }

  // entry (row a, column b) of a cell's block: scaled, Dirichlet rows identity
  __device__ __forceinline__ double
  nd_cell_entry(const NDCells &C, int64_t cell, int a, int b)
  {
    if (C.dflag[cell * C.Nt + a])
      return a == b ? 1. : 0.;
    return C.tt[(cell * C.Nt + a) * (int64_t)C.Nt + b] * nd_cell_scale(C, cell, a);
  }

  __device__ __forceinline__ double
  nd_cell_rhs(const NDCells &C, int64_t cell, int a)
  {
    const int64_t i = cell * C.Nt + a;
    return C.dflag[i] ? C.dval[i] : C.rhs[i] * nd_cell_scale(C, cell, a);
  }

  // entry (kept row jr, kept column jc) of child s
  __device__ __forceinline__ double
  nd_kid(const NDNode &n, const double *fronts, int s, int jr, int jc)
  {
    // selects, not indices: the node stays out of local memory
    return fronts[(s ? n.coff[1] : n.coff[0]) + (int64_t)jc * (s ? n.cld[1] : n.cld[0]) +
                  (s ? n.cEp[1] : n.cEp[0]) + jr];
  }

  // Front entries by position: rows and columns 0..nE-1 are E, column nK of
  // the K columns is the right-hand side.  Used by the kernels of the larger
  // fronts, whose children always keep their own fronts in memory.
  struct NDFront
  {
    const NDNode  &n;
    const NDCells &C;
    const int32_t *map;
    const double  *fronts;
    __device__ __forceinline__ double
    EE(int i, int j) const
    {
      if (n.cell >= 0)
        return nd_cell_entry(C, n.cell, map[i], map[j]);
      return nd_kid(n, fronts, 0, map[i], map[j]) + nd_kid(n, fronts, 1, map[n.nE + i], map[n.nE + j]);
    }
    __device__ __forceinline__ double
    KE(int r, int j) const
    {
      if (n.cell >= 0)
        return nd_cell_entry(C, n.cell, map[n.nE + r], map[j]);
      const int k = map[2 * n.nE + r], s = k >> NDKidBit;
      return nd_kid(n, fronts, s, k & ((1 << NDKidBit) - 1), map[s * n.nE + j]);
    }
    __device__ __forceinline__ double
    EK(int i, int c) const // c == nK: the right-hand side
    {
      if (n.cell >= 0)
        return c == n.nK ? nd_cell_rhs(C, n.cell, map[i]) : nd_cell_entry(C, n.cell, map[i], map[n.nE + c]);
      if (c == n.nK)
        return nd_kid(n, fronts, 0, map[i], n.cnK[0]) + nd_kid(n, fronts, 1, map[n.nE + i], n.cnK[1]);
      const int k = map[2 * n.nE + c], s = k >> NDKidBit;
      return nd_kid(n, fronts, s, map[s * n.nE + i], k & ((1 << NDKidBit) - 1));
    }
    __device__ __forceinline__ double
    KK(int r, int c) const
    {
      if (n.cell >= 0)
        return c == n.nK ? nd_cell_rhs(C, n.cell, map[n.nE + r]) :
                           nd_cell_entry(C, n.cell, map[n.nE + r], map[n.nE + c]);
      const int kr = map[2 * n.nE + r], sr = kr >> NDKidBit, jr = kr & ((1 << NDKidBit) - 1);
      if (c == n.nK)
        return nd_kid(n, fronts, sr, jr, sr ? n.cnK[1] : n.cnK[0]);
      const int kc = map[2 * n.nE + c];
      return (kc >> NDKidBit) == sr ? nd_kid(n, fronts, sr, jr, kc & ((1 << NDKidBit) - 1)) : 0.;
    }
  };

  // 32-bit pivot key of a candidate: the high word of |x| (sign, exponent,
  // 20 mantissa bits) plus one, so that 0 marks rows that cannot be chosen;
  // the pivot is within 2^-20 of the largest candidate, ties go to the first
  __device__ __forceinline__ unsigned
  nd_pivot_key(double x)
  {
    return (unsigned)((unsigned long long)__double_as_longlong(fabs(x)) >> 32) + 1u;
  }

  // barrier of a whole cluster, for warps that need not be converged
  __device__ __forceinline__ void
  nd_cluster_sync()
  {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
  }

  // ------------------------------------------------------------ small fronts
  // nE <= NEM <= 36: the whole elimination of a front in one CTA.
  // - F_EE goes into the registers of one warp (two for NEM > 32), a row per
  //   lane: LU with virtual partial pivoting, the pivot search one warp
  //   max-reduction, the pivot row broadcast through shared memory; the other
  //   warps stage [F_EK | r_E] and -F_KE.
  // - W: a thread per column, its nE entries in registers, the factors
  //   broadcast from shared memory; no barrier between its steps.
  // - F_KK - F_KE W: 16 x 32 warp tiles on the FP64 tensor path with the
  //   children's entries as the initial accumulators, stored once.
  // Bound by memory (the children's Schur complements in, W and the own one
  // out) and, per front, by the nE dependent pivot steps; several CTAs per
  // SM overlap the two.
  __host__ __device__ constexpr int
  nd_small_class(int nE)
  {
    return nE <= 4 ? 4 : nE <= 12 ? 12 : nE <= 20 ? 20 : nE <= 28 ? 28 : 36;
  }

  constexpr int NDSmallE = 36;

  __host__ __device__ inline size_t
  nd_small_smem(int NEM, int nK)
  {
    // rows of Bs / Ks hold NEM doubles: NEM = 4 or 12 (mod 16), so the
    // tensor-path fragments read distinct banks
    return ((size_t)NEM * NEM + NEM + (size_t)(2 * nK + 1) * NEM + 2 * (size_t)nK + 4 * NEM) * sizeof(double) +
           ((size_t)nK * 2 + 4 * NEM) * sizeof(int);
  }

  template <int NEM, bool LEAF>
  __global__ void __launch_bounds__(NEM > 28 ? 512 : 256, NEM <= 12 ? 4 : NEM <= 20 ? 3 : NEM <= 28 ? 2 : 1)
  nd_small_kernel(const NDNode *nodes, const int32_t *maps, NDCells C, int nKmax, int *sing, double *fronts)
  {
    extern __shared__ __align__(16) double sm[];
    constexpr int LDW = NEM;
    constexpr int NLW = NEM > 32 ? 2 : 1; // warps of the LU, a row per lane
    __shared__ __align__(16) double prow_s[2][NLW][NEM];
    __shared__ double   phr_s[2][NLW];
    __shared__ unsigned pkey_s[2][NLW];
    __shared__ int      pid_s[2][NLW];
    const NDNode  n   = nodes[blockIdx.x];
    const int     nE = n.nE, nK = n.nK;
    double       *LU   = sm;                     // factors, [column][pivot order]
    double       *dinv = LU + NEM * NEM;         // 1 / U_jj
    double       *Bs   = dinv + NEM;             // [column of K, r][E row]
    double       *Ks   = Bs + (nKmax + 1) * LDW; // -F_KE: [K row][E column]
    // Every position of the front as a row and as a column of the child (or
    // cell) that holds it: an entry is rs * rp[column offset].  A K position
    // belongs to one child, an E position to both.
    double        *krs  = Ks + nKmax * LDW;                    // row scale
    double        *ers  = krs + nKmax;                         // [2][NEM]
    const double **krp  = (const double **)(ers + 2 * NEM);    // row pointer
    const double **erp  = krp + nKmax;                         // [2][NEM]
    int           *kco  = reinterpret_cast<int *>(erp + 2 * NEM); // column offset
    int           *kid  = kco + nKmax;                         // child of a K position
    int           *eco  = kid + nKmax;                         // [2][NEM]
    int           *perm = eco + 2 * NEM;
    const int      tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, T = blockDim.x;
    const int32_t *map = maps + n.map;
    constexpr int  KM  = (1 << NDKidBit) - 1;
    // row jr, column offset jc of child s; raw cells carry the row scaling,
    // their Dirichlet rows are identity rows, marked by the scale -1 (a scale
    // is never negative; it is 0 for a row that holds an infinity)
    const auto place = [&](int s, int j, const double *&rp, double &rs, int &co) {
      const int64_t cell = LEAF ? n.cell : (s ? n.ccell[1] : n.ccell[0]);
      if (cell >= 0)
        {
          rp = C.tt + (cell * C.Nt + j) * (int64_t)C.Nt;
          rs = C.dflag[cell * C.Nt + j] ? -1. : nd_cell_scale(C, cell, j);
          co = j;
        }
      else
        {
          rp = fronts + (s ? n.coff[1] : n.coff[0]) + (s ? n.cEp[1] : n.cEp[0]) + j;
          rs = 1.;
          co = j * (s ? n.cld[1] : n.cld[0]);
        }
    };
    for (int i = tid; i < nE; i += T)
#pragma unroll
      for (int s = 0; s < (LEAF ? 1 : 2); ++s)
        place(s, map[LEAF ? i : s * nE + i], erp[s * NEM + i], ers[s * NEM + i], eco[s * NEM + i]);
    for (int i = tid; i < nK; i += T)
      {
        const int k = LEAF ? map[nE + i] : map[2 * nE + i], s = LEAF ? 0 : k >> NDKidBit;
        place(s, k & KM, krp[i], krs[i], kco[i]);
        kid[i] = s;
      }
    const bool cells = LEAF || n.ccell[0] >= 0 || n.ccell[1] >= 0;
    __syncthreads();
    // value of an entry from what its place holds: row scale, column offsets
    // of the row's own position and of the entry
    const auto entry = [&](double x, double rs, int own, int co) -> double {
      if (cells && rs < 0.)
        return own == co ? 1. : 0.;
      return rs * x;
    };
    // place of the right-hand side of a row of child s (Dirichlet rows: their
    // value, unscaled)
    const auto rhs_at = [&](int s, const double *rp, double rs, int own) -> const double * {
      const int64_t cell = LEAF ? n.cell : (s ? n.ccell[1] : n.ccell[0]);
      if (cell >= 0)
        return (rs < 0. ? C.dval : C.rhs) + cell * C.Nt + own;
      return rp + (int64_t)(s ? n.cnK[1] : n.cnK[0]) * (s ? n.cld[1] : n.cld[0]);
    };
    const auto rhs_scale = [&](double rs) { return cells && rs < 0. ? 1. : rs; };
    for (int idx = tid; idx < NEM * NEM; idx += T)
      {
        const int i = idx % NEM, c = idx / NEM;
        double    x = (i == c) ? 1. : 0.;
        if (i < nE && c < nE)
          {
            x = entry(erp[i][eco[c]], ers[i], eco[i], eco[c]);
            if (!LEAF)
              x += entry(erp[NEM + i][eco[NEM + c]], ers[NEM + i], eco[NEM + i], eco[NEM + c]);
          }
        LU[idx] = x;
      }
    __syncthreads();
    if (warp < NLW)
      {
        // rolled steps (the instruction cache holds the body): the row is
        // rotated by one register per step, the current column in v[0]
        double v[NEM];
#pragma unroll
        for (int c = 0; c < NEM; ++c)
          v[c] = LU[c * NEM + min(tid, NEM - 1)];
        bool used = tid >= nE, bad = false;
        int  pos  = -1;
#pragma unroll 1
        for (int j = 0; j < nE; ++j)
          {
            const int      buf  = j & 1;
            const double   x0   = v[0];
            const unsigned key  = used ? 0u : nd_pivot_key(x0);
            const double   hx   = reciprocal_normal(x0); // overlaps the reduction
            const unsigned kmax = __reduce_max_sync(0xffffffffu, key);
            const int      src  = __ffs(__ballot_sync(0xffffffffu, key == kmax)) - 1;
            if (lane == src)
              {
                // finished columns, at the end, are published as zeros
                double2 *dst = reinterpret_cast<double2 *>(prow_s[buf][warp]);
#pragma unroll
                for (int k = 0; k < NEM; k += 2)
                  dst[k / 2] = make_double2(k < NEM - j ? v[k] : 0., k + 1 < NEM - j ? v[k + 1] : 0.);
                phr_s[buf][warp]  = reciprocal(x0, hx);
                pkey_s[buf][warp] = kmax;
                pid_s[buf][warp]  = tid;
              }
            if (NLW > 1)
              asm volatile("barrier.sync 1, 64;" ::: "memory");
            else
              __syncwarp();
            const int     ww   = (NLW > 1 && pkey_s[buf][NLW - 1] > pkey_s[buf][0]) ? NLW - 1 : 0;
            const double *prow = prow_s[buf][ww];
            const double  hr   = phr_s[buf][ww];
            const int     pid  = pid_s[buf][ww];
            const bool    me   = tid == pid;
            const double  l    = (used || me) ? 0. : x0 * hr;
#pragma unroll
            for (int k = 1; k < NEM; ++k)
              v[k - 1] = v[k] - l * prow[k];
            v[NEM - 1] = (used || me) ? x0 : l;
            if (me)
              {
                used    = true;
                pos     = j;
                dinv[j] = hr;
                perm[j] = tid;
                bad |= hr == 0. || isnan(hr); // zero or non-finite pivot
              }
          }
#pragma unroll 1
        for (int j = nE; j < NEM; ++j)
          {
            // the unit rows and columns beyond nE keep their places
            const double x0 = v[0];
#pragma unroll
            for (int k = 1; k < NEM; ++k)
              v[k - 1] = v[k];
            v[NEM - 1] = x0;
            if (tid == 0)
              {
                dinv[j] = 1.;
                perm[j] = j;
              }
          }
        if (pos >= 0)
          {
#pragma unroll
            for (int c = 0; c < NEM; ++c)
              LU[c * NEM + pos] = v[c];
          }
        if (bad)
          atomicExch(sing, 1);
      }
    else
      {
        const int t0 = tid - 32 * NLW, TT = T - 32 * NLW;
        // GU entries in flight per thread: their loads are unconditional, so
        // that they do not wait for each other
        constexpr int GU = 4;
        const int     nB = nE * nK;
        for (int i0 = t0; i0 < nB; i0 += GU * TT)
          {
            double x[GU];
#pragma unroll
            for (int u = 0; u < GU; ++u)
              {
                const int idx = min(i0 + u * TT, nB - 1), i = idx % nE, c = idx / nE;
                const int e   = kid[c] * NEM + i;
                x[u]          = entry(erp[e][kco[c]], ers[e], eco[e], kco[c]);
              }
#pragma unroll
            for (int u = 0; u < GU; ++u)
              {
                const int idx = i0 + u * TT;
                if (idx < nB)
                  Bs[(idx / nE) * LDW + idx % nE] = x[u];
              }
          }
        for (int i0 = t0; i0 < nB; i0 += GU * TT)
          {
            double x[GU];
#pragma unroll
            for (int u = 0; u < GU; ++u)
              {
                const int idx = min(i0 + u * TT, nB - 1), r = idx % nK, j = idx / nK;
                const int co  = eco[kid[r] * NEM + j];
                x[u]          = entry(krp[r][co], krs[r], kco[r], co);
              }
#pragma unroll
            for (int u = 0; u < GU; ++u)
              {
                const int idx = i0 + u * TT;
                if (idx < nB)
                  Ks[(idx % nK) * LDW + idx / nK] = -x[u];
              }
          }
        for (int i = t0; i < nE; i += TT)
          {
            double x = rhs_scale(ers[i]) * *rhs_at(0, erp[i], ers[i], eco[i]);
            if (!LEAF)
              x += rhs_scale(ers[NEM + i]) * *rhs_at(1, erp[NEM + i], ers[NEM + i], eco[NEM + i]);
            Bs[nK * LDW + i] = x;
          }
        // beyond nE
        for (int idx = t0; idx < (NEM - nE) * (nK + 1); idx += TT)
          Bs[idx / (NEM - nE) * LDW + nE + idx % (NEM - nE)] = 0.;
        for (int idx = t0; idx < (NEM - nE) * nK; idx += TT)
          Ks[idx / (NEM - nE) * LDW + nE + idx % (NEM - nE)] = 0.;
      }
    __syncthreads();
    // W, a thread per column
    for (int c = tid; c <= nK; c += T)
      {
        double  x[NEM];
        double *b = Bs + c * LDW;
#pragma unroll
        for (int i = 0; i < NEM; ++i)
          x[i] = b[perm[i]];
#pragma unroll
        for (int r = 0; r < NEM; ++r)
          {
            // the factors are read where they are used: hoisted out of the
            // column loop they would spill
            asm volatile("" ::: "memory");
#pragma unroll
            for (int q = (r + 1) & ~1; q < NEM; q += 2)
              {
                const double2 lv = *reinterpret_cast<const double2 *>(LU + r * NEM + q);
                if (q > r)
                  x[q] -= lv.x * x[r];
                x[q + 1] -= lv.y * x[r];
              }
          }
#pragma unroll
        for (int r = NEM - 1; r >= 0; --r)
          {
            asm volatile("" ::: "memory");
            x[r] *= dinv[r];
#pragma unroll
            for (int q = 0; q < r; q += 2)
              {
                const double2 uv = *reinterpret_cast<const double2 *>(LU + r * NEM + q);
                x[q] -= uv.x * x[r];
                if (q + 1 < r)
                  x[q + 1] -= uv.y * x[r];
              }
          }
#pragma unroll
        for (int i = 0; i < NEM; ++i)
          b[i] = x[i];
      }
    __syncthreads();
    double *Fv = fronts + n.koff;
    for (int idx = tid; idx < nE * (nK + 1); idx += T)
      {
        const int i = idx % nE, c = idx / nE;
        Fv[(int64_t)c * n.ld + i] = Bs[c * LDW + i];
      }
    // Schur complement
    const int g = lane >> 2, tq = lane & 3;
    const int rt = (nK + 15) / 16, ctn = (nK + 1 + 31) / 32;
    for (int tile = warp; tile < rt * ctn; tile += T / 32)
      {
        const int r0 = (tile % rt) * 16, c0 = (tile / rt) * 32;
        double    acc[2][4][2];
        {
          const double *rp[2], *rr[2];
          double        rs[2];
          int           rk[2], ro[2];
#pragma unroll
          for (int i = 0; i < 2; ++i)
            {
              const int r = min(r0 + i * 8 + g, nK - 1);
              rp[i]       = krp[r];
              rs[i]       = krs[r];
              rk[i]       = kid[r];
              ro[i]       = kco[r];
              rr[i]       = rhs_at(rk[i], rp[i], rs[i], ro[i]);
            }
#pragma unroll
          for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int e = 0; e < 2; ++e)
              {
                const int c  = c0 + j * 8 + 2 * tq + e, cc = min(c, nK - 1);
                const int ck = c < nK ? kid[cc] : -1, co = kco[cc];
                // every load is made (behind branches they would wait for
                // each other), from the row's right-hand side where the entry
                // is zero
#pragma unroll
                for (int i = 0; i < 2; ++i)
                  {
                    const bool   in = ck == rk[i];
                    const double x  = *(in ? rp[i] + co : rr[i]);
                    acc[i][j][e]    = in ? entry(x, rs[i], ro[i], co) : (c == nK ? rhs_scale(rs[i]) * x : 0.);
                  }
              }
        }
#pragma unroll
        for (int ks = 0; ks < NEM / 4; ++ks)
          {
            double a[2], b[4];
#pragma unroll
            for (int i = 0; i < 2; ++i)
              a[i] = Ks[min(r0 + i * 8 + g, nK - 1) * LDW + ks * 4 + tq];
#pragma unroll
            for (int j = 0; j < 4; ++j)
              b[j] = Bs[min(c0 + j * 8 + g, nK) * LDW + ks * 4 + tq];
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
              for (int j = 0; j < 4; ++j)
                dmma8x8x4(acc[i][j][0], acc[i][j][1], a[i], b[j]);
          }
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e)
            {
              const int c = c0 + j * 8 + 2 * tq + e;
#pragma unroll
              for (int i = 0; i < 2; ++i)
                {
                  const int r = r0 + i * 8 + g;
                  if (r < nK && c <= nK)
                    Fv[(int64_t)c * n.ld + n.nEp + r] = acc[i][j][e];
                }
            }
      }
  }

  // ------------------------------------------------- E columns of the fronts
  // F_EE and F_KE into the batch's scratch; CTA (some of the columns, node)
  __global__ void __launch_bounds__(256)
  nd_gather_e_kernel(const NDNode *nodes, const int32_t *maps, NDCells C, const double *fronts, double *ecols)
  {
    const NDNode  n = nodes[blockIdx.y];
    const NDFront F{n, C, maps + n.map, fronts};
    for (int j = blockIdx.x; j < n.nE; j += gridDim.x)
      {
        double *A = ecols + n.eoff + (int64_t)j * n.ld;
#pragma unroll 4
        for (int i = threadIdx.x; i < n.ld; i += 256)
          {
            double x = 0.; // the pad rows stay zero
            if (i < n.nE)
              x = F.EE(i, j);
            else if (i >= n.nEp && i - n.nEp < n.nK)
              x = F.KE(i - n.nEp, j);
            A[i] = x;
          }
      }
  }

  // [F_EK | r_E], rows in pivot order, into the E rows of the front; CTA
  // (node, cb columns), staged in shared memory so that both sides are
  // coalesced
  __global__ void __launch_bounds__(256)
  nd_gather_b_kernel(const NDNode *nodes, const int32_t *maps, NDCells C, const int32_t *perm_all, int cb,
                     double *fronts)
  {
    extern __shared__ __align__(16) double sm[];
    const NDNode n  = nodes[blockIdx.y];
    const int    c0 = blockIdx.x * cb, nE = n.nE;
    const int    nc = min(cb, n.nK + 1 - c0);
    if (nc <= 0)
      return;
    const NDFront  F{n, C, maps + n.map, fronts};
    const int32_t *perm = perm_all + n.poff;
#pragma unroll 4
    for (int idx = threadIdx.x; idx < nc * nE; idx += 256)
      sm[idx] = F.EK(idx % nE, c0 + idx / nE);
    __syncthreads();
    double *B = fronts + n.koff + (int64_t)c0 * n.ld;
    for (int idx = threadIdx.x; idx < nc * n.nEp; idx += 256)
      {
        const int i = idx % n.nEp, c = idx / n.nEp;
        B[(int64_t)c * n.ld + i] = i < nE ? sm[c * nE + perm[i]] : 0.; // the pad row stays zero
      }
  }

  // -------------------------------------------------------------- dense LU
  // Right-looking LU with partial pivoting of F_EE for all fronts of a batch,
  // NDPanel columns per step, two launches per step.  Rows never move: every
  // step works on the list of rows not chosen yet, and the factors are
  // written in pivot order to their own array.
  //
  // nd_panel_kernel factorises a panel.  Each thread holds one row of it in
  // registers; per column a warp max-reduction, one CTA barrier and, for the
  // fronts whose rows need more than one CTA, one exchange of the C
  // candidates through the distributed shared memory of a cluster of C CTAs.
  // The kernel is a chain of NDPanel dependent column steps, bound by the
  // instructions and latencies of a step, not by any rate: one barrier per
  // step (the candidates' rows and reciprocals travel with their keys), and
  // code that stays in the instruction cache: the eight steps of a group are
  // unrolled, the groups are a loop (all 32 steps unrolled: 47 us per panel,
  // instruction fetches; all 32 rolled with a rotating row: 25 us, masking).
  // After a group the row is rotated by its eight columns, so the current
  // group is always in the first registers.
  constexpr int NDPanel   = 32;
  constexpr int NDPanelT  = 512;           // threads per CTA at most
  constexpr int NDPanelC  = 8;             // CTAs per cluster at most
  constexpr int NDPanelLd = NDPanel + 4;   // shared row stride (= 4 mod 16)
  constexpr int NDPanelG  = 8;             // columns per group
  constexpr int NDPanelN  = NDPanel / NDPanelG;

  // pivot key of a panel row: sign-free high word of the candidate down to 11
  // mantissa bits (the pivot is within 2^-11 of the largest), plus one, and
  // the thread, the first one winning ties
  __device__ __forceinline__ unsigned
  nd_panel_key(double x, int thread)
  {
    const unsigned hi = (unsigned)((unsigned long long)__double_as_longlong(fabs(x)) >> 32);
    return (((hi >> 9) + 1u) << 9) | (unsigned)(NDPanelT - 1 - thread);
  }
  __device__ __forceinline__ int
  nd_panel_key_row(unsigned key)
  {
    return NDPanelT - 1 - (int)(key & (NDPanelT - 1));
  }

  template <int CL>
  struct NDPanelShared
  {
    static constexpr int NW = NDPanelT / 32;
    double   wrow[2][NW][NDPanel]; // candidate row per warp (the columns still active)
    double   crow[2][CL][NDPanel]; // candidate row per CTA of the cluster
    // pivot rows by columns: [0] as they are, [1] rows and columns reversed
    double   LU[2][NDPanel][NDPanel + 2];
    double   whr[2][NW], chr[2][CL]; // reciprocal pivots
    double   rd[NDPanel];            // reciprocals of the diagonal of U (1 beyond w)
    unsigned wkey[2][NW], ckey[2][CL];
    int      ppos[NDPanel]; // list positions of the pivot rows
  };

  // one group of NDPanelG column steps, columns j0 .. j0 + 7 in v[0 .. 7];
  // nact of the blocks of eight columns are still active (this one included)
  template <int CL>
  __device__ __forceinline__ void
  nd_panel_group(double (&v)[NDPanel], NDPanelShared<CL> &S, int j0, int nact, int w, int t, int rank, bool &used,
                 int &mypos)
  {
    namespace cg   = cooperative_groups;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int jj = 0; jj < NDPanelG; ++jj)
      {
        if (j0 + jj >= w)
          break; // no rows are left (the same for every CTA of the cluster)
        constexpr int  PK   = 2; // columns per 16-byte access
        const int      buf  = jj & 1;
        const double   x0   = v[jj];
        const unsigned key  = used ? 0u : nd_panel_key(x0, threadIdx.x);
        const double   hx   = reciprocal_normal(x0);
        const unsigned kmax = __reduce_max_sync(0xffffffffu, key);
        if (key == kmax && key != 0u)
          {
            double2 *dst = reinterpret_cast<double2 *>(S.wrow[buf][warp]);
#pragma unroll
            for (int k = (jj + 1) / PK * PK; k < NDPanelG; k += PK)
              dst[k / PK] = make_double2(v[k], v[k + 1]);
#pragma unroll
            for (int b = 1; b < NDPanelN; ++b)
              if (b < nact)
#pragma unroll
                for (int k = b * NDPanelG; k < (b + 1) * NDPanelG; k += PK)
                  dst[k / PK] = make_double2(v[k], v[k + 1]);
            S.whr[buf][warp] = reciprocal(x0, hx);
          }
        if (lane == 0)
          S.wkey[buf][warp] = kmax;
        __syncthreads();
        const unsigned m2   = __reduce_max_sync(0xffffffffu, lane < nw ? S.wkey[buf][lane] : 0u);
        const int      tw   = nd_panel_key_row(m2); // thread of the CTA's candidate
        const double  *prow = S.wrow[buf][tw >> 5];
        double         hr   = S.whr[buf][tw >> 5];
        int            pid  = rank * (int)blockDim.x + tw;
        if (CL > 1)
          {
            cg::cluster_group cl = cg::this_cluster();
            if (warp < CL)
              {
                double *dst = cl.map_shared_rank(&S.crow[buf][rank][0], warp);
                dst[lane]   = prow[lane]; // the inactive columns are not read
                if (lane == 0)
                  {
                    *cl.map_shared_rank(&S.ckey[buf][rank], warp) = m2;
                    *cl.map_shared_rank(&S.chr[buf][rank], warp)  = hr;
                  }
              }
            nd_cluster_sync();
            const unsigned k3 = lane < CL ? S.ckey[buf][lane] : 0u;
            const unsigned m3 = __reduce_max_sync(0xffffffffu, k3);
            const int      cc = __ffs(__ballot_sync(0xffffffffu, lane < CL && k3 == m3)) - 1;
            prow              = S.crow[buf][cc];
            hr                = S.chr[buf][cc];
            pid               = cc * (int)blockDim.x + nd_panel_key_row(m3);
          }
        const bool    me = !used && t == pid;
        const double  l  = (used || me) ? 0. : -x0 * hr;
        const double2 *pr = reinterpret_cast<const double2 *>(prow);
#pragma unroll
        for (int k = (jj + 1) / PK * PK; k < NDPanelG; k += PK)
          {
            const double2 p = pr[k / PK];
            if (k > jj)
              v[k] = fma(l, p.x, v[k]);
            v[k + 1] = fma(l, p.y, v[k + 1]);
          }
#pragma unroll
        for (int b = 1; b < NDPanelN; ++b)
          if (b < nact)
#pragma unroll
            for (int k = b * NDPanelG; k < (b + 1) * NDPanelG; k += PK)
              {
                const double2 p = pr[k / PK];
                v[k]            = fma(l, p.x, v[k]);
                v[k + 1]        = fma(l, p.y, v[k + 1]);
              }
        if (!used && !me)
          v[jj] = -l;
        if (me)
          {
            used  = true;
            mypos = j0 + jj;
          }
        if (threadIdx.x == 0)
          {
            S.ppos[j0 + jj] = pid;
            S.rd[j0 + jj]   = hr;
          }
      }
    // the finished columns to the end
    double f[NDPanelG];
#pragma unroll
    for (int k = 0; k < NDPanelG; ++k)
      f[k] = v[k];
#pragma unroll
    for (int k = NDPanelG; k < NDPanel; ++k)
      v[k - NDPanelG] = v[k];
#pragma unroll
    for (int k = 0; k < NDPanelG; ++k)
      v[NDPanel - NDPanelG + k] = f[k];
  }

  template <int CL>
  __global__ void __launch_bounds__(NDPanelT, 1)
  nd_panel_kernel(const NDNode *nodes, int k0, const int32_t *ul_in, int32_t *ul_out, double *ecols,
                  double *luf, int32_t *perm, double *tinv, int *sing)
  {
    namespace cg = cooperative_groups;
    __shared__ __align__(16) NDPanelShared<CL> S;
    const NDNode &n  = nodes[blockIdx.x / CL];
    const int     nE = n.nE;
    if (nE <= k0)
      return; // every CTA of the cluster
    const int rank = CL > 1 ? (int)(blockIdx.x % CL) : 0;
    const int m = nE - k0, w = min(NDPanel, m);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, T = blockDim.x;
    const int t    = rank * T + tid; // position in the row list
    const bool has = t < m;
    const int  row = has ? (k0 ? ul_in[n.poff + t] : t) : 0;
    double    *A   = ecols + n.eoff + (int64_t)k0 * n.ld;
    double     v[NDPanel];
#pragma unroll
    for (int c = 0; c < NDPanel; ++c)
      v[c] = (has && c < w) ? A[(int64_t)c * n.ld + row] : 0.;
    bool used  = !has;
    int  mypos = -1;
    if (rank == 0)
      for (int i = tid; i < 2 * NDPanel * (NDPanel + 2); i += T)
        (&S.LU[0][0][0])[i] = 0.;
    if (tid < NDPanel)
      S.rd[tid] = 1.;
    if (CL > 1)
      nd_cluster_sync(); // every CTA of the cluster runs before its shared memory is written
    else
      __syncthreads();
#pragma unroll 1
    for (int g = 0; g < NDPanelN; ++g)
      nd_panel_group<CL>(v, S, g * NDPanelG, NDPanelN - g, w, t, rank, used, mypos);
    if (mypos >= 0)
      {
        double *d0 = &S.LU[0][0][mypos], *d1 = &S.LU[1][NDPanel - 1][NDPanel - 1 - mypos];
        if (CL > 1)
          {
            d0 = cg::this_cluster().map_shared_rank(d0, 0);
            d1 = cg::this_cluster().map_shared_rank(d1, 0);
          }
#pragma unroll
        for (int c = 0; c < NDPanel; ++c)
          {
            d0[c * (NDPanel + 2)]  = v[c];
            d1[-c * (NDPanel + 2)] = v[c];
          }
      }
    if (CL > 1)
      nd_cluster_sync(); // also: no CTA's shared memory is written after this
    else
      __syncthreads();
    if (rank == 0 && tid < w && (S.rd[tid] == 0. || isnan(S.rd[tid])))
      atomicExch(sing, 1); // a zero or non-finite pivot
    if (mypos >= 0)
      perm[n.poff + k0 + mypos] = row;
    else if (has)
      {
        int below = 0;
#pragma unroll
        for (int j = 0; j < NDPanel; ++j)
          below += (j < w && S.ppos[j] < t) ? 1 : 0;
        ul_out[n.poff + t - below] = row;
#pragma unroll
        for (int c = 0; c < NDPanel; ++c)
          A[(int64_t)c * n.ld + row] = v[c]; // rows are left only when w == NDPanel
      }
    if (rank == 0)
      {
        // inverses of the unit lower and of the upper diagonal block (identity
        // beyond w), a lane per column: substitution by columns, the upper
        // block on its reversed copy; groups as above
        if (warp < 2)
          {
            const bool up = warp == 1;
            double     y[NDPanel];
#pragma unroll
            for (int r = 0; r < NDPanel; ++r)
              y[r] = ((up ? NDPanel - 1 - r : r) == lane) ? 1. : 0.;
            double *out = tinv + n.tioff + ((int64_t)(k0 / NDPanel) * 2 + warp) * NDPanel * NDPanel + lane * NDPanel;
#pragma unroll 1
            for (int g = 0; g < NDPanelN; ++g)
              {
#pragma unroll
                for (int jj = 0; jj < NDPanelG; ++jj)
                  {
                    const int c = g * NDPanelG + jj;
                    if (up)
                      y[jj] *= S.rd[NDPanel - 1 - c];
                    const double  x = -y[jj];
                    const double *f = &S.LU[warp][c][g * NDPanelG];
#pragma unroll
                    for (int k = jj + 1; k < NDPanelG; ++k)
                      y[k] = fma(f[k], x, y[k]);
#pragma unroll
                    for (int b = 1; b < NDPanelN; ++b)
                      if (b < NDPanelN - g)
#pragma unroll
                        for (int k = b * NDPanelG; k < (b + 1) * NDPanelG; k += 2)
                          {
                            const double2 p = *reinterpret_cast<const double2 *>(f + k);
                            y[k]            = fma(p.x, x, y[k]);
                            y[k + 1]        = fma(p.y, x, y[k + 1]);
                          }
                  }
#pragma unroll
                for (int k = 0; k < NDPanelG; ++k)
                  out[up ? NDPanel - 1 - g * NDPanelG - k : g * NDPanelG + k] = y[k];
#pragma unroll
                for (int k = NDPanelG; k < NDPanel; ++k)
                  y[k - NDPanelG] = y[k];
              }
          }
        const int ldl = n.nEp;
        double   *LUF = luf + n.luoff + (int64_t)k0 * ldl + k0;
        for (int idx = tid; idx < w * w; idx += T)
          LUF[(int64_t)(idx / w) * ldl + idx % w] = S.LU[0][idx / w][idx % w];
      }
  }

  __device__ __forceinline__ void
  nd_cp_async8(double *dst, const double *src, bool valid)
  {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    const int      b = valid ? 8 : 0; // 0 source bytes: zero-filled
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(b));
  }
  __device__ __forceinline__ void
  nd_cp_async16(double *dst, const double *src, int bytes)
  {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes));
  }
  __device__ __forceinline__ void
  nd_cp_commit()
  {
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  template <int N>
  __device__ __forceinline__ void
  nd_cp_wait()
  {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
  }

  // The step's trailing update: CTA (64 rows of the list x 64 columns) forms
  // U12 = L11^-1 A[pivot rows] of its columns (the row tiles repeat it; the
  // first one stores it in the factors) and subtracts L21 U12, both on the
  // FP64 tensor path.
  constexpr int NDUpd = 64;

  __host__ __device__ constexpr size_t
  nd_update_smem()
  {
    return (size_t)(3 * NDUpd + NDPanel) * NDPanelLd * sizeof(double);
  }

  __global__ void __launch_bounds__(128)
  nd_update_kernel(const NDNode *nodes, int k0, int ctiles, const int32_t *ul, double *ecols, double *luf,
                   const int32_t *perm, const double *tinv)
  {
    extern __shared__ __align__(16) double sm[];
    __shared__ int rl[NDUpd];
    double       (*Gs)[NDPanelLd] = reinterpret_cast<double (*)[NDPanelLd]>(sm); // [column][pivot row]
    double       (*Us)[NDPanelLd] = Gs + NDUpd;                                  // [column][pivot row]
    double       (*Ls)[NDPanelLd] = Us + NDUpd;                                  // [row][panel column]
    double       (*Li)[NDPanelLd] = Ls + NDUpd;                                  // L11^-1, [column][row]
    const NDNode  &n  = nodes[blockIdx.y];
    const int      kn = k0 + NDPanel; // first trailing column
    const int      m  = n.nE - kn;    // trailing rows and columns
    const int      ct = blockIdx.x % ctiles, rt = blockIdx.x / ctiles;
    if (ct * NDUpd >= m || rt * NDUpd >= m)
      return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int c0 = kn + ct * NDUpd, nc = min(NDUpd, m - ct * NDUpd), nr = min(NDUpd, m - rt * NDUpd);
    double   *A  = ecols + n.eoff;
    const int64_t ld = n.ld;
    if (tid < NDUpd)
      rl[tid] = tid < nr ? ul[n.poff + rt * NDUpd + tid] : 0;
    {
      const int     k  = lane;
      const double *gr = A + perm[n.poff + k0 + k];
      for (int c = warp; c < NDUpd; c += 4)
        nd_cp_async8(&Gs[c][k], gr + (c0 + min(c, nc - 1)) * ld, c < nc);
      const double *ti = tinv + n.tioff + (int64_t)(k0 / NDPanel) * 2 * NDPanel * NDPanel;
      for (int idx = tid; idx < NDPanel * NDPanel / 2; idx += 128)
        nd_cp_async16(&Li[idx / 16][(idx % 16) * 2], ti + idx * 2, 16);
    }
    nd_cp_commit();
    __syncthreads(); // rl
    for (int idx = tid; idx < NDUpd * NDPanel; idx += 128)
      {
        const int r = idx % NDUpd, k = idx / NDUpd;
        nd_cp_async8(&Ls[r][k], A + (k0 + k) * ld + rl[r], r < nr);
      }
    nd_cp_commit();
    const int g = lane >> 2, q = lane & 3;
    const int wm = (warp & 1) * 32, wn = (warp >> 1) * 32;
    double    acc[4][4][2];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e)
        {
          const int c = wn + j * 8 + 2 * q + e;
#pragma unroll
          for (int i = 0; i < 4; ++i)
            {
              const int r  = wm + i * 8 + g;
              acc[i][j][e] = (r < nr && c < nc) ? A[(c0 + c) * ld + rl[r]] : 0.;
            }
        }
    nd_cp_wait<1>();
    __syncthreads();
    {
      double u[4][2][2];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
          u[i][j][0] = u[i][j][1] = 0.;
#pragma unroll
      for (int ks = 0; ks < NDPanel / 4; ++ks)
        {
          double b[2];
#pragma unroll
          for (int j = 0; j < 2; ++j)
            b[j] = Gs[warp * 16 + j * 8 + g][ks * 4 + q];
#pragma unroll
          for (int i = 0; i < 4; ++i)
            {
              const double a = Li[ks * 4 + q][i * 8 + g];
#pragma unroll
              for (int j = 0; j < 2; ++j)
                dmma8x8x4(u[i][j][0], u[i][j][1], a, b[j]);
            }
        }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e)
            Us[warp * 16 + j * 8 + 2 * q + e][i * 8 + g] = u[i][j][e];
    }
    nd_cp_wait<0>();
    __syncthreads();
    if (rt == 0)
      {
        double *U = luf + n.luoff + (int64_t)c0 * n.nEp + k0;
        for (int c = warp; c < nc; c += 4)
          U[(int64_t)c * n.nEp + lane] = Us[c][lane];
      }
#pragma unroll
    for (int ks = 0; ks < NDPanel / 4; ++ks)
      {
        double a[4], b[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
          a[i] = -Ls[wm + i * 8 + g][ks * 4 + q];
#pragma unroll
        for (int j = 0; j < 4; ++j)
          b[j] = Us[wn + j * 8 + g][ks * 4 + q];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j)
            dmma8x8x4(acc[i][j][0], acc[i][j][1], a[i], b[j]);
      }
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e)
        {
          const int c = wn + j * 8 + 2 * q + e;
#pragma unroll
          for (int i = 0; i < 4; ++i)
            {
              const int r = wm + i * 8 + g;
              if (r < nr && c < nc)
                A[(c0 + c) * ld + rl[r]] = acc[i][j][e];
            }
        }
  }

  // L below the diagonal blocks, from the rows' places into pivot order
  __global__ void __launch_bounds__(256)
  nd_lu_finish_kernel(const NDNode *nodes, const double *ecols, const int32_t *perm, double *luf)
  {
    const NDNode &n   = nodes[blockIdx.y];
    const int     nE = n.nE, ldl = n.nEp;
    const double *A = ecols + n.eoff;
    double       *L = luf + n.luoff;
    for (int c = blockIdx.x; c < (nE - 1) / NDPanel * NDPanel; c += gridDim.x)
      for (int i = (c / NDPanel + 1) * NDPanel + threadIdx.x; i < nE; i += 256)
        L[(int64_t)c * ldl + i] = A[(int64_t)c * n.ld + perm[n.poff + i]];
  }

  // The fronts beyond the panel kernel's rows: LU by cuSOLVER in place of
  // F_EE; its row swaps (1-based) turned into the pivot order, the factors
  // copied, the diagonal blocks inverted.  One front per launch.
  __global__ void
  nd_lib_perm_kernel(const NDNode *node, const int *ipiv, const int *info, int32_t *perm, int *sing)
  {
    int32_t *pm = perm + node->poff;
    for (int i = threadIdx.x; i < node->nE; i += blockDim.x)
      pm[i] = i;
    __syncthreads();
    if (threadIdx.x)
      return;
    if (*info)
      atomicExch(sing, 1);
    for (int j = 0; j < node->nE; ++j)
      {
        // within the front, whatever the library makes of NaN entries
        const int k = max(j, min(ipiv[j] - 1, node->nE - 1)), x = pm[j];
        pm[j]       = pm[k];
        pm[k]       = x;
      }
  }

  __global__ void __launch_bounds__(256)
  nd_lib_copy_kernel(const NDNode *node, const double *ecols, double *luf)
  {
    const NDNode &n = *node;
    for (int c = blockIdx.x; c < n.nE; c += gridDim.x)
      for (int i = threadIdx.x; i < n.nE; i += 256)
        luf[n.luoff + (int64_t)c * n.nEp + i] = ecols[n.eoff + (int64_t)c * n.ld + i];
  }

  __global__ void __launch_bounds__(64)
  nd_lib_inverse_kernel(const NDNode *node, const double *luf, double *tinv)
  {
    __shared__ double S[NDPanel][NDPanel + 1];
    const NDNode &n  = *node;
    const int     r0 = blockIdx.x * NDPanel, w = min(NDPanel, n.nE - r0);
    const int     lane = threadIdx.x & 31, which = threadIdx.x >> 5;
    for (int idx = threadIdx.x; idx < NDPanel * NDPanel; idx += 64)
      {
        const int r = idx % NDPanel, c = idx / NDPanel;
        S[r][c] = (r < w && c < w) ? luf[n.luoff + (int64_t)(r0 + c) * n.nEp + r0 + r] : (r == c ? 1. : 0.);
      }
    __syncthreads();
    double x[NDPanel];
    if (which == 0)
      {
#pragma unroll
        for (int r = 0; r < NDPanel; ++r)
          {
            double y = (r == lane) ? 1. : 0.;
#pragma unroll
            for (int s = 0; s < r; ++s)
              y -= S[r][s] * x[s];
            x[r] = y;
          }
      }
    else
      {
#pragma unroll
        for (int r = NDPanel - 1; r >= 0; --r)
          {
            double y = (r == lane) ? 1. : 0.;
#pragma unroll
            for (int s = r + 1; s < NDPanel; ++s)
              y -= S[r][s] * x[s];
            x[r] = y / S[r][r];
          }
      }
    double *out = tinv + n.tioff + ((int64_t)blockIdx.x * 2 + which) * NDPanel * NDPanel;
    for (int r = 0; r < NDPanel; ++r)
      out[lane * NDPanel + r] = x[r];
  }

  // ------------------------------------------------------ triangular solves
  // W_b = U_bb^-1 L_bb^-1 B_b for the rows [b0, b0 + bs) of the fronts
  // (dir bit 0: L, bit 1: U), in place.  CTA (32 columns, front): the whole
  // column tile stays in shared memory for both sweeps; the 32 x 32 blocks of
  // the factors stream through a ring of cp.async stages, the diagonal blocks
  // as their inverses, all products on the FP64 tensor path.  Bound by the
  // factors' L2 reads and the tensor path; one read and one write of B.
  // CT columns per CTA: 64 where there are enough tiles to fill the GPU (half
  // the factor reads and twice the products per barrier), else 32.
  constexpr int NDSolveStages = 3;

  __host__ __device__ constexpr int
  nd_solve_rows(int CT) // rows of a column tile that fit in shared memory
  {
    return CT == 64 ? 288 : 576;
  }

  __host__ __device__ inline size_t
  nd_solve_smem(int CT, int bs)
  {
    const int rows = (bs + NDPanel - 1) / NDPanel * NDPanel;
    return ((size_t)CT * (rows + 4) + (size_t)NDSolveStages * NDPanel * NDPanelLd) * sizeof(double);
  }

  template <int CT>
  __global__ void __launch_bounds__(256)
  nd_solve_kernel(const NDNode *nodes, int b0, int bs, int dir, const double *luf, const double *tinv,
                  double *fronts)
  {
    extern __shared__ __align__(16) double sm[];
    const NDNode &n  = nodes[blockIdx.y];
    const int     c0 = blockIdx.x * CT, nc = min(CT, n.nK + 1 - c0);
    const int     nr = min(bs, n.nE - b0);
    if (nc <= 0 || nr <= 0)
      return;
    const int     nblk = (nr + NDPanel - 1) / NDPanel;
    const int     ldb  = (bs + NDPanel - 1) / NDPanel * NDPanel + 4;
    double       *Bs   = sm;                                   // [column][row]
    double       *Ts   = sm + (size_t)CT * ldb;               // stages of [column][row] blocks
    const int     tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int     g = lane >> 2, q = lane & 3;
    constexpr int NT = CT / 16; // column tiles per warp
    const int     mt = warp & 3, nt = (warp >> 2) * NT;
    double       *B  = fronts + n.koff + (int64_t)c0 * n.ld + b0;
    const double *LU = luf + n.luoff + (int64_t)b0 * n.nEp + b0;
    const double *TI = tinv + n.tioff + (int64_t)(b0 / NDPanel) * 2 * NDPanel * NDPanel;
    const int     ldl = n.nEp;
    for (int c = warp; c < CT; c += 8)
      for (int r = lane; r < nblk * NDPanel; r += 32)
        Bs[c * ldb + r] = (c < nc && r < nr) ? B[(int64_t)c * n.ld + r] : 0.;

    // the blocks in the order of use: (sweep, block row i, block column j);
    // j == i stands for the diagonal block's inverse, the last of its row
    struct It
    {
      int d, i, j;
    };
    const auto first = [&](int d) { return d == 0 ? It{0, 0, 0} : It{1, nblk - 1, nblk - 1}; };
    const auto next  = [&](It t) {
      // forward rows: j = 0 .. i; backward rows: j = nblk - 1 .. i
      if (t.d == 0)
        {
          if (t.j < t.i)
            return It{0, t.i, t.j + 1};
          if (t.i + 1 < nblk)
            return It{0, t.i + 1, 0};
          return (dir & 2) ? first(1) : It{2, 0, 0};
        }
      if (t.j > t.i)
        return It{1, t.i, t.j - 1};
      if (t.i > 0)
        return It{1, t.i - 1, nblk - 1};
      return It{2, 0, 0};
    };
    const auto issue = [&](It t, int stage) {
      if (t.d < 2)
        {
          double *dst = Ts + (size_t)stage * NDPanel * NDPanelLd;
#pragma unroll
          for (int h = 0; h < 2; ++h)
            {
              const int idx = tid + 256 * h, r = (idx % 16) * 2, k = idx / 16;
              if (t.j == t.i)
                nd_cp_async16(dst + k * NDPanelLd + r,
                              TI + ((int64_t)t.i * 2 + t.d) * NDPanel * NDPanel + k * NDPanel + r, 16);
              else
                {
                  const int rr = t.i * NDPanel + r, kk = t.j * NDPanel + k;
                  const int bytes = kk < nr ? 8 * max(0, min(2, nr - rr)) : 0;
                  nd_cp_async16(dst + k * NDPanelLd + r, bytes ? LU + (int64_t)kk * ldl + rr : LU, bytes);
                }
            }
        }
      nd_cp_commit();
    };
    It p = first((dir & 1) ? 0 : 1), t = p;
#pragma unroll
    for (int s = 0; s < NDSolveStages - 1; ++s)
      {
        issue(p, s);
        if (p.d < 2)
          p = next(p);
      }
    double acc[NT][2] = {};
    bool   fresh     = true; // the row's accumulators are not loaded yet
    for (int it = 0; t.d < 2; ++it)
      {
        nd_cp_wait<NDSolveStages - 2>();
        __syncthreads();
        issue(p, (it + NDSolveStages - 1) % NDSolveStages);
        if (p.d < 2)
          p = next(p);
        const double *A = Ts + (size_t)(it % NDSolveStages) * NDPanel * NDPanelLd;
        const int     row = t.i * NDPanel + mt * 8 + g;
        if (fresh && t.j != t.i)
          {
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
              for (int e = 0; e < 2; ++e)
                acc[j][e] = Bs[((nt + j) * 8 + 2 * q + e) * ldb + row];
            fresh = false;
          }
        if (t.j != t.i)
          {
            // all fragments of the block first: the loads overlap
            double a[NDPanel / 4], b[NDPanel / 4][NT];
#pragma unroll
            for (int ks = 0; ks < NDPanel / 4; ++ks)
              {
                a[ks] = -A[(ks * 4 + q) * NDPanelLd + mt * 8 + g];
#pragma unroll
                for (int j = 0; j < NT; ++j)
                  b[ks][j] = Bs[((nt + j) * 8 + g) * ldb + t.j * NDPanel + ks * 4 + q];
              }
#pragma unroll
            for (int ks = 0; ks < NDPanel / 4; ++ks)
#pragma unroll
              for (int j = 0; j < NT; ++j)
                dmma8x8x4(acc[j][0], acc[j][1], a[ks], b[ks][j]);
          }
        else
          {
            if (!fresh)
              {
#pragma unroll
                for (int j = 0; j < NT; ++j)
#pragma unroll
                  for (int e = 0; e < 2; ++e)
                    Bs[((nt + j) * 8 + 2 * q + e) * ldb + row] = acc[j][e];
                __syncthreads();
              }
            double o[NT][2] = {};
#pragma unroll
            for (int ks = 0; ks < NDPanel / 4; ++ks)
              {
                const double a = A[(ks * 4 + q) * NDPanelLd + mt * 8 + g];
#pragma unroll
                for (int j = 0; j < NT; ++j)
                  dmma8x8x4(o[j][0], o[j][1], a, Bs[((nt + j) * 8 + g) * ldb + t.i * NDPanel + ks * 4 + q]);
              }
            __syncthreads();
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
              for (int e = 0; e < 2; ++e)
                Bs[((nt + j) * 8 + 2 * q + e) * ldb + row] = o[j][e];
            fresh = true;
          }
        t = next(t);
      }
    nd_cp_wait<0>();
    __syncthreads();
    for (int c = warp; c < nc; c += 8)
      for (int r = lane; r < nr; r += 32)
        B[(int64_t)c * n.ld + r] = Bs[c * ldb + r];
  }

  // ------------------------------------------------------------ C -= A B
  // 64 x 64 tiles of C, 128 threads (2 x 2 warps of 32 x 32), 16-deep stages
  // of A and B through cp.async.
  // SCHUR: F_KK - F_KE W with the front's entries (the children's) as the
  // initial accumulators, stored once, the right-hand-side column included.
  // Otherwise: rows [r0, r0 + mr) of the E rows of the fronts minus the
  // factors' block times the solved rows [b0, b0 + bs) (blocked triangular
  // solves of the fronts whose columns do not fit in shared memory).
  constexpr int NDGM = 64, NDGN = 64, NDGK = 16;
  constexpr int NDGLA = NDGM + 4; // As[k][m] row stride (= 4 mod 16)
  constexpr int NDGLB = NDGK + 4; // Bs[n][k] row stride
  constexpr int NDGStages = 3;

  __host__ __device__ constexpr size_t
  nd_gemm_smem()
  {
    return (size_t)NDGStages * (NDGK * NDGLA + NDGN * NDGLB) * sizeof(double);
  }

  template <bool SCHUR>
  __global__ void __launch_bounds__(128)
  nd_gemm_kernel(const NDNode *nodes, const int32_t *maps, NDCells Cc, int tiles_m, int r0, int mr, int b0, int bs,
                 const double *ecols, const double *luf, double *fronts)
  {
    extern __shared__ __align__(16) double sm[];
    const NDNode  n  = nodes[blockIdx.y];
    const int     m0 = (blockIdx.x % tiles_m) * NDGM, n0 = (blockIdx.x / tiles_m) * NDGN;
    const int     m  = SCHUR ? n.nK : min(mr, n.nE - r0);
    const int     nn = n.nK + 1;
    const int     k  = SCHUR ? n.nE : min(bs, n.nE - b0);
    if (m0 >= m || n0 >= nn || k <= 0)
      return;
    const int64_t lda = SCHUR ? n.ld : n.nEp;
    const double *A   = SCHUR ? ecols + n.eoff + n.nEp : luf + n.luoff + (int64_t)b0 * n.nEp + r0;
    double       *F   = fronts + n.koff;
    const double *Bm  = F + (SCHUR ? 0 : b0);
    double       *Cm  = F + (SCHUR ? n.nEp : r0);
    const int     tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int     wm = (warp & 1) * 32, wn = (warp >> 1) * 32;
    const int     nchunk = (k + NDGK - 1) / NDGK;
    const int     g = lane >> 2, q = lane & 3;

    const auto As = [&](int st) { return sm + (size_t)st * (NDGK * NDGLA + NDGN * NDGLB); };
    const auto issue = [&](int chunk, int st) {
      if (chunk < nchunk)
        {
          double   *a = As(st), *b = a + NDGK * NDGLA;
          const int k0 = chunk * NDGK;
#pragma unroll
          for (int h = 0; h < NDGM * NDGK / 2 / 128; ++h)
            {
              const int  idx = tid + 128 * h, mm = (idx % (NDGM / 2)) * 2, kk = idx / (NDGM / 2);
              const bool ok = m0 + mm < m && k0 + kk < k; // rows are padded to even
              nd_cp_async16(a + kk * NDGLA + mm, ok ? A + (k0 + kk) * lda + m0 + mm : A, ok ? 16 : 0);
            }
#pragma unroll
          for (int h = 0; h < NDGN * NDGK / 2 / 128; ++h)
            {
              const int idx = tid + 128 * h, kk = (idx % (NDGK / 2)) * 2, c = idx / (NDGK / 2);
              const int bytes = n0 + c < nn ? 8 * max(0, min(2, k - k0 - kk)) : 0;
              nd_cp_async16(b + c * NDGLB + kk, bytes ? Bm + (int64_t)(n0 + c) * n.ld + k0 + kk : Bm, bytes);
            }
        }
      nd_cp_commit();
    };
#pragma unroll
    for (int s = 0; s < NDGStages - 1; ++s)
      issue(s, s);
    double acc[4][4][2];
    if (SCHUR && n.cell >= 0)
      {
        const NDFront F_{n, Cc, maps + n.map, fronts};
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e)
            {
              const int c = n0 + wn + j * 8 + 2 * q + e;
#pragma unroll
              for (int i = 0; i < 4; ++i)
                {
                  const int r  = m0 + wm + i * 8 + g;
                  acc[i][j][e] = (r < m && c < nn) ? F_.KK(r, c) : 0.;
                }
            }
      }
    else if (SCHUR)
      {
        // rows as pointers into the child that holds them, columns as offsets
        const int32_t *km = maps + n.map + 2 * n.nE;
        constexpr int  KM = (1 << NDKidBit) - 1;
        const double  *rp[4];
        int            rk[4];
        int64_t        rr[4]; // offset of the right-hand-side column
#pragma unroll
        for (int i = 0; i < 4; ++i)
          {
            const int k = km[min(m0 + wm + i * 8 + g, m - 1)];
            rr[i]       = (int64_t)((k >> NDKidBit) ? n.cnK[1] : n.cnK[0]) * ((k >> NDKidBit) ? n.cld[1] : n.cld[0]);
            rk[i]       = k >> NDKidBit;
            rp[i]       = fronts + (rk[i] ? n.coff[1] : n.coff[0]) + (rk[i] ? n.cEp[1] : n.cEp[0]) + (k & KM);
          }
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e)
            {
              const int     c  = n0 + wn + j * 8 + 2 * q + e;
              const int     k  = km[min(c, n.nK - 1)];
              const int     ck = c < n.nK ? k >> NDKidBit : -1;
              const int64_t co = (int64_t)(k & KM) * (ck > 0 ? n.cld[1] : n.cld[0]);
              // every load is made, from a fixed place where the entry is
              // zero: behind branches the loads would wait for each other
#pragma unroll
              for (int i = 0; i < 4; ++i)
                {
                  const bool    in  = ck == rk[i] || c == n.nK;
                  const int64_t off = c == n.nK ? rr[i] : co;
                  const double  x   = *(in ? rp[i] + off : fronts);
                  acc[i][j][e]      = in ? x : 0.;
                }
            }
      }
    else
      {
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e)
            {
              const int c = n0 + wn + j * 8 + 2 * q + e;
#pragma unroll
              for (int i = 0; i < 4; ++i)
                {
                  const int r  = m0 + wm + i * 8 + g;
                  acc[i][j][e] = (r < m && c < nn) ? Cm[(int64_t)c * n.ld + r] : 0.;
                }
            }
      }
    for (int c = 0; c < nchunk; ++c)
      {
        nd_cp_wait<NDGStages - 2>();
        __syncthreads();
        issue(c + NDGStages - 1, (c + NDGStages - 1) % NDGStages);
        const double *a_s = As(c % NDGStages), *b_s = a_s + NDGK * NDGLA;
#pragma unroll
        for (int ks = 0; ks < NDGK / 4; ++ks)
          {
            double a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
              a[i] = -a_s[(ks * 4 + q) * NDGLA + wm + i * 8 + g];
#pragma unroll
            for (int j = 0; j < 4; ++j)
              b[j] = b_s[(wn + j * 8 + g) * NDGLB + ks * 4 + q];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
              for (int j = 0; j < 4; ++j)
                dmma8x8x4(acc[i][j][0], acc[i][j][1], a[i], b[j]);
          }
      }
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e)
        {
          const int c = n0 + wn + j * 8 + 2 * q + e;
#pragma unroll
          for (int i = 0; i < 4; ++i)
            {
              const int r = m0 + wm + i * 8 + g;
              if (r < m && c < nn)
                Cm[(int64_t)c * n.ld + r] = acc[i][j][e];
            }
        }
  }

  // The triangular solves of a front without kept dofs (the root): one
  // column, resident in shared memory of one CTA per front.  Per block of
  // NDPanel rows the inverted diagonal block (a warp per row), then the other
  // rows a thread each: a chain of 2 nE / NDPanel L2 round trips, where the
  // column tiles above would pad one column to 32 and sweep it in several
  // launches (2304 rows: 1.3 ms before).
  constexpr int NDRootT = 512;

  __global__ void __launch_bounds__(NDRootT, 1)
  nd_root_solve_kernel(const NDNode *nodes, const double *luf, const double *tinv, double *fronts)
  {
    extern __shared__ __align__(16) double sm[]; // the column, padded to whole blocks
    __shared__ double xb[NDPanel];
    const NDNode &n    = nodes[blockIdx.x];
    const int     nE   = n.nE, nblk = (nE + NDPanel - 1) / NDPanel, ldl = n.nEp;
    const double *LU = luf + n.luoff, *TI = tinv + n.tioff;
    double       *B  = fronts + n.koff;
    const int     tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int r = tid; r < nblk * NDPanel; r += NDRootT)
      sm[r] = r < nE ? B[r] : 0.;
    __syncthreads();
    for (int s = 0; s < 2 * nblk; ++s)
      {
        const bool    up = s >= nblk;
        const int     i  = up ? 2 * nblk - 1 - s : s, r0 = i * NDPanel;
        const double *inv = TI + ((int64_t)i * 2 + (up ? 1 : 0)) * NDPanel * NDPanel;
        for (int row = warp; row < NDPanel; row += NDRootT / 32)
          {
            double v = inv[lane * NDPanel + row] * sm[r0 + lane];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
              v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0)
              xb[row] = v;
          }
        __syncthreads();
        if (tid < NDPanel)
          sm[r0 + tid] = xb[tid];
        const int f = up ? 0 : r0 + NDPanel, l = up ? r0 : nE, w = min(NDPanel, nE - r0);
        for (int r = f + tid; r < l; r += NDRootT)
          {
            const double *col = LU + (int64_t)r0 * ldl + r;
            double        a   = 0.;
            if (w == NDPanel)
              {
                double f[NDPanel]; // all loads in flight
#pragma unroll
                for (int k = 0; k < NDPanel; ++k)
                  f[k] = col[(int64_t)k * ldl];
#pragma unroll
                for (int k = 0; k < NDPanel; ++k)
                  a += f[k] * xb[k];
              }
            else
              for (int k = 0; k < w; ++k)
                a += col[(int64_t)k * ldl] * xb[k];
            sm[r] -= a;
          }
        __syncthreads();
      }
    for (int r = tid; r < nE; r += NDRootT)
      B[r] = sm[r];
  }

  // ------------------------------------------------------ back substitution
  // x_E = y_E - W x_K for every node of a batch.  CTA (node, block of R
  // eliminated rows) of R x S threads: thread (row t % R, slice t / R) sums
  // the terms k = slice, slice + S, ... of W x_K (for one k the R rows are
  // consecutive in memory), and the S partial sums of a row are added in
  // shared memory.  Short dependency chains: the top fronts have few rows per
  // node and thousands of kept dofs.
  __global__ void
  nd_backsolve_kernel(int R, const NDNode *nodes, const int32_t *fdofs, const double *fronts, double *x)
  {
    extern __shared__ __align__(16) double sm[];
    const NDNode &n  = nodes[blockIdx.x];
    const int     nE = n.nE, nK = n.nK;
    if ((int)blockIdx.y * R >= nE)
      return;
    const int      S    = blockDim.x / R;
    double        *xk   = sm;
    double        *part = sm + nK;
    const int32_t *dl   = fdofs + n.doff;
    for (int k = threadIdx.x; k < nK; k += blockDim.x)
      xk[k] = x[dl[nE + k]];
    __syncthreads();
    const double *Fv = fronts + n.koff;
    const int     t = threadIdx.x, il = t % R, sl = t / R;
    const int     i = blockIdx.y * R + il;
    if (sl < S)
      {
        double v = 0.;
        if (i < nE)
          for (int k = sl; k < nK; k += S)
            v += Fv[(int64_t)k * n.ld + i] * xk[k];
        part[sl * R + il] = v;
      }
    __syncthreads();
    if (t < R && i < nE)
      {
        double v = Fv[(int64_t)nK * n.ld + i];
        for (int s = 0; s < S; ++s)
          v -= part[s * R + t];
        x[dl[i]] = v;
      }
  }
} // namespace ddhdg
