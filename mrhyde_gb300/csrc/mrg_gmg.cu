// Geometric multigrid preconditioner for Q1 problems on the structured graph, and the CG that uses it.
//
// The reference's linear solver is Belos with an algebraic multigrid preconditioner (MueLu) or its own
// Jacobi PCG (src/managers/solver/solverManager_solvers.hpp:812-901; Belos/MueLu options in
// src/interfaces/linear_algebra/linearAlgebraInterface_solvers.hpp:15-160).  On the structured box the
// multigrid hierarchy is known in closed form, so it is built geometrically and Galerkin-exactly:
//
//   * levels: vertex coarsening by 2 along the axes that still have >= 3 cells and whose cells are at
//     most twice as long as the shortest (semi-coarsening on stretched grids); a fine node with an
//     even index is a coarse node, and when the cell count is odd the last fine node is kept as a coarse
//     node too (the last coarse cell is one fine cell wide).  Every level has the canonical 27-point
//     (9-point in 2-D) layout of a p = 1 grid, so the level operators use the same CSR layout, row
//     formulas and staged SpMV as the fine one.
//   * interpolation P: tensor product of 1-D linear interpolation (weights 1 or 1/2); rows of fixed
//     (strong Dirichlet) fine nodes and columns of fixed coarse nodes are zero, so the hierarchy acts on
//     the free unknowns only, where J is symmetric.
//   * coarse operators A_c = P^T A_f P (restricted to free nodes; fixed coarse rows are identity rows),
//     computed as one 1-D Galerkin sweep per coarsened axis (the masked P is a tensor product).
//   * smoother: Chebyshev polynomial of degree 2 in D^{-1} A on [0.25 L, L], L the Gershgorin bound
//     max_i sum_j |a_ij| / a_ii of the level (computed on the device; no host synchronisation);
//   * coarsest level (at most 27 unknowns): dense inverse, Gauss-Jordan on the device.
//   * V(2,2) cycle, symmetric, so it preconditions CG.
//
// The CG keeps q = A p by recurrence (p <- z + beta p, q <- A z + beta q) so the SpMV reads z and no
// separate direction update is needed; dot products reduce deterministically (per-block partials,
// last block sums in index order).  The hierarchy and the CG run in the precision of the Jacobian
// (FP64, or FP32 for the inner solve of the mixed path).  Chunks of iterations are captured as CUDA
// graphs; the host reads the done flag once per chunk.
#include <algorithm>
#include <cmath>
#include <mutex>
#include <string>
#include <type_traits>
#include <vector>

#include "mrg_device.cuh"
#include "mrg_internal.h"

namespace {

using namespace mrgdev;

constexpr int NT = WST;            // threads per CTA
constexpr int NU = 2;              // Chebyshev degree (pre and post smoothing)
constexpr double CHEB_LO = 0.25;   // lower end of the smoothed interval, fraction of the bound
constexpr int GCHUNK = 2;          // Krylov iterations per captured graph (2: fewer nodes to instantiate and fewer iterations past convergence than 4; measured on small and large problems)
constexpr int MAXC = 32;           // largest coarsest level solved densely
constexpr int MAXLEV = 16;
constexpr int64_t RAP_WARP_ROWS = 24576;  // Galerkin sweeps with fewer output rows: one warp per row

// CTAs per SM of the kernels with the staged row loop: what their shared buffers allow
template <typename T>
constexpr int staged_per_sm() { return sizeof(T) == 8 ? 4 : 7; }

// ---- 1-D transfer along one axis ----------------------------------------------------------------
// Parents of fine node i (fine nodes 0..nnf-1, coarse nodes 0..nnc-1) with interpolation weights.
__host__ __device__ inline int axis_parents(int i, int nnf, int nnc, int coarsen, int* pc, float* pw) {
  if (!coarsen) { pc[0] = i; pw[0] = 1.0f; return 1; }
  if ((i & 1) == 0) { pc[0] = i >> 1; pw[0] = 1.0f; return 1; }
  if (i == nnf - 1) { pc[0] = nnc - 1; pw[0] = 1.0f; return 1; }  // odd last node is kept
  pc[0] = (i - 1) >> 1; pw[0] = 0.5f;
  pc[1] = (i + 1) >> 1; pw[1] = 0.5f;
  return 2;
}

// Children of coarse node c with their weights (the transpose of axis_parents).
__device__ inline int axis_children(int c, int nnf, int nnc, int coarsen, int* ci, float* cw) {
  if (!coarsen) { ci[0] = c; cw[0] = 1.0f; return 1; }
  int n = 0;
  for (int i = 2 * c - 1; i <= 2 * c + 1; ++i) {
    if (i < 0 || i >= nnf) continue;
    int pc[2];
    float pw[2];
    const int np = axis_parents(i, nnf, nnc, 1, pc, pw);
    for (int k = 0; k < np; ++k)
      if (pc[k] == c) { ci[n] = i; cw[n] = pw[k]; ++n; }
  }
  return n;
}

struct Xfer {
  int co[3];  // axis coarsened from the finer level
};

template <typename T>
struct LevDev {
  Grid g;
  int64_t n;
  const T* A;
  T* minv;
  T *xa, *xb, *d, *b, *r;
};

struct GScal {
  double rho, pq, alpha, beta, r0, rnorm, tol;
  double omega, rv;  // BiCGStab
  float alpha32, beta32, omega32;  // FP32 copies, rounded once by the thread that sets the scalar
  int iter, maxiter, done, status;
  unsigned int counter;
  int err;
};

// a scalar in the vectors' precision
template <typename T>
__device__ __forceinline__ T alpha_of(const GScal* S) {
  if constexpr (sizeof(T) == 4) return S->alpha32; else return S->alpha;
}
template <typename T>
__device__ __forceinline__ T beta_of(const GScal* S) {
  if constexpr (sizeof(T) == 4) return S->beta32; else return S->beta;
}
template <typename T>
__device__ __forceinline__ T omega_of(const GScal* S) {
  if constexpr (sizeof(T) == 4) return S->omega32; else return S->omega;
}

template <int P, typename T>
__device__ __forceinline__ auto row_prod(const Grid& g, const RowInfo& R, const T* vals, const T* x) {
  if constexpr (sizeof(T) == 4) return row_apply_f<P, true>(g, R, vals, x);
  else return row_apply<P, double, double, true>(g, R, vals, x);
}

// f(n, R, vals) for every row: Q1 rows through the per-warp staged loop, Q2 rows (125-point) read directly.  gate
// waits for the predecessor (pdl_wait) and says whether to go on.
template <int P, typename T, typename F, typename Gate>
__device__ __forceinline__ bool level_rows(const Grid& g, int64_t n, const T* __restrict__ A, unsigned char* smem_raw,
                                           uint64_t* mbar, F&& f, Gate&& gate) {
  if constexpr (P == 1) {
    return warp_staged_rows<T>(g, n, A, smem_raw, mbar, f, gate);
  } else {
    if (!gate()) return true;
    for (int64_t i = (int64_t)blockIdx.x * NT + threadIdx.x; i < n; i += (int64_t)gridDim.x * NT) {
      int ix, iy, iz;
      decompose(g, i, ix, iy, iz);
      const RowInfo R = row_info<P>(g, ix, iy, iz);
      f(i, R, A + R.rp);
    }
    return true;
  }
}

// Per-axis polynomial order of a grid's coupling ranges (an intermediate grid of the Q2 -> Q1 Galerkin
// sweeps couples +-1 along the swept axes and +-2 along the others).
struct P3 {
  int p[3];
};

__device__ __forceinline__ RowInfo row_info_p3(const Grid& g, const P3& pp, int ix, int iy, int iz) {
  RowInfo R;
  axis_range(ix, g.nn[0], pp.p[0], R.lx, R.cx);
  axis_range(iy, g.nn[1], pp.p[1], R.ly, R.cy);
  if (g.dim == 3) axis_range(iz, g.nn[2], pp.p[2], R.lz, R.cz); else { R.lz = 0; R.cz = 1; }
  R.rp = g.P[2][iz] * g.T[1] * g.T[0] + (int64_t)R.cz * (g.P[1][iy] * g.T[0] + (int64_t)R.cy * g.P[0][ix]);
  return R;
}

__device__ __forceinline__ bool is_done(const GScal* S) { return ((volatile const GScal*)S)->done != 0; }

// whether coordinate i of axis a lies on no Dirichlet face of that axis
__device__ __forceinline__ bool axis_free(const Grid& g, int a, int i) {
  if (a >= g.dim) return true;
  return !(((g.faces >> (2 * a)) & 1u) && i == 0) && !(((g.faces >> (2 * a + 1)) & 1u) && i == g.nn[a] - 1);
}

// ---- setup kernels ------------------------------------------------------------------------------
// One axis of the Galerkin product, one thread per row of the output grid gc (gc = gf coarsened along
// `axis` only).  The free nodes form a Cartesian product (Dirichlet faces are axis-aligned), so the
// masked interpolation is a tensor product and P^T A P is three such sweeps (x, then y, then z),
// each keeping the 27-point layout on an intermediate grid: ~160 multiply-adds per output row instead
// of ~5,800 for the direct triple product.
//
// The h-levels (order 1) take k_rap_line, which adds the same products in the same order as the general loop (children
// ascending, then the row's entries in storage order, then the lower and upper parent).
// One child's contribution to an output row of an order-1 grid: the child at 2 I + DC along A, vals its row.  The row's
// neighbours along an axis that do not exist or are fixed have m[axis][.] false; plo, phi: the weights with which the
// fine column at 2 I + s (s = -2 .. 2) goes to the coarse columns I + floor(s / 2) and I + ceil(s / 2) (0: fixed or none).
template <typename T, int A, int DC>
__device__ __forceinline__ void rap_child(const T* vals, const RowInfo& R, const int (&lo)[3], const bool (&m)[3][3],
                                          const float (&plo)[5], const float (&phi)[5], T wc, T* acc) {
  // lo[a]: 1 if the row has a coupling at offset -1 along a
  const T* v0 = vals + (lo[2] * R.cy + lo[1]) * R.cx + lo[0];
#pragma unroll
  for (int ez = -1; ez <= 1; ++ez)
#pragma unroll
    for (int ey = -1; ey <= 1; ++ey) {
      const T* v1 = v0 + (ez * R.cy + ey) * R.cx;
#pragma unroll
      for (int ex = -1; ex <= 1; ++ex) {
        const bool in = m[0][ex + 1] && m[1][ey + 1] && m[2][ez + 1];
        const T a = (in ? v1[ex] : T(0)) * wc;
        const int e[3] = {ex, ey, ez};
        const int sft = DC + e[A];
        int o[3] = {ex, ey, ez};
        o[A] = sft >= 0 ? sft / 2 : -((1 - sft) / 2);  // floor
        acc[(o[2] + 1) * 9 + (o[1] + 1) * 3 + (o[0] + 1)] += a * (T)plo[sft + 2];
        if (sft & 1) {
          o[A] += 1;
          acc[(o[2] + 1) * 9 + (o[1] + 1) * 3 + (o[0] + 1)] += a * (T)phi[sft + 2];
        }
      }
    }
}

template <typename T>
__global__ void __launch_bounds__(NT) k_rap_axis(Grid gf, P3 pf, Grid gc, P3 pc, int axis, const T* __restrict__ Af,
                                                 T* __restrict__ Ac, int* __restrict__ err) {
  const int64_t n = (int64_t)blockIdx.x * NT + threadIdx.x;
  const int64_t nrows = (int64_t)gc.nn[0] * gc.nn[1] * gc.nn[2];
  if (n >= nrows) return;
  int I[3];
  decompose(gc, n, I[0], I[1], I[2]);
  const RowInfo Rc = row_info_p3(gc, pc, I[0], I[1], I[2]);
  const int lenc = Rc.cx * Rc.cy * Rc.cz;
  T* out = Ac + Rc.rp;
  if (node_fixed(gc, I[0], I[1], I[2])) {
    const int dg = (int)(diag_pos(Rc, I[0], I[1], I[2]) - Rc.rp);
    for (int e = 0; e < lenc; ++e) out[e] = (e == dg) ? T(1) : T(0);
    return;
  }
  constexpr int MAXROW = 75;  // 3 x 5 x 5: the widest output row (one axis swept from a Q2 grid)
  if (lenc > MAXROW) { atomicExch(err, 1); return; }
  T acc[MAXROW];
  for (int e = 0; e < lenc; ++e) acc[e] = T(0);
  int ci[3];
  float cw[3];
  const int nci = axis_children(I[axis], gf.nn[axis], gc.nn[axis], 1, ci, cw);
  for (int c = 0; c < nci; ++c) {
    int f[3] = {I[0], I[1], I[2]};
    f[axis] = ci[c];
    if (node_fixed(gf, f[0], f[1], f[2])) continue;
    const RowInfo Rf = row_info_p3(gf, pf, f[0], f[1], f[2]);
    const T* vals = Af + Rf.rp;
    int e = 0;
    for (int jz = Rf.lz; jz < Rf.lz + Rf.cz; ++jz)
      for (int jy = Rf.ly; jy < Rf.ly + Rf.cy; ++jy)
        for (int jx = Rf.lx; jx < Rf.lx + Rf.cx; ++jx, ++e) {
          if (node_fixed(gf, jx, jy, jz)) continue;
          const T a = vals[e] * (T)cw[c];
          int jj[3] = {jx, jy, jz};
          int pc[2];
          float pw[2];
          const int np = axis_parents(jj[axis], gf.nn[axis], gc.nn[axis], 1, pc, pw);
          for (int k = 0; k < np; ++k) {
            jj[axis] = pc[k];
            if (node_fixed(gc, jj[0], jj[1], jj[2])) continue;
            const int pos = ((jj[2] - Rc.lz) * Rc.cy + (jj[1] - Rc.ly)) * Rc.cx + (jj[0] - Rc.lx);
            if (pos < 0 || pos >= lenc) { atomicExch(err, 1); continue; }
            acc[pos] += a * (T)pw[k];
          }
        }
  }
  for (int e = 0; e < lenc; ++e) out[e] = acc[e];
}

// The sweep of the 3-D h-levels (order 1 throughout), one warp per 32 output rows of a grid line.  The children's rows
// are consecutive in CSR (axis 0: the fine rows 2 x0 - 1 .. 2 x1 + 1 of the line; otherwise 32 rows of each of the three
// child lines), so the warp copies them into its shared buffer with consecutive lanes on consecutive addresses, each
// lane works on its row there, and the output rows leave the same way.  Read and written row by row from global memory
// the first sweep of a 97^3 grid took 239 us (every load instruction on 32 lines).
__device__ __forceinline__ bool col_at(const bool (&col)[5], int s) { return s < -2 || s > 2 ? false : col[s + 2]; }

constexpr int RAP_W = 4;             // warps per CTA
constexpr int RAP_BUF = 3 * 32 * 27;  // the longest copy: three lines of 32 rows (axis 0: 65 rows)
template <typename T>
constexpr int rap_smem() { return RAP_W * RAP_BUF * (int)sizeof(T); }
template <typename T, int A>
__global__ void __launch_bounds__(RAP_W * 32) k_rap_line(Grid gf, Grid gc, int tiles, int64_t ntile,
                                                         const T* __restrict__ Af, T* __restrict__ Ac) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* buf = reinterpret_cast<T*>(smem_raw) + (threadIdx.x >> 5) * RAP_BUF;
  const int lane = threadIdx.x & 31;
  const int64_t tile = (int64_t)blockIdx.x * RAP_W + (threadIdx.x >> 5);
  if (tile >= ntile) return;  // uniform over the warp
  const int64_t line = tile / tiles;
  const int x0 = (int)(tile - line * tiles) * 32, x1 = min(x0 + 32, gc.nn[0]) - 1;
  int I[3] = {min(x0 + lane, x1), (int)(line % gc.nn[1]), (int)(line / gc.nn[1])};
  const bool on = x0 + lane <= x1;
  int fixed_at = -1;  // a Dirichlet row: its diagonal's position
  // the children's rows: shared offset of the first row of each copied segment
  const int clo = A == 0 ? 0 : max(2 * I[A] - 1, 0), chi = A == 0 ? 0 : min(2 * I[A] + 1, gf.nn[A] - 1);
  int64_t seg[3];
  int at[3], used = 0;
#pragma unroll
  for (int c = 0; c < (A == 0 ? 1 : 3); ++c) {
    int f0[3] = {x0, I[1], I[2]}, f1[3] = {x1, I[1], I[2]};
    if (A == 0) {
      f0[0] = max(2 * x0 - 1, 0);
      f1[0] = min(2 * x1 + 1, gf.nn[0] - 1);
    } else {
      if (clo + c > chi) break;
      f0[A] = f1[A] = clo + c;
    }
    const RowInfo R0 = row_info<1>(gf, f0[0], f0[1], f0[2]), R1 = row_info<1>(gf, f1[0], f1[1], f1[2]);
    const int n = (int)(R1.rp + R1.cx * R1.cy * R1.cz - R0.rp);
    seg[c] = R0.rp;
    at[c] = used;
#pragma unroll 8
    for (int k = lane; k < n; k += 32) buf[used + k] = __ldg(Af + R0.rp + k);
    used += n;
  }
  __syncwarp();
  const RowInfo Rc = row_info<1>(gc, I[0], I[1], I[2]);
  const int lenc = Rc.cx * Rc.cy * Rc.cz;
  T acc[27];
#pragma unroll
  for (int k = 0; k < 27; ++k) acc[k] = T(0);
  auto fine = [&](int f, int64_t rp) {  // values of the fine row at coordinate f along A
    if constexpr (A == 0) return buf + (rp - seg[0]);
    else {
      const int c = f - clo;
      return c == 0 ? buf + at[0] + (rp - seg[0]) : (c == 1 ? buf + at[1] + (rp - seg[1]) : buf + at[2] + (rp - seg[2]));
    }
  };
  if (on) {
    if (node_fixed(gc, I[0], I[1], I[2])) {
      const int dg = (int)(diag_pos(Rc, I[0], I[1], I[2]) - Rc.rp);
      fixed_at = dg;
    } else {
      // fine columns along A relative to 2 I: they exist, are free, and go to free coarse columns with these weights
      float plo[5], phi[5];
      bool col[5];
#pragma unroll
      for (int s = -2; s <= 2; ++s) {
        const int f = 2 * I[A] + s, p0 = I[A] + (s >= 0 ? s / 2 : -((1 - s) / 2));
        col[s + 2] = f >= 0 && f < gf.nn[A] && axis_free(gf, A, f);
        plo[s + 2] = phi[s + 2] = 0.0f;
        if (s & 1) {
          const bool last = f == gf.nn[A] - 1;  // an odd last node is kept: its parent is the last coarse node, weight 1
          if (p0 >= 0 && !last && axis_free(gc, A, p0)) plo[s + 2] = 0.5f;
          if (p0 + 1 < gc.nn[A] && axis_free(gc, A, p0 + 1)) phi[s + 2] = last ? 1.0f : 0.5f;
        } else if (p0 >= 0 && p0 < gc.nn[A] && axis_free(gc, A, p0)) {
          plo[s + 2] = 1.0f;
        }
      }
      bool m[3][3];
      int lo[3];
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        lo[b] = I[b] > 0 ? 1 : 0;
#pragma unroll
        for (int e = -1; e <= 1; ++e) m[b][e + 1] = I[b] + e >= 0 && I[b] + e < gf.nn[b] && axis_free(gf, b, I[b] + e);
      }
      auto child = [&](auto dc_tag) {
        constexpr int DC = decltype(dc_tag)::value;
        int f[3] = {I[0], I[1], I[2]};
        f[A] = 2 * I[A] + DC;
        // the child exists, is free and has this row among its parents
        const float wc = DC == 0 ? plo[2] : (DC < 0 ? phi[1] : plo[3]);
        if (!col[DC + 2] || wc == 0.0f) return;
        lo[A] = f[A] > 0 ? 1 : 0;
#pragma unroll
        for (int e = -1; e <= 1; ++e) m[A][e + 1] = col_at(col, DC + e);
        const RowInfo R = row_info<1>(gf, f[0], f[1], f[2]);
        rap_child<T, A, DC>(fine(f[A], R.rp), R, lo, m, plo, phi, (T)wc, acc);
      };
      child(std::integral_constant<int, -1>{});
      child(std::integral_constant<int, 0>{});
      child(std::integral_constant<int, 1>{});
    }
  }
  __syncwarp();
  // the output rows are one segment of CSR
  const int64_t out0 = __shfl_sync(0xffffffffu, Rc.rp, 0);
  const int total = (int)(__shfl_sync(0xffffffffu, Rc.rp + lenc, x1 - x0) - out0);
  T* mine = buf + (Rc.rp - out0);
  if (on && fixed_at >= 0) {
    for (int e = 0; e < lenc; ++e) mine[e] = e == fixed_at ? T(1) : T(0);
  } else if (on) {
#pragma unroll
    for (int e = 0; e < 27; ++e) {  // the couplings the row has, in storage order
      const int x = I[0] + e % 3 - 1, y = I[1] + e / 3 % 3 - 1, z = I[2] + e / 9 - 1;
      if (x >= 0 && x < gc.nn[0] && y >= 0 && y < gc.nn[1] && z >= 0 && z < gc.nn[2])
        mine[((z - Rc.lz) * Rc.cy + (y - Rc.ly)) * Rc.cx + (x - Rc.lx)] = acc[e];
    }
  }
  __syncwarp();
  for (int k = lane; k < total; k += 32) Ac[out0 + k] = buf[k];
}

// The same sweep with one warp per output row and the lanes over the row's entries: an entry sums, over
// the children c of the row and the fine columns j whose parent is the entry's column, a_c(j) w_c w_j --
// the row loop above adds exactly these products, in the same order (children ascending, then fine
// columns ascending), so the result is bit-identical.  Used on small levels (below ~25k output rows),
// where one thread's serial walk over a row set the duration of the thread-per-row loop (42 µs for a
// 128-row level against 8 µs here); above that the thread-per-row fast path is faster.
// Children of coarse node c along a coarsened axis in three fixed slots (fine 2c-1, 2c, 2c+1): the
// same set, order and weights as axis_children, without its run-time slot index.
__device__ __forceinline__ void children3(int c, int nnf, int nnc, int ci[3], float cw[3], bool ok[3]) {
  ci[0] = 2 * c - 1;
  ci[1] = 2 * c;
  ci[2] = 2 * c + 1;
  // 2c-1 (odd): parents (i-1)/2, (i+1)/2 = c with weight 1/2, or the kept odd last node (parent nnc-1, 1)
  ok[0] = c >= 1 && ci[0] <= nnf - 1 && (ci[0] != nnf - 1 || c == nnc - 1);
  cw[0] = (ci[0] == nnf - 1) ? 1.0f : 0.5f;
  ok[1] = ci[1] <= nnf - 1;  // even: parent c, weight 1
  cw[1] = 1.0f;
  ok[2] = ci[2] <= nnf - 2;  // odd, not the last node: parents c and c+1, weight 1/2
  cw[2] = 0.5f;
}

template <typename T, int A>
__global__ void __launch_bounds__(NT) k_rap_axis_w(Grid gf, P3 pf, Grid gc, P3 pc, const T* __restrict__ Af,
                                                   T* __restrict__ Ac) {
  const int lane = threadIdx.x & 31;
  const int64_t n = ((int64_t)blockIdx.x * NT + threadIdx.x) >> 5;
  const int64_t nrows = (int64_t)gc.nn[0] * gc.nn[1] * gc.nn[2];
  if (n >= nrows) return;  // uniform over the warp
  int I[3];
  decompose(gc, n, I[0], I[1], I[2]);
  const RowInfo Rc = row_info_p3(gc, pc, I[0], I[1], I[2]);
  const int lenc = Rc.cx * Rc.cy * Rc.cz;
  T* out = Ac + Rc.rp;
  if (node_fixed(gc, I[0], I[1], I[2])) {
    const int dg = (int)(diag_pos(Rc, I[0], I[1], I[2]) - Rc.rp);
    for (int e = lane; e < lenc; e += 32) out[e] = (e == dg) ? T(1) : T(0);
    return;
  }
  const int nnf = gf.nn[A], nnc = gc.nn[A];
  int ci[3];
  float cw[3];
  bool cok[3];
  children3(I[A], nnf, nnc, ci, cw, cok);
  RowInfo Rf[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    int f[3] = {I[0], I[1], I[2]};
    f[A] = ci[c];
    cok[c] = cok[c] && !node_fixed(gf, f[0], f[1], f[2]);
    if (cok[c]) Rf[c] = row_info_p3(gf, pf, f[0], f[1], f[2]);
  }
  for (int e = lane; e < lenc; e += 32) {
    int o[3];
    o[0] = Rc.lx + e % Rc.cx;
    o[1] = Rc.ly + (e / Rc.cx) % Rc.cy;
    o[2] = Rc.lz + e / (Rc.cx * Rc.cy);
    T acc = T(0);
    if (!node_fixed(gc, o[0], o[1], o[2])) {
      int cj[3];
      float wj[3];
      bool jok[3];
      children3(o[A], nnf, nnc, cj, wj, jok);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        if (!cok[c]) continue;
        const RowInfo& R = Rf[c];
        const T* vals = Af + R.rp;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          if (!jok[k]) continue;
          int j[3] = {o[0], o[1], o[2]};
          j[A] = cj[k];
          if (j[0] < R.lx || j[0] >= R.lx + R.cx || j[1] < R.ly || j[1] >= R.ly + R.cy || j[2] < R.lz ||
              j[2] >= R.lz + R.cz)
            continue;
          if (node_fixed(gf, j[0], j[1], j[2])) continue;
          const T a = vals[((j[2] - R.lz) * R.cy + (j[1] - R.ly)) * R.cx + (j[0] - R.lx)] * (T)cw[c];
          acc += a * (T)wj[k];
        }
      }
    }
    out[e] = acc;
  }
}

// minv = 1 / diag; Gershgorin bound max_i sum_j |a_ij| / |a_ii| into lmax (as float bits, atomicMax)
template <int P, typename T>
__global__ void __launch_bounds__(NT, staged_per_sm<T>()) k_diag(Grid g, const T* __restrict__ A, T* __restrict__ minv,
                                                                 unsigned int* __restrict__ lmax_bits, int* __restrict__ err) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t mbar[2 * (NT / 32)];
  const int64_t nrows = (int64_t)g.nn[0] * g.nn[1] * g.nn[2];
  float v = 0.0f;
  const bool ok = level_rows<P, T>(
      g, nrows, A, smem_raw, mbar,
      [&](int64_t n, const RowInfo& R, const T* vals) {
        int ix, iy, iz;
        decompose(g, n, ix, iy, iz);
        const int len = R.cx * R.cy * R.cz;
        const T dgv = vals[diag_pos(R, ix, iy, iz) - R.rp];
        T s = T(0);  // a bound: the level's precision is enough
        for (int e = 0; e < len; ++e) s += fabs(vals[e]);
        minv[n] = T(1) / dgv;
        v = fmaxf(v, (float)(s / fabs(dgv)));
      },
      AlwaysGo{});
  if (!ok) atomicExch(err, 3);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_down_sync(0xffffffffu, v, o));
  if ((threadIdx.x & 31) == 0 && v > 0.0f) atomicMax(lmax_bits, __float_as_uint(v));
}

// Dense inverse of the coarsest operator (n <= MAXC), Gauss-Jordan with partial pivoting, one CTA, in
// the hierarchy's precision (FP32 for the inner solve's hierarchy: FP64 arithmetic there cost the FP64
// pipe's latency on every step for a preconditioner that is FP32 anyway).  The pivot is the first row
// of largest magnitude, found by warp 0 with shuffles.
// A thread owns one column (of MAXC + n) of two rows, so a pivot step is three barriers and no index arithmetic (with
// 128 threads walking the elements a step took 2.2 us).
constexpr int IT = 1024;
template <typename T>
__global__ void __launch_bounds__(IT) k_coarse_inv(Grid g, const T* __restrict__ A, T* __restrict__ inv,
                                                   int* __restrict__ err) {
  __shared__ T M[MAXC][2 * MAXC];  // [A | inverse]; the inverse begins at column MAXC
  __shared__ int piv;
  const int n = g.nn[0] * g.nn[1] * g.nn[2];
  for (int k = threadIdx.x; k < MAXC * 2 * MAXC; k += IT) (&M[0][0])[k] = T(0);
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += IT) {
    int ix, iy, iz;
    decompose(g, i, ix, iy, iz);
    const RowInfo R = row_info<1>(g, ix, iy, iz);
    int e = 0;
    for (int jz = R.lz; jz < R.lz + R.cz; ++jz)
      for (int jy = R.ly; jy < R.ly + R.cy; ++jy)
        for (int jx = R.lx; jx < R.lx + R.cx; ++jx, ++e)
          M[i][jx + g.nn[0] * (jy + g.nn[1] * jz)] = A[R.rp + e];
    M[i][MAXC + i] = T(1);
  }
  __syncthreads();
  const int k = threadIdx.x & (2 * MAXC - 1), r0 = threadIdx.x / (2 * MAXC);
  constexpr int RS = IT / (2 * MAXC);  // rows per pass
  for (int c = 0; c < n; ++c) {
    if (threadIdx.x < 32) {
      const int r = threadIdx.x;
      T v = (r >= c && r < n) ? fabs(M[r][c]) : T(-1);
      int bi = r;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const T ov = __shfl_down_sync(0xffffffffu, v, o);
        const int oi = __shfl_down_sync(0xffffffffu, bi, o);
        if (ov > v || (ov == v && oi < bi)) {
          v = ov;
          bi = oi;
        }
      }
      if (threadIdx.x == 0) {
        piv = bi;
        if (!(v > T(0))) atomicExch(err, 2);
      }
    }
    __syncthreads();
    // rows c and pr change places; row c is scaled, column c leaves the other rows
    const int pr = piv;
    const T pk = M[pr][k] * (T(1) / M[pr][c]), qk = M[c][k], qc = M[c][c];
    T out[MAXC / RS];
#pragma unroll
    for (int j = 0; j < MAXC / RS; ++j) {
      const int r = r0 + j * RS;
      const T f = r == pr ? qc : M[r][c], v = r == pr ? qk : M[r][k];
      out[j] = r == c ? pk : (k == c ? T(0) : v - f * pk);
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < MAXC / RS; ++j) M[r0 + j * RS][k] = out[j];
    __syncthreads();
  }
  for (int idx = threadIdx.x; idx < n * n; idx += IT) inv[idx] = M[idx / n][MAXC + idx % n];
}

// Chebyshev coefficients of every level and step (one thread per level, at setup): coef[(l NU + k) 3 + m]
// = {1/theta, rho_k rho_{k-1}, 2 rho_k / delta} on [CHEB_LO L, L], L the level's Gershgorin bound.
// in the levels' precision: converted once here, not by every thread that uses them (a conversion takes the FP64 pipe).
template <typename T>
__global__ void k_cheb_coef(const unsigned int* __restrict__ lmax_bits, int nlev, T* __restrict__ coef) {
  const int l = threadIdx.x;
  if (l >= nlev) return;
  const double hi = (double)__uint_as_float(lmax_bits[l]), lo = CHEB_LO * hi;
  const double theta = 0.5 * (hi + lo), delta = 0.5 * (hi - lo), sigma = theta / delta;
  double rho_prev = 1.0 / sigma, rho = rho_prev;
  for (int k = 0; k < NU; ++k) {
    if (k > 0) {
      const double rn = 1.0 / (2.0 * sigma - rho);
      rho_prev = rho;
      rho = rn;
    }
    T* c = coef + ((size_t)l * NU + k) * 3;
    c[0] = 1.0 / theta;
    c[1] = rho * rho_prev;
    c[2] = 2.0 * rho / delta;
  }
}

// Rounded operations that the compiler does not contract: the row updates shared by the per-step kernels
// and k_vcycle_tail must round the same way in both.
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float sub_rn(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ double sub_rn(double a, double b) { return __dsub_rn(a, b); }

// Chebyshev-Jacobi step k for row n given ax = (A x_in)_n: d = c_first z (k = 0) or c_old d + c_new z with
// z = D^{-1} (b - ax); x_out = x_in + d (x_in = 0 when zero_x).  Shared by k_cheb and k_vcycle_tail.
template <typename T>
__device__ __forceinline__ void cheb_row(const LevDev<T>& L, int64_t n, T ax, const T* xin,
                                         T* xout, int k, int zero_x, T c_first, T c_old, T c_new) {
  const T z = mul_rn(L.minv[n], sub_rn(L.b[n], ax));
  const T d = (k == 0) ? mul_rn(c_first, z) : fma(c_old, L.d[n], mul_rn(c_new, z));
  L.d[n] = d;
  xout[n] = add_rn(zero_x ? T(0) : xin[n], d);
}
// Step 0 from x = 0, taken by the kernel that writes b: a launch and a pass over b less for each level of a cycle.  coef is
// null where the cycle does not smooth (coarsest level, levels of k_vcycle_tail).
template <typename T>
struct FirstStep {
  const T *coef, *minv;
  T *d, *xa;
  __device__ __forceinline__ T diag(int64_t n) const { return coef ? minv[n] : T(0); }  // to be in flight with b's terms
  __device__ __forceinline__ void operator()(int64_t n, T b, T mi) const {
    if (!coef) return;
    const T v = mul_rn(coef[0], mul_rn(mi, b));
    d[n] = v;
    xa[n] = add_rn(T(0), v);
  }
};

// r = b - A x, row n
template <typename T>
__device__ __forceinline__ void resid_row(const LevDev<T>& L, int64_t n, T ax) {
  L.r[n] = sub_rn(L.b[n], ax);
}

template <int P, typename T>
__global__ void __launch_bounds__(NT, staged_per_sm<T>()) k_cheb(LevDev<T> L, const T* xin, T* xout, int k,
                                             int zero_x, const T* __restrict__ coef,
                                             const GScal* __restrict__ S, int* __restrict__ err) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t mbar[2 * (NT / 32)];
  pdl_trigger();
  const T c_first = coef[3 * k], c_old = coef[3 * k + 1], c_new = coef[3 * k + 2];
  auto fin = [&](int64_t n, T ax) { cheb_row<T>(L, n, ax, xin, xout, k, zero_x, c_first, c_old, c_new); };
  if (zero_x) {
    pdl_wait();
    if (is_done(S)) return;
    for (int64_t n = (int64_t)blockIdx.x * NT + threadIdx.x; n < L.n; n += (int64_t)gridDim.x * NT) fin(n, T(0));
    return;
  }
  const bool ok = level_rows<P, T>(
      L.g, L.n, L.A, smem_raw, mbar,
      [&](int64_t n, const RowInfo& R, const T* vals) { fin(n, (T)row_prod<P, T>(L.g, R, vals, xin)); },
      [&] { pdl_wait(); return !is_done(S); });
  if (!ok) atomicExch(err, 3);
}

// r = b - A x
template <int P, typename T>
__global__ void __launch_bounds__(NT, staged_per_sm<T>()) k_resid(LevDev<T> L, const T* x, const GScal* __restrict__ S,
                                              int* __restrict__ err) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t mbar[2 * (NT / 32)];
  pdl_trigger();
  const bool ok = level_rows<P, T>(
      L.g, L.n, L.A, smem_raw, mbar,
      [&](int64_t n, const RowInfo& R, const T* vals) { resid_row<T>(L, n, (T)row_prod<P, T>(L.g, R, vals, x)); },
      [&] { pdl_wait(); return !is_done(S); });
  if (!ok) atomicExch(err, 3);
}

// b_c = P^T r_f
// Per-axis transfer slots with validity flags (registers, no run-time indexed arrays): children of a
// coarse node (fine 2c-1, 2c, 2c+1 on a coarsened axis, the node itself otherwise) and parents of a
// fine node (1 or 2).  Same sets, order and weights as axis_children / axis_parents.
__device__ __forceinline__ void child_slots(int c, int nnf, int nnc, int co, bool in_dim, int ci[3], float cw[3],
                                            bool ok[3]) {
  if (!in_dim) {
    ci[0] = ci[1] = ci[2] = 0;
    cw[0] = cw[1] = cw[2] = 1.0f;
    ok[0] = ok[2] = false;
    ok[1] = true;
    return;
  }
  if (!co) {
    ci[0] = ci[1] = ci[2] = c;
    cw[0] = cw[1] = cw[2] = 1.0f;
    ok[0] = ok[2] = false;
    ok[1] = true;
    return;
  }
  children3(c, nnf, nnc, ci, cw, ok);
}

__device__ __forceinline__ void parent_slots(int i, int nnf, int nnc, int co, bool in_dim, int pc[2], float pw[2],
                                             bool ok[2]) {
  if (!in_dim) {
    pc[0] = pc[1] = 0;
    pw[0] = pw[1] = 1.0f;
    ok[0] = true;
    ok[1] = false;
    return;
  }
  const int np = axis_parents(i, nnf, nnc, co, pc, pw);
  ok[0] = true;
  ok[1] = np == 2;
  if (np < 2) {
    pc[1] = pc[0];
    pw[1] = 0.0f;
  }
}

// b_c = P^T r_f, coarse row n (shared by k_restrict and k_vcycle_tail)
// The free nodes are a Cartesian product, so a child counts if it exists and is free along each axis; the others are
// loaded as zeros (no branches: the lanes of a warp have children missing at different places).
template <typename T>
__device__ __forceinline__ T restrict_row(const Grid& gf, const Grid& gc, const Xfer& X, const T* rf, int64_t n) {
  int I[3];
  decompose(gc, n, I[0], I[1], I[2]);
  if (node_fixed(gc, I[0], I[1], I[2])) return T(0);
  int c[3][3];
  float w[3][3];
  bool k[3][3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    child_slots(I[a], gf.nn[a], gc.nn[a], X.co[a], gf.dim > a, c[a], w[a], k[a]);
#pragma unroll
    for (int e = 0; e < 3; ++e) k[a][e] = k[a][e] && axis_free(gf, a, c[a][e]);
  }
  const int NX = gf.nn[0];
  const int64_t plane = (int64_t)NX * gf.nn[1];
  T s = T(0);
#pragma unroll
  for (int a2 = 0; a2 < 3; ++a2)
#pragma unroll
    for (int a1 = 0; a1 < 3; ++a1) {
      const T* r = rf + NX * c[1][a1] + plane * c[2][a2];
      const float w12 = w[1][a1] * w[2][a2];
#pragma unroll
      for (int a0 = 0; a0 < 3; ++a0) {
        const bool in = k[2][a2] && k[1][a1] && k[0][a0];
        s = fma((T)(w[0][a0] * w12), in ? r[c[0][a0]] : T(0), s);  // the weights are powers of two
      }
    }
  return s;
}

// and the coarse level's first smoothing step
template <typename T>
__global__ void __launch_bounds__(NT) k_restrict(Grid gf, Grid gc, Xfer X, const T* rf, T* bc,
                                                 FirstStep<T> first, const GScal* __restrict__ S) {
  pdl_trigger();
  pdl_wait();
  if (is_done(S)) return;
  const int64_t nc = (int64_t)gc.nn[0] * gc.nn[1] * gc.nn[2];
  for (int64_t n = (int64_t)blockIdx.x * NT + threadIdx.x; n < nc; n += (int64_t)gridDim.x * NT) {
    const T mi = first.diag(n), b = restrict_row<T>(gf, gc, X, rf, n);
    bc[n] = b;
    first(n, b, mi);
  }
}

// x_f += P x_c, fine row n (k_vcycle_tail; k_prolong takes two rows at once)
template <typename T>
__device__ __forceinline__ void prolong_row(const Grid& gf, const Grid& gc, const Xfer& X, const T* xc,
                                            T* xf, int64_t n) {
  int i[3];
  decompose(gf, n, i[0], i[1], i[2]);
  if (node_fixed(gf, i[0], i[1], i[2])) return;
  int p[3][2];
  float w[3][2];
  bool k[3][2];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    parent_slots(i[a], gf.nn[a], gc.nn[a], X.co[a], gf.dim > a, p[a], w[a], k[a]);
#pragma unroll
    for (int e = 0; e < 2; ++e) k[a][e] = k[a][e] && axis_free(gc, a, p[a][e]);
  }
  const int NX = gc.nn[0];
  const int64_t plane = (int64_t)NX * gc.nn[1];
  T s = T(0);
#pragma unroll
  for (int b2 = 0; b2 < 2; ++b2)
#pragma unroll
    for (int b1 = 0; b1 < 2; ++b1) {
      const T* r = xc + NX * p[1][b1] + plane * p[2][b2];
      const float w12 = w[1][b1] * w[2][b2];
#pragma unroll
      for (int b0 = 0; b0 < 2; ++b0) {
        const bool in = k[2][b2] && k[1][b1] && k[0][b0];
        s = fma((T)(w[0][b0] * w12), in ? r[p[0][b0]] : T(0), s);
      }
    }
  xf[n] = add_rn(xf[n], s);
}

// FP32: two neighbours along x a thread (nodes 2 j and 2 j + 1).  Their parents are the nodes j and j + 1 (2 j and 2 j + 1
// where x is not coarsened), so 8 loads and one set of index arithmetic serve two rows (97^3 nodes: 14.2 -> 9.2 us).
// Terms in prolong_row's order; those it multiplies by a weight of 0 are left out.  FP64: a row a thread; pairs halve the
// warps that the FP64 pipe's latency is hidden behind (Newton solves on 48^3 cells with pairs 2 % slower).
template <typename T>
__global__ void __launch_bounds__(NT) k_prolong(Grid gf, Grid gc, Xfer X, const T* xc, T* xf,
                                                const GScal* __restrict__ S) {
  pdl_trigger();
  pdl_wait();
  if (is_done(S)) return;
  if constexpr (sizeof(T) == 8) {
    const int64_t nf = (int64_t)gf.nn[0] * gf.nn[1] * gf.nn[2];
    for (int64_t n = (int64_t)blockIdx.x * NT + threadIdx.x; n < nf; n += (int64_t)gridDim.x * NT)
      prolong_row<T>(gf, gc, X, xc, xf, n);
    return;
  }
  const unsigned NXF = (unsigned)gf.nn[0], pairs = (NXF + 1) / 2, NY = (unsigned)gf.nn[1];
  const unsigned np = pairs * NY * (unsigned)gf.nn[2];  // at most the number of rows, which is at most INT32_MAX
  const int NX = gc.nn[0];
  const int64_t plane = (int64_t)NX * gc.nn[1];
  for (unsigned m = blockIdx.x * NT + threadIdx.x; m < np; m += gridDim.x * NT) {
    const unsigned line = m / pairs, j = m - line * pairs;
    const int i0 = 2 * (int)j, i[3] = {i0, (int)(line % NY), (int)(line / NY)};
    int p[3][2], p1[2];
    float w[3][2], w1[2];
    bool k[3][2], k1[2];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      parent_slots(i[a], gf.nn[a], gc.nn[a], X.co[a], gf.dim > a, p[a], w[a], k[a]);
#pragma unroll
      for (int e = 0; e < 2; ++e) k[a][e] = k[a][e] && axis_free(gc, a, p[a][e]);
    }
    const bool second = i0 + 1 < (int)NXF;
    parent_slots(min(i0 + 1, (int)NXF - 1), gf.nn[0], gc.nn[0], X.co[0], true, p1, w1, k1);
#pragma unroll
    for (int e = 0; e < 2; ++e) k1[e] = k1[e] && axis_free(gc, 0, p1[e]);
    const int b0 = p[0][0], b1 = min(b0 + 1, NX - 1);  // parents of both
    const bool f0 = axis_free(gc, 0, b0), f1 = axis_free(gc, 0, b1);
    T s0 = T(0), s1 = T(0);
#pragma unroll
    for (int e2 = 0; e2 < 2; ++e2)
#pragma unroll
      for (int e1 = 0; e1 < 2; ++e1) {
        const T* r = xc + NX * p[1][e1] + plane * p[2][e2];
        const float w12 = w[1][e1] * w[2][e2];
        const bool in = k[2][e2] && k[1][e1];
        const T t0 = in && f0 ? r[b0] : T(0), t1 = in && f1 ? r[b1] : T(0);
        s0 = fma((T)(w[0][0] * w12), t0, s0);
        s1 = fma((T)(w1[0] * w12), k1[0] ? (p1[0] == b0 ? t0 : t1) : T(0), s1);
        s1 = fma((T)(w1[1] * w12), k1[1] ? t1 : T(0), s1);
      }
    const bool fr = !node_fixed(gf, i0, i[1], i[2]), fr1 = second && !node_fixed(gf, i0 + 1, i[1], i[2]);
    T* x = xf + (int64_t)line * NXF + i0;
    const T v0 = fr ? x[0] : T(0), v1 = fr1 ? x[1] : T(0);
    if (fr) x[0] = add_rn(v0, s0);
    if (fr1) x[1] = add_rn(v1, s1);
  }
}

// x = inv b on the coarsest level, row i (shared by k_coarse_apply and k_vcycle_tail)
template <typename T>
__device__ __forceinline__ void coarse_row(int n, const T* __restrict__ inv, const T* b, T* x,
                                           int i) {
  T s = T(0);
  for (int j = 0; j < n; ++j) s = fma(inv[i * n + j], b[j], s);
  x[i] = s;
}

template <typename T>
__global__ void __launch_bounds__(NT) k_coarse_apply(int n, const T* __restrict__ inv, const T* b,
                                                     T* x, const GScal* __restrict__ S) {
  pdl_trigger();
  pdl_wait();
  if (is_done(S)) return;
  for (int i = threadIdx.x; i < n; i += NT) coarse_row<T>(n, inv, b, x, i);
}

// ---- the coarse end of the V-cycle in one CTA ---------------------------------------------------------
// The smallest levels take a microsecond of work per step but a launch each (seven per level and cycle).
// k_vcycle_tail runs the whole cycle below the first such level -- pre-smoothing, residual and restriction
// down to the coarsest level, the dense coarsest solve, prolongation and post-smoothing back up -- in one
// CTA, with a CTA barrier between steps.  What bounds it is the chain of steps, so everything they touch is in
// shared memory: the levels' operators and diagonals are copied there before the kernel waits for its predecessor
// (no kernel of a solve writes them), the vectors live there, and each row's start and extents are worked out once.
// From global memory, with the row decoding at every step, the tail of a 97^3 hierarchy (7^3 nodes) took 42 us.  Every
// row's arithmetic is that of the per-step kernels, in the same order, so the result is bit-identical
// (MRG_PREC_GMG_SPLIT keeps the per-step launches for comparison).
constexpr int TT = 1024;               // threads of the tail CTA
constexpr int MAXTAIL = 8;             // levels the tail can hold
constexpr int64_t TAIL_ROWS32 = 1024;  // FP32: first level taken into the tail has at most this many rows
constexpr size_t TAIL_SMEM = 200 * 1024;
// A level's sweep in one SM must cost less than the launches it replaces.  FP64 takes no tail: its pipe (1/64 of the
// FP32 rate) makes a single-SM sweep of a 729-row level as long as a launch.
template <typename T>
constexpr int64_t tail_rows() { return sizeof(T) == 4 ? TAIL_ROWS32 : 0; }

template <typename T>
struct TailArgs {
  int nlev = 0;                  // levels in the tail; the last is the coarsest
  LevDev<T> L[MAXTAIL];
  Xfer X[MAXTAIL];               // X[j]: how tail level j was coarsened from level j - 1
  const T* coef[MAXTAIL];        // Chebyshev coefficients of each level
  const T* cinv = nullptr;       // dense inverse of the coarsest operator
};

// shared memory of one smoothed level: row records, operator, 1/diag and five vectors
template <typename T>
__host__ __device__ inline size_t tail_level_bytes(const Grid& g, int64_t n) {
  const size_t nnz = (size_t)(g.T[0] * g.T[1] * g.T[2]);
  return (size_t)n * sizeof(int4) + (((nnz + 6 * (size_t)n) * sizeof(T) + 15) & ~(size_t)15);
}
template <typename T>
inline size_t tail_smem(const TailArgs<T>& A) {
  size_t b = 0;
  for (int j = 0; j + 1 < A.nlev; ++j) b += tail_level_bytes<T>(A.L[j].g, A.L[j].n);
  const size_t n = (size_t)A.L[A.nlev - 1].n;
  return b + n * (n + 2) * sizeof(T);
}

// a level in shared memory; LevDev with row records
template <typename T>
struct TailLev {
  LevDev<T> D;
  const int4* row;  // start in A, first coupled node, extents cx | cy << 2 | cz << 4
};

template <typename T>
__device__ __forceinline__ T tail_prod(const TailLev<T>& L, int n, const T* x) {
  const int4 q = L.row[n];
  const T* a = L.D.A + q.x;
  const T* xb = x + q.y;
  const int NX = L.D.g.nn[0], plane = NX * L.D.g.nn[1];
  T acc = T(0);
  if (q.z == (3 | 3 << 2 | 3 << 4)) {
#pragma unroll
    for (int k = 0; k < 27; ++k) acc = fma(a[k], xb[(k % 3) + NX * ((k / 3) % 3) + plane * (k / 9)], acc);
    return acc;
  }
  const int cx = q.z & 3, cy = (q.z >> 2) & 3, cz = q.z >> 4;
  int pos = 0;
#pragma unroll
  for (int z = 0; z < 3; ++z)
    if (z < cz)
#pragma unroll
      for (int y = 0; y < 3; ++y)
        if (y < cy)
#pragma unroll
          for (int i = 0; i < 3; ++i)
            if (i < cx) acc = fma(a[pos++], xb[i + NX * y + plane * z], acc);
  return acc;
}

template <typename T>
__device__ __forceinline__ void tail_cheb(const TailLev<T>& L, const T* xin, T* xout, int k, int zero_x,
                                          const T* __restrict__ coef) {
  const T c_first = coef[3 * k], c_old = coef[3 * k + 1], c_new = coef[3 * k + 2];
  for (int n = threadIdx.x; n < (int)L.D.n; n += TT)
    cheb_row<T>(L.D, n, zero_x ? T(0) : tail_prod<T>(L, n, xin), xin, xout, k, zero_x, c_first, c_old, c_new);
  __syncthreads();
}

template <typename T>
__global__ void __launch_bounds__(TT) k_vcycle_tail(const __grid_constant__ TailArgs<T> A, const GScal* __restrict__ S) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ TailLev<T> lev[MAXTAIL];
  pdl_trigger();
  const int nl = A.nlev;
  {
    unsigned char* at = smem_raw;
    for (int j = 0; j < nl; ++j) {
      const LevDev<T>& G = A.L[j];
      const int n = (int)G.n;
      TailLev<T> L;
      L.D = G;
      if (j == nl - 1) {  // coarsest: inverse, right-hand side, solution
        T* v = reinterpret_cast<T*>(at);
        for (int k = threadIdx.x; k < n * n; k += TT) v[k] = A.cinv[k];
        L.D.A = v;
        L.D.b = v + n * n;
        L.D.xb = L.D.b + n;
        L.row = nullptr;
      } else {
        int4* row = reinterpret_cast<int4*>(at);
        T* v = reinterpret_cast<T*>(row + n);
        const int nnz = (int)(G.g.T[0] * G.g.T[1] * G.g.T[2]);
        for (int k = threadIdx.x; k < nnz; k += TT) v[k] = G.A[k];
        L.D.A = v;
        L.D.minv = v + nnz;
        L.D.xa = L.D.minv + n;
        L.D.xb = L.D.xa + n;
        L.D.d = L.D.xb + n;
        L.D.b = L.D.d + n;
        L.D.r = L.D.b + n;
        for (int k = threadIdx.x; k < n; k += TT) {
          L.D.minv[k] = G.minv[k];
          int ix, iy, iz;
          decompose(G.g, k, ix, iy, iz);
          const RowInfo R = row_info<1>(G.g, ix, iy, iz);
          row[k] = make_int4((int)R.rp, R.lx + G.g.nn[0] * (R.ly + G.g.nn[1] * R.lz), R.cx | R.cy << 2 | R.cz << 4, 0);
        }
        L.row = row;
        at += tail_level_bytes<T>(G.g, n);
      }
      if (threadIdx.x == 0) lev[j] = L;
    }
  }
  pdl_wait();
  if (is_done(S)) return;
  __syncthreads();
  for (int n = threadIdx.x; n < (int)A.L[0].n; n += TT) lev[0].D.b[n] = A.L[0].b[n];
  __syncthreads();
  for (int j = 0; j < nl - 1; ++j) {
    const TailLev<T>& L = lev[j];
    const LevDev<T>& D = L.D;
    tail_cheb<T>(L, D.xa, D.xa, 0, 1, A.coef[j]);
    tail_cheb<T>(L, D.xa, D.xb, 1, 0, A.coef[j]);
    for (int n = threadIdx.x; n < (int)D.n; n += TT) resid_row<T>(D, n, tail_prod<T>(L, n, D.xb));
    __syncthreads();
    const LevDev<T>& C = lev[j + 1].D;
    for (int64_t n = threadIdx.x; n < C.n; n += TT) C.b[n] = restrict_row<T>(D.g, C.g, A.X[j + 1], D.r, n);
    __syncthreads();
  }
  const LevDev<T>& Lc = lev[nl - 1].D;
  for (int i = threadIdx.x; i < (int)Lc.n; i += TT) coarse_row<T>((int)Lc.n, Lc.A, Lc.b, Lc.xb, i);
  __syncthreads();
  for (int j = nl - 2; j >= 0; --j) {
    const TailLev<T>& L = lev[j];
    const LevDev<T>& D = L.D;
    const LevDev<T>& C = lev[j + 1].D;
    for (int64_t n = threadIdx.x; n < D.n; n += TT) prolong_row<T>(D.g, C.g, A.X[j + 1], C.xb, D.xb, n);
    __syncthreads();
    tail_cheb<T>(L, D.xb, D.xa, 0, 0, A.coef[j]);
    tail_cheb<T>(L, D.xa, D.xb, 1, 0, A.coef[j]);
  }
  // what the level above reads
  for (int n = threadIdx.x; n < (int)A.L[0].n; n += TT) A.L[0].xb[n] = lev[0].D.xb[n];
}

// Vector updates with a dot product: RED_PER_SM CTAs per SM (each CTA's FP64 tree takes the FP64 pipe for 320 cycles, so
// 16 per SM spent more time on the trees than on the vectors), four elements of a thread in flight, each with a partial sum
// of its own (Dot), so that a partial has no more terms than with 16 CTAs per SM.
constexpr int RED_PER_SM = 4;
template <typename L, typename F>
__device__ __forceinline__ void each4(int64_t n, L&& load, F&& use) {
  const int64_t st = (int64_t)gridDim.x * NT;
  for (int64_t i = (int64_t)blockIdx.x * NT + threadIdx.x; i < n; i += 4 * st) {
    decltype(load(i)) v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (i + k * st < n) v[k] = load(i + k * st);
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (i + k * st < n) use(i + k * st, v[k], k);
  }
}
template <typename T, int N>
struct Vals { T v[N]; };

// Four partial sums of products in the vectors' precision, added up in FP64.  FP32: with one FP64 addition, of the sum and
// what it lacks (two-sum), where four conversions and three additions would hold the FP64 pipe.
template <typename T>
struct Dot {
  T s[4] = {T(0), T(0), T(0), T(0)};
  __device__ __forceinline__ void add(int k, T a, T b) { s[k] = fma(a, b, s[k]); }
  __device__ __forceinline__ double total() const {
    if constexpr (sizeof(T) == 8) {
      return (s[0] + s[1]) + (s[2] + s[3]);
    } else {
      float t = s[0], c = 0.0f;
#pragma unroll
      for (int k = 1; k < 4; ++k) {
        const float n = __fadd_rn(t, s[k]), z = __fsub_rn(n, t);
        c = __fadd_rn(c, __fadd_rn(__fsub_rn(t, __fsub_rn(n, z)), __fsub_rn(s[k], z)));
        t = n;
      }
      // c is not finite where t is not, and subnormal beside sums whose squares underflow
      return (double)t + (mrgdev::widen_special(c) ? 0.0 : mrgdev::widen(c));
    }
  }
};

// ---- CG kernels -----------------------------------------------------------------------------------
template <typename T>
struct CgVec {
  T *x, *r, *p, *q;
  const T* z;
  double* parts;
  GScal* S;
};

// x = 0, r = b (FP64 in, T out), p = q = 0; r0 = |r|
template <typename T>
__global__ void __launch_bounds__(NT) k_cg_init(int64_t n, const double* __restrict__ b, CgVec<T> V) {
  Dot<T> rr;  // per-thread partials in the vector precision (no per-element FP64 work for FP32)
  each4(n, [&](int64_t i) { return (T)b[i]; },
        [&](int64_t i, T r, int k) {
          V.x[i] = T(0);
          V.r[i] = r;
          V.p[i] = T(0);
          V.q[i] = T(0);
          rr.add(k, r, r);
        });
  double m[1] = {block_sum(rr.total())};
  if (last_block<1>(V.parts, m, &V.S->counter)) {
    double t[1];
    sum_parts<1>(V.parts, t, &V.S->counter);
    if (threadIdx.x == 0) {
      GScal* S = V.S;
      S->r0 = sqrt(t[0]);
      S->rnorm = S->r0;
      S->iter = 0;
      S->status = MRG_OK;
      S->beta = 0.0;
      S->beta32 = 0.0f;
      S->rho = 0.0;
      S->done = (S->r0 == 0.0 || S->maxiter <= 0) ? 1 : 0;
      if (!isfinite(S->r0)) { S->done = 1; S->status = MRG_ENUMERIC; }
    }
  }
}

// rho_new = r . z ; beta = rho_new / rho (0 on the first call)
template <typename T>
__global__ void __launch_bounds__(NT) k_cg_rz(int64_t n, CgVec<T> V, int first) {
  pdl_trigger();
  pdl_wait();
  if (is_done(V.S)) return;
  Dot<T> rz;
  each4(n, [&](int64_t i) { return Vals<T, 2>{{V.r[i], V.z[i]}}; },
        [&](int64_t, const Vals<T, 2>& e, int k) { rz.add(k, e.v[0], e.v[1]); });
  double m[1] = {block_sum(rz.total())};
  if (last_block<1>(V.parts, m, &V.S->counter)) {
    double t[1];
    sum_parts<1>(V.parts, t, &V.S->counter);
    if (threadIdx.x == 0) {
      GScal* S = V.S;
      S->beta = first ? 0.0 : t[0] / S->rho;
      S->beta32 = (float)S->beta;
      S->rho = t[0];
      if (!(t[0] > 0.0) || !isfinite(t[0])) { S->status = MRG_ENUMERIC; S->done = 1; }
    }
  }
}

// w = A z ; p = z + beta p ; q = w + beta q ; partial p.q ; alpha = rho / p.q
template <int P, typename T>
__global__ void __launch_bounds__(NT, staged_per_sm<T>()) k_cg_spmv(Grid g, int64_t n, const T* __restrict__ A, CgVec<T> V) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t mbar[2 * (NT / 32)];
  pdl_trigger();
  T beta = T(0), pq = T(0);
  bool go = false;
  const bool ok = level_rows<P, T>(
      g, n, A, smem_raw, mbar,
      [&](int64_t i, const RowInfo& R, const T* vals) {
        const T w = (T)row_prod<P, T>(g, R, vals, V.z);
        const T pn = V.z[i] + beta * V.p[i];
        const T qn = w + beta * V.q[i];
        V.p[i] = pn;
        V.q[i] = qn;
        pq = fma(pn, qn, pq);
      },
      [&] {
        pdl_wait();
        beta = beta_of<T>(V.S);
        return go = !is_done(V.S);
      });
  if (!go) return;
  if (!ok) atomicExch(&V.S->err, 3);
  double m[1] = {block_sum((double)pq)};
  if (last_block<1>(V.parts, m, &V.S->counter)) {
    double t[1];
    sum_parts<1>(V.parts, t, &V.S->counter);
    if (threadIdx.x == 0) {
      GScal* S = V.S;
      S->pq = t[0];
      S->alpha = S->rho / t[0];
      S->alpha32 = (float)S->alpha;
      if (!(t[0] > 0.0) || !isfinite(S->alpha)) { S->status = MRG_ENUMERIC; S->done = 1; }
      if (S->err) { S->status = MRG_ETIMEOUT; S->done = 1; }
    }
  }
}

// x += alpha p ; r -= alpha q ; |r| ; stopping test
template <typename T>
__global__ void __launch_bounds__(NT) k_cg_update(int64_t n, CgVec<T> V, FirstStep<T> first) {
  pdl_trigger();
  pdl_wait();
  if (is_done(V.S)) return;
  const T alpha = alpha_of<T>(V.S);
  Dot<T> rr;
  each4(n, [&](int64_t i) { return Vals<T, 5>{{V.x[i], V.p[i], V.r[i], V.q[i], first.diag(i)}}; },
        [&](int64_t i, const Vals<T, 5>& e, int k) {
          V.x[i] = e.v[0] + alpha * e.v[1];
          const T r = e.v[2] - alpha * e.v[3];
          V.r[i] = r;
          rr.add(k, r, r);
          first(i, r, e.v[4]);
        });
  double m[1] = {block_sum(rr.total())};
  if (last_block<1>(V.parts, m, &V.S->counter)) {
    double t[1];
    sum_parts<1>(V.parts, t, &V.S->counter);
    if (threadIdx.x == 0) {
      GScal* S = V.S;
      S->rnorm = sqrt(t[0]);
      S->iter += 1;
      if (!(S->rnorm / S->r0 > S->tol) || S->iter >= S->maxiter) S->done = 1;
      if (!isfinite(S->rnorm)) { S->done = 1; S->status = MRG_ENUMERIC; }
    }
  }
}

template <typename T>
__global__ void k_to_f64(int64_t n, const T* __restrict__ a, double* __restrict__ b) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) b[i] = (double)a[i];
}

// ---- BiCGStab kernels (right preconditioning by the same V-cycle) ------------------------------
template <typename T>
struct BgVec {
  T *x, *r, *rh, *p, *v, *s, *t, *ph, *sh;
  double* parts;
  GScal* S;
};

// x = 0, r = rh = b, p = v = 0; rho = (rh . r), alpha = omega = 1, beta = 0
template <typename T>
__global__ void __launch_bounds__(NT) k_bg_init(int64_t n, const double* __restrict__ b, BgVec<T> V) {
  Dot<T> rr;
  each4(n, [&](int64_t i) { return (T)b[i]; },
        [&](int64_t i, T r, int k) {
          V.x[i] = T(0);
          V.r[i] = r;
          V.rh[i] = r;
          V.p[i] = T(0);
          V.v[i] = T(0);
          rr.add(k, r, r);
        });
  double m[1] = {block_sum(rr.total())};
  if (last_block<1>(V.parts, m, &V.S->counter)) {
    double t[1];
    sum_parts<1>(V.parts, t, &V.S->counter);
    if (threadIdx.x == 0) {
      GScal* S = V.S;
      S->r0 = sqrt(t[0]);
      S->rnorm = S->r0;
      S->rho = t[0];
      S->alpha = 1.0;
      S->omega = 1.0;
      S->beta = 0.0;
      S->alpha32 = S->omega32 = 1.0f;
      S->beta32 = 0.0f;
      S->iter = 0;
      S->status = MRG_OK;
      S->done = (S->r0 == 0.0 || S->maxiter <= 0) ? 1 : 0;
      if (!isfinite(S->r0)) { S->done = 1; S->status = MRG_ENUMERIC; }
    }
  }
}

// p = r + beta (p - omega v)
template <typename T>
__global__ void __launch_bounds__(NT) k_bg_p(int64_t n, BgVec<T> V, FirstStep<T> first) {
  pdl_trigger();
  pdl_wait();
  if (is_done(V.S)) return;
  const T beta = beta_of<T>(V.S), omega = omega_of<T>(V.S);
  for (int64_t i = (int64_t)blockIdx.x * NT + threadIdx.x; i < n; i += (int64_t)gridDim.x * NT) {
    const T mi = first.diag(i);
    const T b = V.r[i] + beta * (V.p[i] - omega * V.v[i]);
    V.p[i] = b;
    first(i, b, mi);
  }
}

// STEP 0: v = A ph, rv = rh . v, alpha = rho / rv.   STEP 1: t = A sh, omega = (t . s) / (t . t).
template <int P, typename T, int STEP>
__global__ void __launch_bounds__(NT, staged_per_sm<T>()) k_bg_spmv(Grid g, int64_t n, const T* __restrict__ A, BgVec<T> V) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t mbar[2 * (NT / 32)];
  pdl_trigger();
  const T* in = STEP == 0 ? V.ph : V.sh;
  T* out = STEP == 0 ? V.v : V.t;
  T d0 = T(0), d1 = T(0);
  bool go = false;
  const bool ok = level_rows<P, T>(
      g, n, A, smem_raw, mbar,
      [&](int64_t i, const RowInfo& R, const T* vals) {
        const T y = (T)row_prod<P, T>(g, R, vals, in);
        out[i] = y;
        if (STEP == 0) {
          d0 = fma(V.rh[i], y, d0);
        } else {
          d0 = fma(y, V.s[i], d0);
          d1 = fma(y, y, d1);
        }
      },
      [&] {
        pdl_wait();
        return go = !is_done(V.S);
      });
  if (!go) return;
  if (!ok) atomicExch(&V.S->err, 3);
  double m[2] = {block_sum((double)d0), block_sum((double)d1)};
  if (last_block<2>(V.parts, m, &V.S->counter)) {
    double t[2];
    sum_parts<2>(V.parts, t, &V.S->counter);
    if (threadIdx.x == 0) {
      GScal* S = V.S;
      if (STEP == 0) {
        S->rv = t[0];
        S->alpha = S->rho / t[0];
        S->alpha32 = (float)S->alpha;
        if (!(t[0] != 0.0) || !isfinite(S->alpha)) { S->status = MRG_ENUMERIC; S->done = 1; }
      } else {
        S->omega = (t[1] > 0.0) ? t[0] / t[1] : 0.0;
        S->omega32 = (float)S->omega;
      }
      if (S->err) { S->status = MRG_ETIMEOUT; S->done = 1; }
    }
  }
}

// s = r - alpha v
template <typename T>
__global__ void __launch_bounds__(NT) k_bg_s(int64_t n, BgVec<T> V, FirstStep<T> first) {
  pdl_trigger();
  pdl_wait();
  if (is_done(V.S)) return;
  const T alpha = alpha_of<T>(V.S);
  for (int64_t i = (int64_t)blockIdx.x * NT + threadIdx.x; i < n; i += (int64_t)gridDim.x * NT) {
    const T mi = first.diag(i);
    const T b = V.r[i] - alpha * V.v[i];
    V.s[i] = b;
    first(i, b, mi);
  }
}

// x += alpha ph + omega sh ; r = s - omega t ; |r|, rh . r -> beta for the next direction; stopping test
template <typename T>
__global__ void __launch_bounds__(NT) k_bg_update(int64_t n, BgVec<T> V) {
  pdl_trigger();
  pdl_wait();
  if (is_done(V.S)) return;
  const T alpha = alpha_of<T>(V.S), omega = omega_of<T>(V.S);
  Dot<T> rr, rhr;
  each4(n, [&](int64_t i) { return Vals<T, 6>{{V.x[i], V.ph[i], V.sh[i], V.s[i], V.t[i], V.rh[i]}}; },
        [&](int64_t i, const Vals<T, 6>& e, int k) {
          V.x[i] = e.v[0] + (alpha * e.v[1] + omega * e.v[2]);
          const T r = e.v[3] - omega * e.v[4];
          V.r[i] = r;
          rr.add(k, r, r);
          rhr.add(k, e.v[5], r);
        });
  double m[2] = {block_sum(rr.total()), block_sum(rhr.total())};
  if (last_block<2>(V.parts, m, &V.S->counter)) {
    double t[2];
    sum_parts<2>(V.parts, t, &V.S->counter);
    if (threadIdx.x == 0) {
      GScal* S = V.S;
      S->rnorm = sqrt(t[0]);
      S->iter += 1;
      S->beta = (t[1] / S->rho) * (S->alpha / S->omega);
      S->beta32 = (float)S->beta;
      S->rho = t[1];
      if (!(S->rnorm / S->r0 > S->tol) || S->iter >= S->maxiter) S->done = 1;
      if (!isfinite(S->rnorm)) { S->done = 1; S->status = MRG_ENUMERIC; }
      else if (!S->done && (!(t[1] != 0.0) || !(S->omega != 0.0))) { S->done = 1; S->status = MRG_ENUMERIC; }
    }
  }
}

inline unsigned nblk(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

int num_sms() { return mrg_device_sms(); }

unsigned grid_for(int64_t n, int per_sm) {
  const unsigned need = nblk(n, NT), cap = (unsigned)(per_sm * num_sms());
  return need < cap ? need : cap;
}

// ---- hierarchy ------------------------------------------------------------------------------------
struct HLevel {
  Grid g;
  int64_t n = 0, nnz = 0;
  Xfer X{{0, 0, 0}};          // how this level was coarsened from the finer one
  P3 pp{{1, 1, 1}};           // per-axis coupling order of this level (2 only on a Q2 level 0)
  int nsweep = 0;             // Galerkin sweeps from the finer level (one per coarsened axis)
  int sweep_axis[3] = {0, 0, 0};
  Grid mid[2];                // intermediate grids after all but the last sweep
  P3 mid_pp[2];
  int64_t* d_mid_pref[2] = {nullptr, nullptr};
  int64_t* d_pref = nullptr;  // prefix tables (coarse levels)
  void* A = nullptr;          // coarse levels: owned; level 0: the caller's Jacobian
  void *minv = nullptr, *xa = nullptr, *xb = nullptr, *d = nullptr, *b = nullptr, *r = nullptr;
};

template <typename T>
struct Hier {
  std::vector<HLevel> L;
  T* cinv = nullptr;
  T* mid[2] = {nullptr, nullptr};  // intermediate operators of the Galerkin sweeps
  unsigned int* lmax = nullptr;   // [nlev] float bits
  T* coef = nullptr;              // [nlev][NU][3] Chebyshev coefficients
  int* err = nullptr;             // setup / cycle error word
  T *x = nullptr, *r = nullptr, *p = nullptr, *q = nullptr;  // CG vectors (level-0 size)
  double* parts = nullptr;
  GScal* S = nullptr;
  GScal* h_S = nullptr;           // pinned mirror
  cudaGraphExec_t graph = nullptr;
  const void* graph_A = nullptr;
  cudaStream_t graph_stream = nullptr;
  // BiCGStab vectors (allocated on first use) and its captured chunk
  T *rh = nullptr, *v = nullptr, *sv = nullptr, *t = nullptr, *ph = nullptr, *sh = nullptr;
  cudaGraphExec_t bgraph = nullptr;
  const void* bgraph_A = nullptr;
  cudaStream_t bgraph_stream = nullptr;
  const void* setup_J = nullptr;  // Jacobian of the last setup
  // levels >= tail run in k_vcycle_tail (tail == number of levels: every step its own launch)
  int tail = -1;
  int graph_tail = -1, bgraph_tail = -1;  // the tail the captured chunks were recorded with
  TailArgs<T> targs;
};

struct GmgData {
  int kind = MRG_PREC_JACOBI;
  bool split = false;  // MRG_PREC_GMG_SPLIT: no fused coarse-level tail
  Hier<double>* h64 = nullptr;
  Hier<float>* h32 = nullptr;
};

GmgData* gdata(mrg_problem* p) {
  if (!p->gmg) p->gmg = new GmgData();
  return reinterpret_cast<GmgData*>(p->gmg);
}

// Host grid of a p = 1 level with nn nodes per axis (prefix tables uploaded to d_pref).
int make_level_grid(const Grid& fine, const int nn[3], const P3& pp, cudaStream_t s, Grid& g, int64_t*& d_pref) {
  g = fine;
  g.p = std::max(pp.p[0], std::max(pp.p[1], pp.p[2]));
  for (int k = 0; k < 3; ++k) {
    g.nn[k] = nn[k];
    g.nc[k] = (k < fine.dim) ? (nn[k] - 1) / pp.p[k] : 1;
  }
  std::vector<int64_t> pref;
  int64_t offs[3];
  for (int k = 0; k < 3; ++k) {
    offs[k] = (int64_t)pref.size();
    int64_t acc = 0;
    pref.push_back(0);
    for (int i = 0; i < g.nn[k]; ++i) {
      int lo, cnt;
      if (k < g.dim) axis_range(i, g.nn[k], pp.p[k], lo, cnt); else cnt = 1;
      acc += cnt;
      pref.push_back(acc);
    }
    g.T[k] = acc;
  }
  MRG_CUDA(cudaMallocAsync(&d_pref, pref.size() * sizeof(int64_t), s));
  MRG_CUDA(cudaMemcpyAsync(d_pref, pref.data(), pref.size() * sizeof(int64_t), cudaMemcpyHostToDevice, s));
  for (int k = 0; k < 3; ++k) g.P[k] = d_pref + offs[k];
  return MRG_OK;
}

template <typename T>
void free_hier(Hier<T>* H, cudaStream_t s) {
  if (!H) return;
  if (H->graph) cudaGraphExecDestroy(H->graph);
  if (H->bgraph) cudaGraphExecDestroy(H->bgraph);
  for (void* ptr : {(void*)H->rh, (void*)H->v, (void*)H->sv, (void*)H->t, (void*)H->ph, (void*)H->sh})
    if (ptr) cudaFreeAsync(ptr, s);
  for (size_t l = 0; l < H->L.size(); ++l) {
    HLevel& L = H->L[l];
    if (l > 0) {
      if (L.A) cudaFreeAsync(L.A, s);
      if (L.d_pref) cudaFreeAsync(L.d_pref, s);
      for (int k = 0; k < 2; ++k)
        if (L.d_mid_pref[k]) cudaFreeAsync(L.d_mid_pref[k], s);
    }
    for (void* ptr : {L.minv, L.xa, L.xb, L.d, L.b, L.r})
      if (ptr) cudaFreeAsync(ptr, s);
  }
  for (void* ptr : {(void*)H->mid[0], (void*)H->mid[1]})
    if (ptr) cudaFreeAsync(ptr, s);
  for (void* ptr : {(void*)H->cinv, (void*)H->lmax, (void*)H->coef, (void*)H->err, (void*)H->x, (void*)H->r, (void*)H->p,
                    (void*)H->q, (void*)H->parts, (void*)H->S})
    if (ptr) cudaFreeAsync(ptr, s);
  mrg_pinned_release(H->h_S);
  delete H;
}

// Builds the level structure (sizes, grids, buffers).  Values are computed by setup_values.
template <typename T>
int build_hier(const mrg_problem* p, Hier<T>*& out, cudaStream_t s) {
  Hier<T>* H = new Hier<T>();
  auto fail = [&](int rc) {
    free_hier(H, s);
    return rc;
  };
  HLevel L0;
  L0.g = p->g;
  L0.n = p->ndof;
  L0.nnz = p->nnz;
  for (int k = 0; k < 3; ++k) L0.pp.p[k] = (k < p->g.dim) ? p->g.p : 1;
  H->L.push_back(L0);
  // cell size per axis (box estimate); an axis is coarsened only while its cells are at most twice as
  // long as the shortest ones (semi-coarsening keeps point smoothing effective on stretched grids)
  double h[3] = {p->h[0], p->h[1], p->h[2]};
  while ((int)H->L.size() < MAXLEV) {
    const Grid& gf = H->L.back().g;
    const P3 pf = H->L.back().pp;
    const bool ptransfer = pf.p[0] == 2;  // Q2 level 0 -> Q1 on the same cells: every axis, h unchanged
    int nn[3], co[3] = {0, 0, 0}, any = 0;
    double hmin = 1e300;
    for (int k = 0; k < gf.dim; ++k) hmin = std::fmin(hmin, h[k]);
    for (int pass = 0; pass < 2 && !any; ++pass)
      for (int k = 0; k < gf.dim; ++k)
        if (ptransfer || (gf.nn[k] - 1 >= 3 && (pass == 1 || h[k] <= 2.0 * hmin * (1.0 + 1e-9)))) {
          co[k] = 1;
          any = 1;
        }
    for (int k = 0; k < 3; ++k) {
      nn[k] = gf.nn[k];
      if (co[k]) {
        nn[k] = (gf.nn[k] - 1 + 1) / 2 + 1;
        if (!ptransfer) h[k] *= 2.0;
      }
    }
    const int64_t nfine = H->L.back().n;
    if (!any || (nfine <= MAXC && !ptransfer)) break;
    HLevel Lc;
    int rc = make_level_grid(gf, nn, Lc.pp, s, Lc.g, Lc.d_pref);
    if (rc) { H->L.push_back(Lc); return fail(rc); }
    for (int k = 0; k < 3; ++k) Lc.X.co[k] = co[k];
    // sweep plan: coarsen the axes one at a time; intermediate grids for all but the last sweep (a
    // swept axis couples at order 1, the others keep the finer level's order)
    int cur[3] = {gf.nn[0], gf.nn[1], gf.nn[2]};
    P3 cp = pf;
    for (int k = 0; k < 3; ++k)
      if (co[k]) Lc.sweep_axis[Lc.nsweep++] = k;
    for (int w = 0; w + 1 < Lc.nsweep; ++w) {
      cur[Lc.sweep_axis[w]] = nn[Lc.sweep_axis[w]];
      cp.p[Lc.sweep_axis[w]] = 1;
      Lc.mid_pp[w] = cp;
      rc = make_level_grid(gf, cur, cp, s, Lc.mid[w], Lc.d_mid_pref[w]);
      if (rc) { H->L.push_back(Lc); return fail(rc); }
    }
    Lc.n = (int64_t)nn[0] * nn[1] * nn[2];
    Lc.nnz = Lc.g.T[0] * Lc.g.T[1] * Lc.g.T[2];
    H->L.push_back(Lc);
  }
  if (H->L.back().n > MAXC) return fail(mrg_fail(MRG_ENOTSUP, "multigrid: coarsest level too large"));
  for (size_t l = 0; l < H->L.size(); ++l) {
    HLevel& L = H->L[l];
    const size_t vb = (size_t)L.n * sizeof(T);
    if (l > 0 && cudaMallocAsync(&L.A, (size_t)L.nnz * sizeof(T), s) != cudaSuccess) return fail(mrg_fail(MRG_ENOMEM, "multigrid level matrix"));
    for (void** ptr : {&L.minv, &L.xa, &L.xb, &L.d, &L.b, &L.r})
      if (cudaMallocAsync(ptr, vb, s) != cudaSuccess) return fail(mrg_fail(MRG_ENOMEM, "multigrid level vectors"));
  }
  // scratch for the intermediate operators (largest over all levels)
  size_t midmax[2] = {0, 0};
  for (size_t l = 1; l < H->L.size(); ++l)
    for (int w = 0; w + 1 < H->L[l].nsweep; ++w) {
      const Grid& gm = H->L[l].mid[w];
      midmax[w] = std::max(midmax[w], (size_t)(gm.T[0] * gm.T[1] * gm.T[2]));
    }
  for (int w = 0; w < 2; ++w)
    if (midmax[w] && cudaMallocAsync(&H->mid[w], midmax[w] * sizeof(T), s) != cudaSuccess)
      return fail(mrg_fail(MRG_ENOMEM, "multigrid Galerkin scratch"));
  const int64_t n0 = p->ndof, nc = H->L.back().n;
  const size_t nparts = (size_t)2 * grid_for(n0, 16) + 64;
  if (cudaMallocAsync(&H->cinv, (size_t)nc * nc * sizeof(T), s) != cudaSuccess ||
      cudaMallocAsync(&H->lmax, MAXLEV * sizeof(unsigned int), s) != cudaSuccess ||
      cudaMallocAsync(&H->coef, (size_t)MAXLEV * NU * 3 * sizeof(T), s) != cudaSuccess ||
      cudaMallocAsync(&H->err, sizeof(int), s) != cudaSuccess ||
      cudaMallocAsync(&H->x, n0 * sizeof(T), s) != cudaSuccess || cudaMallocAsync(&H->r, n0 * sizeof(T), s) != cudaSuccess ||
      cudaMallocAsync(&H->p, n0 * sizeof(T), s) != cudaSuccess || cudaMallocAsync(&H->q, n0 * sizeof(T), s) != cudaSuccess ||
      cudaMallocAsync(&H->parts, nparts * sizeof(double), s) != cudaSuccess ||
      cudaMallocAsync(&H->S, sizeof(GScal), s) != cudaSuccess)
    return fail(mrg_fail(MRG_ENOMEM, "multigrid workspace"));
  static_assert(sizeof(GScal) <= 256, "pinned slot size");
  H->h_S = (GScal*)mrg_pinned_slot();
  if (!H->h_S) return fail(mrg_fail(MRG_ENOMEM, "multigrid pinned scalars"));
  MRG_CUDA(cudaMemsetAsync(H->S, 0, sizeof(GScal), s));
  MRG_CUDA(cudaMemsetAsync(H->parts, 0, nparts * sizeof(double), s));
  out = H;
  return MRG_OK;
}

template <typename T>
LevDev<T> levdev(const HLevel& L) {
  return LevDev<T>{L.g, L.n, (const T*)L.A, (T*)L.minv, (T*)L.xa, (T*)L.xb, (T*)L.d, (T*)L.b, (T*)L.r};
}

// First level of the fused tail: the first level below the finest with at most tail_rows<T>() rows (all
// levels below the finest are Q1), unless the caller asked for the split cycle or the tail would be too
// deep.  Fills the tail's kernel arguments.
template <typename T>
void set_tail(Hier<T>* H, bool split) {
  const int nl = (int)H->L.size();
  int t = nl;
  if (!split) {
    for (int l = 1; l < nl; ++l)
      if (H->L[l].n <= tail_rows<T>()) { t = l; break; }
    if (nl - t > MAXTAIL) t = nl;
    for (int l = t; l < nl; ++l)
      if (H->L[l].pp.p[0] != 1 || H->L[l].pp.p[1] != 1 || H->L[l].pp.p[2] != 1) t = nl;
  }
  TailArgs<T>& A = H->targs;
  for (;; ++t) {  // a first level that does not fit the shared memory stays with the launches
    A.nlev = nl - t;
    for (int j = 0; j < A.nlev; ++j) {
      A.L[j] = levdev<T>(H->L[t + j]);
      A.X[j] = H->L[t + j].X;
      A.coef[j] = H->coef + (size_t)(t + j) * NU * 3;
    }
    if (A.nlev == 0 || tail_smem<T>(A) <= TAIL_SMEM) break;
  }
  H->tail = t;
  A.cinv = H->cinv;
}

template <typename T>
int set_staged_attr() {
  static std::once_flag once;
  static cudaError_t e = cudaSuccess;
  std::call_once(once, [] {
    const int smem = (NT / 32) * 2 * wbuf_elems<T>() * (int)sizeof(T);
    e = cudaFuncSetAttribute(k_cheb<1, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_diag<1, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_rap_line<T, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, rap_smem<T>());
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_rap_line<T, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, rap_smem<T>());
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_rap_line<T, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, rap_smem<T>());
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_vcycle_tail<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TAIL_SMEM);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_resid<1, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_cg_spmv<1, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_bg_spmv<1, T, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_bg_spmv<1, T, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  });
  return e == cudaSuccess ? MRG_OK : mrg_cuda_check(e, "multigrid smem attribute");
}

template <typename T>
constexpr int staged_smem() { return (NT / 32) * 2 * wbuf_elems<T>() * (int)sizeof(T); }

// Level operators, diagonals, Gershgorin bounds and the coarsest inverse for the Jacobian J.
// Level 0 only: the new J, its Jacobi inverse and Chebyshev bound; the coarse levels stay as they are.
template <typename T>
int setup_level0(Hier<T>* H, const T* J, cudaStream_t s) {
  HLevel& L = H->L[0];
  L.A = const_cast<T*>(J);
  MRG_CUDA(cudaMemsetAsync(H->lmax, 0, sizeof(unsigned int), s));
  if (L.pp.p[0] == 2) k_diag<2, T><<<grid_for(L.n, 16), NT, 0, s>>>(L.g, (const T*)L.A, (T*)L.minv, H->lmax, H->err);
  else k_diag<1, T><<<grid_for(L.n, staged_per_sm<T>()), NT, staged_smem<T>(), s>>>(L.g, (const T*)L.A, (T*)L.minv, H->lmax, H->err);
  k_cheb_coef<T><<<1, 32, 0, s>>>(H->lmax, (int)H->L.size(), H->coef);
  MRG_CUDA(cudaGetLastError());
  return MRG_OK;
}

template <typename T>
int setup_values(Hier<T>* H, const T* J, cudaStream_t s) {
  H->L[0].A = const_cast<T*>(J);
  MRG_CUDA(cudaMemsetAsync(H->lmax, 0, MAXLEV * sizeof(unsigned int), s));
  MRG_CUDA(cudaMemsetAsync(H->err, 0, sizeof(int), s));
  const int nl = (int)H->L.size();
  for (int l = 0; l < nl; ++l) {
    HLevel& L = H->L[l];
    if (l > 0) {
      const HLevel& F = H->L[l - 1];
      const Grid* gin = &F.g;
      P3 pin = F.pp;
      const T* ain = (const T*)F.A;
      for (int w = 0; w < L.nsweep; ++w) {
        const bool last = (w + 1 == L.nsweep);
        const Grid& gout = last ? L.g : L.mid[w];
        const P3 pout = last ? L.pp : L.mid_pp[w];
        T* aout = last ? (T*)L.A : H->mid[w];
        const int64_t nout = (int64_t)gout.nn[0] * gout.nn[1] * gout.nn[2];
        const bool line = gout.dim == 3 && pin.p[0] == 1 && pin.p[1] == 1 && pin.p[2] == 1;
        if (!line && nout < RAP_WARP_ROWS) {
          const unsigned nb = nblk(nout * 32, NT);
          if (L.sweep_axis[w] == 0) k_rap_axis_w<T, 0><<<nb, NT, 0, s>>>(*gin, pin, gout, pout, ain, aout);
          else if (L.sweep_axis[w] == 1) k_rap_axis_w<T, 1><<<nb, NT, 0, s>>>(*gin, pin, gout, pout, ain, aout);
          else k_rap_axis_w<T, 2><<<nb, NT, 0, s>>>(*gin, pin, gout, pout, ain, aout);
        } else if (line) {
          const int tiles = (gout.nn[0] + 31) / 32;
          const int64_t nt = (int64_t)tiles * gout.nn[1] * gout.nn[2];
          const unsigned nb = nblk(nt, RAP_W);
          constexpr int smem = rap_smem<T>();
          if (L.sweep_axis[w] == 0) k_rap_line<T, 0><<<nb, RAP_W * 32, smem, s>>>(*gin, gout, tiles, nt, ain, aout);
          else if (L.sweep_axis[w] == 1) k_rap_line<T, 1><<<nb, RAP_W * 32, smem, s>>>(*gin, gout, tiles, nt, ain, aout);
          else k_rap_line<T, 2><<<nb, RAP_W * 32, smem, s>>>(*gin, gout, tiles, nt, ain, aout);
        } else {
          k_rap_axis<T><<<nblk(nout, NT), NT, 0, s>>>(*gin, pin, gout, pout, L.sweep_axis[w], ain, aout, H->err);
        }
        MRG_CUDA(cudaGetLastError());
        gin = &gout;
        pin = pout;
        ain = aout;
      }
    }
    if (L.pp.p[0] == 2) k_diag<2, T><<<grid_for(L.n, 16), NT, 0, s>>>(L.g, (const T*)L.A, (T*)L.minv, H->lmax + l, H->err);
    else k_diag<1, T><<<grid_for(L.n, staged_per_sm<T>()), NT, staged_smem<T>(), s>>>(L.g, (const T*)L.A, (T*)L.minv, H->lmax + l, H->err);
    MRG_CUDA(cudaGetLastError());
  }
  k_coarse_inv<T><<<1, IT, 0, s>>>(H->L.back().g, (const T*)H->L.back().A, H->cinv, H->err);
  k_cheb_coef<T><<<1, 32, 0, s>>>(H->lmax, nl, H->coef);
  MRG_CUDA(cudaGetLastError());
  return MRG_OK;
}

// Launches of the row kernels for a level: Q1 levels use the staged loop (dynamic shared memory, fewer
// CTAs per SM), a Q2 level 0 the direct row loop.
// A kernel of the cycle on a level of n rows (grid transfers: of the finer level).  Chained launches hide the launch and the
// first copies, but the next kernel's CTAs take their places one by one as those of the one before end, which costs a large
// level, and a large FP64 level more, than that.  Newton solves in ms.
// FP64 thermal, all chained / none / levels up to 2^15 rows / up to 2^13: 128^3 50.3, 39.6, 39.1, 39.1; 48^3 6.94, 6.74,
// 6.36, 6.30; 40^3 5.44, 5.49, 4.96, 5.15; 26^3 3.78, 4.09, 3.77, 3.66; 20^3 1.92, 2.12, 1.93, 1.94 (1+u^2 7.17, 7.42, 7.17,
// 6.74).  FP32 thermal, all / up to 2^20 / 2^19 / 2^16 / 2^12: 192^3 36.8, 32.5; 128^3 11.4, 10.92, 10.93, 11.06, 11.45;
// 96^3 6.42, 6.41, 6.35, 6.49, 6.62; 64^3 3.46, 3.47, 3.47, 3.58, 3.92; 28^3 1.89, 1.89, 1.88, 1.88, 1.94.
constexpr int64_t CHAIN_ROWS64 = 1 << 13, CHAIN_ROWS32 = 1 << 19;
// A refused launch inside a capture leaves the capture intact, without that kernel: so every launch is looked at, the first
// error is kept in e, and nothing is launched after it.
template <typename... A>
void launch_q2(cudaError_t& e, A&&... args) {
  if (e == cudaSuccess) e = launch_whole(args...);
}
template <typename T, typename... A>
void launch_level(cudaError_t& e, int64_t n, A&&... args) {
  if (e != cudaSuccess) return;
  e = n <= (sizeof(T) == 4 ? CHAIN_ROWS32 : CHAIN_ROWS64) ? launch_pdl(args...) : launch_whole(args...);
}

template <typename T>
void launch_cheb(cudaError_t& e, const HLevel& L, const LevDev<T>& D, const T* xin, T* xout, int k, int zero_x,
                 const T* coef, const GScal* S, int* err, cudaStream_t s) {
  if (zero_x)
    launch_level<T>(e, D.n, k_cheb<1, T>, grid_for(D.n, 16), NT, 0, s, D, xin, xout, k, 1, coef, S, err);
  else if (L.pp.p[0] == 2)
    launch_q2(e, k_cheb<2, T>, grid_for(D.n, 16), NT, 0, s, D, xin, xout, k, 0, coef, S, err);
  else
    launch_level<T>(e, D.n, k_cheb<1, T>, grid_for(D.n, staged_per_sm<T>()), NT, staged_smem<T>(), s, D, xin, xout, k, 0, coef, S, err);
}

template <typename T>
void launch_resid(cudaError_t& e, const HLevel& L, const LevDev<T>& D, const T* x, const GScal* S, int* err, cudaStream_t s) {
  if (L.pp.p[0] == 2) launch_q2(e, k_resid<2, T>, grid_for(D.n, 16), NT, 0, s, D, x, S, err);
  else launch_level<T>(e, D.n, k_resid<1, T>, grid_for(D.n, staged_per_sm<T>()), NT, staged_smem<T>(), s, D, x, S, err);
}

template <typename T>
FirstStep<T> first_step(const Hier<T>* H, int l) {
  const int nl = (int)H->L.size(), tail = H->tail < 1 ? nl : H->tail;
  const HLevel& L = H->L[l];
  return FirstStep<T>{l < nl - 1 && l < tail ? H->coef + (size_t)l * NU * 3 : nullptr, (const T*)L.minv, (T*)L.d, (T*)L.xa};
}

// One V(NU, NU) cycle: out = M^{-1} in on level 0 (in, out: level-0 vectors not used by the cycle).  begun: level 0's first
// step is done.
template <typename T>
void enqueue_vcycle(cudaError_t& e, Hier<T>* H, const T* in, T* out, bool begun, cudaStream_t s) {
  const int nl = (int)H->L.size();
  const int tail = H->tail < 1 ? nl : H->tail;  // levels >= tail: k_vcycle_tail
  const GScal* S = H->S;
  for (int l = 0; l < nl - 1 && l < tail; ++l) {
    LevDev<T> D = levdev<T>(H->L[l]);
    if (l == 0) D.b = const_cast<T*>(in);
    // pre-smoothing from x = 0: xa <- step 0 (with the kernel that wrote b), xb <- step 1
    if (l == 0 && !begun) launch_cheb<T>(e, H->L[l], D, D.xa, D.xa, 0, 1, H->coef + (size_t)l * NU * 3, S, H->err, s);
    launch_cheb<T>(e, H->L[l], D, D.xa, D.xb, 1, 0, H->coef + (size_t)l * NU * 3, S, H->err, s);
    launch_resid<T>(e, H->L[l], D, D.xb, S, H->err, s);
    const HLevel& C = H->L[l + 1];
    launch_level<T>(e, D.n, k_restrict<T>, grid_for(C.n, 16), NT, 0, s, D.g, C.g, C.X, D.r, (T*)C.b, first_step(H, l + 1), S);
  }
  if (tail < nl) {
    launch_level<T>(e, H->L[tail - 1].n, k_vcycle_tail<T>, 1, TT, tail_smem<T>(H->targs), s, H->targs, S);
  } else {
    // a mesh of at most MAXC nodes is its own coarsest level: the inverse takes the cycle's input to its output
    const HLevel& Lc = H->L[nl - 1];
    launch_level<T>(e, Lc.n, k_coarse_apply<T>, 1, NT, 0, s, (int)Lc.n, H->cinv, nl == 1 ? in : (const T*)Lc.b,
                    nl == 1 ? out : (T*)Lc.xb, S);
  }
  for (int l = std::min(tail, nl - 1) - 1; l >= 0; --l) {
    LevDev<T> D = levdev<T>(H->L[l]);
    if (l == 0) D.b = const_cast<T*>(in);
    const HLevel& C = H->L[l + 1];
    launch_level<T>(e, D.n, k_prolong<T>, grid_for(sizeof(T) == 4 ? (D.n + 1) / 2 : D.n, 16), NT, 0, s, D.g, C.g, C.X, (const T*)C.xb, D.xb, S);
    // post-smoothing: xb -> xa (step 0), xa -> xb (step 1; level 0: -> out)
    launch_cheb<T>(e, H->L[l], D, D.xb, D.xa, 0, 0, H->coef + (size_t)l * NU * 3, S, H->err, s);
    launch_cheb<T>(e, H->L[l], D, D.xa, l == 0 ? out : D.xb, 1, 0, H->coef + (size_t)l * NU * 3, S, H->err, s);
  }
}

template <typename T>
CgVec<T> cgvec(Hier<T>* H) {
  return CgVec<T>{H->x, H->r, H->p, H->q, (const T*)H->L[0].xb, H->parts, H->S};
}

template <typename T>
cudaError_t enqueue_iters(Hier<T>* H, int count, cudaStream_t s) {
  cudaError_t e = cudaSuccess;
  const HLevel& L0 = H->L[0];
  CgVec<T> V = cgvec(H);
  const unsigned ge = grid_for(L0.n, 16), gs = grid_for(L0.n, staged_per_sm<T>()), gr = grid_for(L0.n, RED_PER_SM);
  for (int it = 0; it < count; ++it) {
    if (L0.pp.p[0] == 2) launch_q2(e, k_cg_spmv<2, T>, ge, NT, 0, s, L0.g, L0.n, (const T*)L0.A, V);
    else launch_level<T>(e, L0.n, k_cg_spmv<1, T>, gs, NT, staged_smem<T>(), s, L0.g, L0.n, (const T*)L0.A, V);
    launch_level<T>(e, L0.n, k_cg_update<T>, gr, NT, 0, s, L0.n, V, first_step(H, 0));
    enqueue_vcycle(e, H, H->r, (T*)H->L[0].xb, true, s);
    launch_level<T>(e, L0.n, k_cg_rz<T>, gr, NT, 0, s, L0.n, V, 0);
  }
  return e;
}

template <typename T>
int finish_solve(mrg_problem* p, Hier<T>* H, cudaGraphExec_t graph, double* x, double rtol, int maxiter,
                 mrg_solve_stats* st, cudaStream_t s, const char* what) {
  const int64_t n = p->ndof;
  const int max_chunks = maxiter / GCHUNK + 2;
  for (int c = 0; c < max_chunks; ++c) {
    MRG_CUDA(cudaGraphLaunch(graph, s));
    MRG_CUDA(cudaMemcpyAsync(H->h_S, H->S, sizeof(GScal), cudaMemcpyDeviceToHost, s));
    MRG_CUDA(cudaStreamSynchronize(s));
    if (H->h_S->done) break;
  }
  int herr = 0;
  MRG_CUDA(cudaMemcpyAsync(&herr, H->err, sizeof(int), cudaMemcpyDeviceToHost, s));
  k_to_f64<T><<<nblk(n, 256), 256, 0, s>>>(n, H->x, x);
  MRG_CUDA(cudaGetLastError());
  MRG_CUDA(cudaStreamSynchronize(s));
  const GScal* h = H->h_S;
  if (st) {
    st->iterations = h->iter;
    st->outer_iterations = 0;
    st->rel_residual = (h->r0 > 0) ? h->rnorm / h->r0 : 0.0;
    st->abs_residual = h->rnorm;
    st->status = h->status;
  }
  if (herr == 3 || h->status == MRG_ETIMEOUT) return mrg_fail(MRG_ETIMEOUT, std::string(what) + ": a staging copy timed out");
  if (herr) return mrg_fail(MRG_ENUMERIC, "multigrid setup: singular coarse operator or transfer out of range");
  if (h->status != MRG_OK) return mrg_fail(h->status, std::string(what) + ": breakdown or non-finite values");
  if (h->r0 > 0 && h->rnorm / h->r0 > rtol) {
    if (st) st->status = MRG_ENOCONV;
    return mrg_fail(MRG_ENOCONV, std::string(what) + ": not converged within maxiter");
  }
  return MRG_OK;
}

// Brings the hierarchy up to date with J as the caller asks (MRG_GMG_SETUP_*); a J other than the one of
// the last setup always gets a full setup.
template <typename T>
int follow_j(Hier<T>* H, const T* J, int setup, cudaStream_t s) {
  if (setup == MRG_GMG_SETUP_FULL || H->setup_J != (const void*)J) {
    const int rc = setup_values(H, J, s);
    if (rc) return rc;
    H->setup_J = J;
  } else if (setup == MRG_GMG_SETUP_LEVEL0) {
    return setup_level0(H, J, s);
  }
  return MRG_OK;
}

template <typename T>
int gmg_cg(mrg_problem* p, Hier<T>* H, const T* J, const double* b, double* x, double rtol, int maxiter,
           mrg_solve_stats* st, int setup, cudaStream_t s) {
  int rc = set_staged_attr<T>();
  if (rc) return rc;
  rc = follow_j(H, J, setup, s);
  if (rc) return rc;
  set_tail(H, gdata(p)->split);
  GScal init{};
  init.tol = rtol;
  init.maxiter = maxiter;
  MRG_CUDA(cudaMemcpyAsync(H->S, &init, sizeof(GScal), cudaMemcpyHostToDevice, s));
  const int64_t n = p->ndof;
  CgVec<T> V = cgvec(H);
  k_cg_init<T><<<grid_for(n, RED_PER_SM), NT, 0, s>>>(n, b, V);
  MRG_CUDA(cudaGetLastError());
  cudaError_t e = cudaSuccess;
  enqueue_vcycle(e, H, H->r, (T*)H->L[0].xb, false, s);
  if (e != cudaSuccess) {
    cudaGetLastError();  // not to be found by the next launch's check
    return mrg_cuda_check(e, "multigrid cycle launch");
  }
  k_cg_rz<T><<<grid_for(n, RED_PER_SM), NT, 0, s>>>(n, V, 1);
  MRG_CUDA(cudaGetLastError());
  // captured chunk of iterations (re-captured when the Jacobian pointer or the stream changes)
  if (!H->graph || H->graph_A != (const void*)J || H->graph_stream != s || H->graph_tail != H->tail) {
    if (H->graph) {
      cudaGraphExecDestroy(H->graph);
      H->graph = nullptr;
    }
    cudaStream_t cs = nullptr;
    MRG_CUDA(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
    cudaGraph_t graph = nullptr;
    e = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
      e = enqueue_iters(H, GCHUNK, cs);
      const cudaError_t ended = cudaStreamEndCapture(cs, &graph);
      if (e == cudaSuccess) e = ended;
    }
    if (e == cudaSuccess) e = cudaGraphInstantiate(&H->graph, graph, 0);
    if (graph) cudaGraphDestroy(graph);
    cudaStreamDestroy(cs);
    if (e != cudaSuccess) {
      cudaGetLastError();  // not to be found by the next launch's check
      return mrg_cuda_check(e, "multigrid CG graph capture");
    }
    H->graph_A = J;
    H->graph_stream = s;
    H->graph_tail = H->tail;
  }
  return finish_solve(p, H, H->graph, x, rtol, maxiter, st, s, "multigrid CG");
}

template <typename T>
BgVec<T> bgvec(Hier<T>* H) {
  return BgVec<T>{H->x, H->r, H->rh, H->p, H->v, H->sv, H->t, H->ph, H->sh, H->parts, H->S};
}

template <typename T>
cudaError_t enqueue_bg_iters(Hier<T>* H, int count, cudaStream_t s) {
  cudaError_t e = cudaSuccess;
  const HLevel& L0 = H->L[0];
  BgVec<T> V = bgvec(H);
  const unsigned ge = grid_for(L0.n, 16), gs = grid_for(L0.n, staged_per_sm<T>()), gr = grid_for(L0.n, RED_PER_SM);
  for (int it = 0; it < count; ++it) {
    launch_level<T>(e, L0.n, k_bg_p<T>, ge, NT, 0, s, L0.n, V, first_step(H, 0));
    enqueue_vcycle(e, H, H->p, H->ph, true, s);
    if (L0.pp.p[0] == 2) launch_q2(e, k_bg_spmv<2, T, 0>, ge, NT, 0, s, L0.g, L0.n, (const T*)L0.A, V);
    else launch_level<T>(e, L0.n, k_bg_spmv<1, T, 0>, gs, NT, staged_smem<T>(), s, L0.g, L0.n, (const T*)L0.A, V);
    launch_level<T>(e, L0.n, k_bg_s<T>, ge, NT, 0, s, L0.n, V, first_step(H, 0));
    enqueue_vcycle(e, H, H->sv, H->sh, true, s);
    if (L0.pp.p[0] == 2) launch_q2(e, k_bg_spmv<2, T, 1>, ge, NT, 0, s, L0.g, L0.n, (const T*)L0.A, V);
    else launch_level<T>(e, L0.n, k_bg_spmv<1, T, 1>, gs, NT, staged_smem<T>(), s, L0.g, L0.n, (const T*)L0.A, V);
    launch_level<T>(e, L0.n, k_bg_update<T>, gr, NT, 0, s, L0.n, V);
  }
  return e;
}

template <typename T>
int gmg_bicgstab(mrg_problem* p, Hier<T>* H, const T* J, const double* b, double* x, double rtol, int maxiter,
                 mrg_solve_stats* st, int setup, cudaStream_t s) {
  int rc = set_staged_attr<T>();
  if (rc) return rc;
  const int64_t n = p->ndof;
  if (!H->rh)
    for (T** ptr : {&H->rh, &H->v, &H->sv, &H->t, &H->ph, &H->sh})
      if (cudaMallocAsync(ptr, n * sizeof(T), s) != cudaSuccess) return mrg_fail(MRG_ENOMEM, "multigrid BiCGStab vectors");
  rc = follow_j(H, J, setup, s);
  if (rc) return rc;
  set_tail(H, gdata(p)->split);
  GScal init{};
  init.tol = rtol;
  init.maxiter = maxiter;
  MRG_CUDA(cudaMemcpyAsync(H->S, &init, sizeof(GScal), cudaMemcpyHostToDevice, s));
  k_bg_init<T><<<grid_for(n, RED_PER_SM), NT, 0, s>>>(n, b, bgvec(H));
  MRG_CUDA(cudaGetLastError());
  if (!H->bgraph || H->bgraph_A != (const void*)J || H->bgraph_stream != s || H->bgraph_tail != H->tail) {
    if (H->bgraph) {
      cudaGraphExecDestroy(H->bgraph);
      H->bgraph = nullptr;
    }
    cudaStream_t cs = nullptr;
    MRG_CUDA(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
    cudaGraph_t graph = nullptr;
    cudaError_t e = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
      e = enqueue_bg_iters(H, GCHUNK, cs);
      const cudaError_t ended = cudaStreamEndCapture(cs, &graph);
      if (e == cudaSuccess) e = ended;
    }
    if (e == cudaSuccess) e = cudaGraphInstantiate(&H->bgraph, graph, 0);
    if (graph) cudaGraphDestroy(graph);
    cudaStreamDestroy(cs);
    if (e != cudaSuccess) {
      cudaGetLastError();  // not to be found by the next launch's check
      return mrg_cuda_check(e, "multigrid BiCGStab graph capture");
    }
    H->bgraph_A = J;
    H->bgraph_stream = s;
    H->bgraph_tail = H->tail;
  }
  return finish_solve(p, H, H->bgraph, x, rtol, maxiter, st, s, "multigrid BiCGStab");
}

}  // namespace

int mrg_gmg_kind(const mrg_problem* p) {
  return p->gmg ? reinterpret_cast<const GmgData*>(p->gmg)->kind : MRG_PREC_JACOBI;
}

void mrg_gmg_drop_hierarchy(mrg_problem* p) {
  GmgData* G = reinterpret_cast<GmgData*>(p->gmg);
  if (!G) return;
  free_hier(G->h64, p->stream);
  free_hier(G->h32, p->stream);
  G->h64 = nullptr;
  G->h32 = nullptr;
}

void mrg_gmg_free(mrg_problem* p) {
  GmgData* G = reinterpret_cast<GmgData*>(p->gmg);
  if (!G) return;
  free_hier(G->h64, p->stream);
  free_hier(G->h32, p->stream);
  delete G;
  p->gmg = nullptr;
}

// Solves J x = b (x0 = 0) with multigrid-preconditioned CG in the precision of J; x receives the FP64
// solution.
int mrg_gmg_solve(mrg_problem* p, const void* J, bool fp32, const double* b, double* x, double rtol, int maxiter,
                  mrg_solve_stats* st, int setup, cudaStream_t s) {
  if (p->g.p > 2) return mrg_fail(MRG_ENOTSUP, "multigrid: Q1 and Q2 problems only");
  GmgData* G = gdata(p);
  int rc;
  if (fp32) {
    if (!G->h32 && (rc = build_hier<float>(p, G->h32, s))) return rc;
    return gmg_cg<float>(p, G->h32, (const float*)J, b, x, rtol, maxiter, st, setup, s);
  }
  if (!G->h64 && (rc = build_hier<double>(p, G->h64, s))) return rc;
  return gmg_cg<double>(p, G->h64, (const double*)J, b, x, rtol, maxiter, st, setup, s);
}

// Same for a nonsymmetric J: right-preconditioned BiCGStab with the multigrid V-cycle.
int mrg_gmg_bicgstab(mrg_problem* p, const void* J, bool fp32, const double* b, double* x, double rtol, int maxiter,
                     mrg_solve_stats* st, int setup, cudaStream_t s) {
  if (p->g.p > 2) return mrg_fail(MRG_ENOTSUP, "multigrid: Q1 and Q2 problems only");
  GmgData* G = gdata(p);
  int rc;
  if (fp32) {
    if (!G->h32 && (rc = build_hier<float>(p, G->h32, s))) return rc;
    return gmg_bicgstab<float>(p, G->h32, (const float*)J, b, x, rtol, maxiter, st, setup, s);
  }
  if (!G->h64 && (rc = build_hier<double>(p, G->h64, s))) return rc;
  return gmg_bicgstab<double>(p, G->h64, (const double*)J, b, x, rtol, maxiter, st, setup, s);
}

extern "C" int mrg_set_preconditioner(mrg_problem* p, int32_t kind) {
  if (!p) return mrg_fail(MRG_EINVAL, "mrg_set_preconditioner: null problem");
  if (kind != MRG_PREC_JACOBI && kind != MRG_PREC_GMG && kind != MRG_PREC_GMG_SPLIT)
    return mrg_fail(MRG_EINVAL, "mrg_set_preconditioner: unknown preconditioner");
  if (kind != MRG_PREC_JACOBI && p->g.p > 2)
    return mrg_fail(MRG_ENOTSUP, "multigrid preconditioner: Q1 and Q2 problems only");
  gdata(p)->kind = (kind == MRG_PREC_GMG_SPLIT) ? MRG_PREC_GMG : kind;
  gdata(p)->split = (kind == MRG_PREC_GMG_SPLIT);
  return MRG_OK;
}
