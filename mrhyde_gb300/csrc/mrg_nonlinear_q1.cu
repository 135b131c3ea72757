// 1 + u^2 diffusion on Q1 hexahedra of identical affine cells (reference: src/physics/thermal.cpp:71-165,
// src/managers/assembly/assemblyManager_jacres.hpp:121-630, assemblyManager_scatter.hpp:164-278).  These are the
// nonlinear requests of the serving loop.
//
// FP64 arithmetic issues at 1/64 of the FP32 rate here, so the FP64 passes are bound by their operation count
// and the cell matrix is formed from few distinct numbers instead of row by row.  A linear node's reference
// gradient along its own axis is the constant +-1/2, and all Gauss weights are equal.  With d_a the difference
// of u along axis a (constant along a), c = 1 + u^2 and w_a = |J| / h_a^2 up to the rule's weight,
//     J[l][j] = sum_a sigma(l_a) Z_a[j_a][t_b][t_c],
//     Z_a[j] = pairs over (q_b, q_c) of  w_a ( sigma(j) sum_{q_a} c + 2 d_a sum_{q_a} u L[q_a][j] ),
// where b, c are the other two axes, sigma(0) = -1, sigma(1) = +1 and t the unordered pair of the two nodes' ends
// along an axis (00, 01 or 11: the weight of a Gauss point is L[q][l] L[q][j]).  So 54 numbers a cell give its 64
// entries: about 225 operations, and 2 additions an entry when the rows gather them (the row-by-row contraction
// took about 200 operations a row and cell, 1600 a cell).  The residual shares c and d_a with it: about 80
// operations a cell besides the 54 of the fields, against 360 with one lane per Gauss point.
//
//   k_nl1_cell   one thread a cell: the 54 numbers and the 8 residual entries to a workspace in blocks of 32 cells,
//                so that lanes write and read consecutive addresses and every offset is an immediate
//   k_nl1_row    one thread a CSR row: 24 loads from each of its 8 cells, the CTA's rows staged in shared memory
//                and written once; the residual adds the cells' entries in the same order
// Measured, FP64 Jacobian and residual on 95^3 cells: 3506 -> 938 us (cells 600, rows 340, FP64 pipe 84 and 83 %
// active; the row-by-row contraction took 2712 and eight coloured residual launches 780); FP32 Jacobian alone on
// 96^3 cells 865 -> about 40 us.
// The workspace is taken from the device's pool in stream order for each call, so calls of one handle may overlap
// on several streams and may be captured; a mesh that would need more than MRG_PIECE_BYTES is worked on in pieces.
#include <cmath>

#include "mrg_device.cuh"
#include "mrg_fixmul.cuh"
#include "mrg_internal.h"

namespace {

constexpr int CT_ = 128;  // cells per CTA
constexpr int RT = 128;   // rows per CTA
constexpr int NZ_ = 54;   // numbers per cell
constexpr int CB = MRG_CELL_BLOCK;  // cells per workspace block

// products and sums that must not be contracted differently from one instance to the next (the residual of the
// separate and of the fused call has the same bits)
__device__ __forceinline__ double mulr(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double addr(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float addr(float a, float b) { return __fadd_rn(a, b); }

template <typename T>
__device__ __forceinline__ T as(double v) {
  if constexpr (sizeof(T) == 4) return mrgfix::f64_to_f32_rn(v);  // on the integer pipes
  else return v;
}
template <typename T>
__device__ __forceinline__ T as(float v) { return (T)v; }

struct Nl1Args {
  Grid g;
  double beta;       // L[0][1] = L[1][0]: the far node's weight at a Gauss point
  double alpha, slope;  // 1 - beta, beta (1 - 2 beta)
  double w[3];       // |J| w_q / h_a^2
  double load;       // f * int(phi_l) over one cell
  float betaf, slopef, wf[3];
  // L L at the Gauss point near node 0 for the pairs 00, 01, 11.  FP64: in units of the pair 01's, which wj has twice
  double near, far;  // 00 / 01 and 11 / 01
  double wj[3];      // w times the pair 01's weight squared
  float m32[3][2];   // FP32: value and what it lacks
  int64_t c0, c1;    // cells of the launch
};

template <typename T>
__device__ __forceinline__ T beta_of(const Nl1Args& A) {
  if constexpr (sizeof(T) == 4) return A.betaf; else return A.beta;
}
template <typename T>
__device__ __forceinline__ T slope_of(const Nl1Args& A) {
  if constexpr (sizeof(T) == 4) return A.slopef; else return A.slope;
}
template <typename T>
__device__ __forceinline__ T w_of(const Nl1Args& A, int a) {
  if constexpr (sizeof(T) == 4) return A.wf[a]; else return A.w[a];
}
template <typename T>
__device__ __forceinline__ T wj_of(const Nl1Args& A, int a) {  // for the 54 numbers
  if constexpr (sizeof(T) == 4) return A.wf[a]; else return A.wj[a];
}

// values at the two Gauss points from two nodes, or node sums from two Gauss points (the 2 x 2 table is
// symmetric); d is the difference
template <typename T>
__device__ __forceinline__ void lerp2(T beta, T a, T b, T& p0, T& p1, T& d) {
  d = addr(b, -a);
  p0 = fma(beta, d, a);
  p1 = fma(-beta, d, b);
}

// Sums of two Gauss points' values against L[q][l] L[q][j]: (00, 01, 11).  FP64: in units of the pair 01's weight, so that
// its sum takes no multiplication: 5 operations, none a difference (6 with the weights themselves).  FP32 is not short of
// operations: the table's values come in two parts, because their rounding would shift every entry the same way (FP32
// matrix at 16 x 16 x 16 cells, 2-norm of the error over that of the matrix: 8.8e-8 with values rounded once, 5.7e-8 so;
// 5.8e-8 for the row-by-row contraction).
__device__ __forceinline__ void pair3(const Nl1Args& A, double v0, double v1, double& t00, double& t01, double& t11) {
  t00 = fma(A.far, v1, A.near * v0);
  t11 = fma(A.far, v0, A.near * v1);
  t01 = v0 + v1;
}
__device__ __forceinline__ void pair3(const Nl1Args& A, float v0, float v1, float& t00, float& t01, float& t11) {
  const float (&m)[3][2] = A.m32;
  const float s = v0 + v1;
  t00 = fmaf(m[2][0], v1, fmaf(m[0][0], v0, fmaf(m[0][1], v0, m[2][1] * v1)));
  t11 = fmaf(m[0][0], v1, fmaf(m[2][0], v0, fmaf(m[0][1], v1, m[2][1] * v0)));
  t01 = fmaf(m[1][0], s, m[1][1] * s);
}

// JT: type of the 54 numbers.  CT: type of the fields at the Gauss points (double whenever the residual is
// formed; float for the FP32 Jacobian alone).
template <typename JT, typename CT, bool DOJ, bool DOR>
__global__ void __launch_bounds__(CT_) k_nl1_cell(const __grid_constant__ Nl1Args A, const double* __restrict__ u_,
                                                  JT* __restrict__ zbuf, double* __restrict__ rbuf) {
  const int64_t cl = A.c0 + (int64_t)blockIdx.x * CT_ + threadIdx.x;
  if (cl >= A.c1) return;
  const Grid& g = A.g;
  const unsigned c32 = (unsigned)cl, t = c32 / (unsigned)g.nc[0];  // n_cells < n_dofs <= INT32_MAX
  const int cx = (int)(c32 - t * (unsigned)g.nc[0]), cz = (int)(t / (unsigned)g.nc[1]);
  const int cy = (int)(t - (unsigned)cz * (unsigned)g.nc[1]);
  const int64_t NX = g.nn[0], plane = NX * g.nn[1];
  const int64_t n0 = cx + NX * cy + plane * cz;
  const CT be = beta_of<CT>(A);
  // u at the Gauss points; differences at the Gauss points of the other two axes
  CT u[2][2][2], gd[3][2][2];
  {
    CT v[2][2][2], X[2][2][2], Y[2][2][2], dx[2][2], dy[2][2];  // [z][y][x]
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k >> 2][(k >> 1) & 1][k & 1] = (CT)__ldg(u_ + n0 + (k & 1) + NX * ((k >> 1) & 1) + plane * (k >> 2));
#pragma unroll
    for (int z = 0; z < 2; ++z)
#pragma unroll
      for (int y = 0; y < 2; ++y) lerp2(be, v[z][y][0], v[z][y][1], X[z][y][0], X[z][y][1], dx[z][y]);
#pragma unroll
    for (int z = 0; z < 2; ++z)
#pragma unroll
      for (int x = 0; x < 2; ++x) lerp2(be, X[z][0][x], X[z][1][x], Y[z][0][x], Y[z][1][x], dy[z][x]);
#pragma unroll
    for (int y = 0; y < 2; ++y)
#pragma unroll
      for (int x = 0; x < 2; ++x) lerp2(be, Y[0][y][x], Y[1][y][x], u[0][y][x], u[1][y][x], gd[2][y][x]);  // [qx], [qy]
    CT t[2][2], unused;
#pragma unroll
    for (int z = 0; z < 2; ++z) lerp2(be, dx[z][0], dx[z][1], t[z][0], t[z][1], unused);
#pragma unroll
    for (int y = 0; y < 2; ++y) lerp2(be, t[0][y], t[1][y], gd[0][0][y], gd[0][1][y], unused);  // [qz][qy]
#pragma unroll
    for (int x = 0; x < 2; ++x) lerp2(be, dy[0][x], dy[1][x], gd[1][0][x], gd[1][1][x], unused);  // [qz][qx]
  }
  // 2 + u^2 at the points of even x + y + z: each pair of neighbours has one of them
  CT c2[2][2][2];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int x = k & 1, y = (k >> 1) & 1, z = k >> 2;
    if ((x + y + z) % 2 == 0) c2[z][y][x] = fma(u[z][y][x], u[z][y][x], CT(2));
  }
  // element (first other axis p, second other axis q, own axis a) of a [z][y][x] array
  auto at = [](const auto& v, int a, int q, int p, int o) {
    const int x = a == 0 ? o : p, y = a == 0 ? p : (a == 1 ? o : q), z = a == 2 ? o : q;
    return v[z][y][x];
  };
  CT R[3][2][2];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    CT C[2][2];
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
      for (int p = 0; p < 2; ++p) {  // sum of 1 + u^2 along the axis
        const int even = (p + q) & 1;
        const CT v = at(u, a, q, p, 1 - even);
        C[q][p] = fma(v, v, at(c2, a, q, p, even));
      }
    if constexpr (DOR) {
      CT m[2][2], unused;
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const CT f0 = mulr(C[q][0], gd[a][q][0]), d = fma(C[q][1], gd[a][q][1], -f0);
        m[q][0] = fma(be, d, f0);
        m[q][1] = fma((CT)A.alpha, d, f0);
      }
#pragma unroll
      for (int p = 0; p < 2; ++p) lerp2(be, m[0][p], m[1][p], R[a][0][p], R[a][1][p], unused);
    }
    if constexpr (DOJ) {
      const JT kj = slope_of<JT>(A);
      const JT w = wj_of<JT>(A, a), w2 = JT(2) * w;
      JT* out = zbuf + ((cl >> 5) * NZ_ + a * 18) * CB + (cl & 31);
      JT Z[2][2][2];  // [j][q][p]
#pragma unroll
      for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int p = 0; p < 2; ++p) {
          // u's sums along the axis against the end nodes: u is linear there, u(1) - u(0) = (1 - 2 beta) gd
          const JT gj = as<JT>(gd[a][q][p]), D = w2 * gj, Cj = w * as<JT>(C[q][p]);
          Z[0][q][p] = fma(D, fma(kj, gj, as<JT>(at(u, a, q, p, 0))), -Cj);
          Z[1][q][p] = fma(D, fma(-kj, gj, as<JT>(at(u, a, q, p, 1))), Cj);
        }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        JT P[2][3];
#pragma unroll
        for (int q = 0; q < 2; ++q) pair3(A, Z[j][q][0], Z[j][q][1], P[q][0], P[q][1], P[q][2]);
#pragma unroll
        for (int t = 0; t < 3; ++t) {
          JT o[3];
          pair3(A, P[0][t], P[1][t], o[0], o[1], o[2]);
#pragma unroll
          for (int s = 0; s < 3; ++s) out[(j * 9 + s * 3 + t) * CB] = o[s];  // [j][second other axis][first]
        }
      }
    }
  }
  if constexpr (DOR) {
#pragma unroll
    for (int l = 0; l < 8; ++l) {
      const int x = l & 1, y = (l >> 1) & 1, z = l >> 2;
      CT v = fma(w_of<CT>(A, 0), x ? R[0][z][y] : -R[0][z][y], (CT)(-A.load));
      v = fma(w_of<CT>(A, 1), y ? R[1][z][x] : -R[1][z][x], v);
      v = fma(w_of<CT>(A, 2), z ? R[2][y][x] : -R[2][y][x], v);
      rbuf[((cl >> 5) * 8 + l) * CB + (cl & 31)] = v;
    }
  }
}

// FP64: 4 CTAs per SM (128 registers): 27 accumulators and a cell's 24 loads in flight; FP32 needs 80 registers
template <typename JT, bool DOJ, bool DOR, bool OVW>
__global__ void __launch_bounds__(RT, !DOJ ? 8 : (sizeof(JT) == 4 ? 6 : 4))
    k_nl1_row(const Grid g, int64_t row0, int64_t row1, const JT* __restrict__ zbuf, const double* __restrict__ rbuf,
              double* __restrict__ r, JT* __restrict__ J) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int64_t s_seg[2];
  const int64_t n0 = row0 + (int64_t)blockIdx.x * RT, n = n0 + threadIdx.x;
  const int64_t nend = n0 + RT < row1 ? n0 + RT : row1;
  const bool active = n < row1;
  const int NX = g.nn[0], NY = g.nn[1], NZ = g.nn[2];
  int ix = 0, iy = 0, iz = 0, cx = 1, cy = 1, cz = 1;
  int64_t row = 0;
  if (active) {
    mrgdev::decompose(g, n, ix, iy, iz);
    int lo;
    axis_range(ix, NX, 1, lo, cx);
    axis_range(iy, NY, 1, lo, cy);
    axis_range(iz, NZ, 1, lo, cz);
    const int64_t px = max(3 * ix - 1, 0), py = max(3 * iy - 1, 0), pz = max(3 * iz - 1, 0);
    row = pz * g.T[1] * g.T[0] + (int64_t)cz * (py * g.T[0] + (int64_t)cy * px);
  }
  int64_t seg0 = 0, seg1 = 0;
  JT* sv = nullptr;
  if constexpr (DOJ) {
    if (threadIdx.x == 0) s_seg[0] = row;
    if (n == nend - 1) s_seg[1] = row + cx * cy * cz;
    __syncthreads();
    seg0 = s_seg[0];
    seg1 = s_seg[1];
    sv = reinterpret_cast<JT*>(smem_raw) + (int)(((uintptr_t)(J + seg0) & 15) / sizeof(JT));
  }
  const bool fixed = active && node_fixed(g, ix, iy, iz);
  int64_t diag = 0;
  if (active) {
    JT acc[DOJ ? 27 : 1];
    double res = DOR && !OVW ? r[n] : 0.0;
    if constexpr (DOJ)
#pragma unroll
      for (int k = 0; k < 27; ++k) acc[k] = JT(0);
    if (!fixed) {
#pragma unroll
      for (int s = 0; s < 8; ++s) {
        const int sx = s & 1, sy = (s >> 1) & 1, sz = s >> 2;  // the cell on the right of the node along an axis
        const int ccx = ix - 1 + sx, ccy = iy - 1 + sy, ccz = iz - 1 + sz;
        if (ccx >= 0 && ccx < g.nc[0] && ccy >= 0 && ccy < g.nc[1] && ccz >= 0 && ccz < g.nc[2]) {
          const int64_t c = ccx + (int64_t)g.nc[0] * (ccy + (int64_t)g.nc[1] * ccz);
          const int l[3] = {1 - sx, 1 - sy, 1 - sz};
          if constexpr (DOR) res = addr(res, -__ldg(rbuf + ((c >> 5) * 8 + l[0] + 2 * l[1] + 4 * l[2]) * CB + (c & 31)));
          if constexpr (DOJ) {
            const JT* z = zbuf + (c >> 5) * (NZ_ * CB) + (c & 31);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const int jj[3] = {j & 1, (j >> 1) & 1, j >> 2};
              const int t[3] = {l[0] + jj[0], l[1] + jj[1], l[2] + jj[2]};  // 00, 01, 11
              // the cell's entry first, then the row's sum: fewer roundings at the size of the sum
              JT v = JT(0);
#pragma unroll
              for (int a = 0; a < 3; ++a) {
                const int p = a == 0 ? 1 : 0, q = a == 2 ? 1 : 2;
                const JT x = __ldg(z + (a * 18 + jj[a] * 9 + t[q] * 3 + t[p]) * CB);
                if (a == 0) v = l[a] ? x : -x;
                else v += l[a] ? x : -x;
              }
              acc[(jj[2] - l[2] + 1) * 9 + (jj[1] - l[1] + 1) * 3 + (jj[0] - l[0] + 1)] += v;
            }
          }
        }
      }
    }
    if constexpr (DOJ) {
      JT* out = sv + (row - seg0);
      if (cx == 3 && cy == 3 && cz == 3 && !fixed) {
#pragma unroll
        for (int k = 0; k < 27; ++k) out[k] = acc[k];
      } else {
        int pos = 0;
#pragma unroll
        for (int k = 0; k < 27; ++k) {
          const int ox = k % 3 - 1, oy = k / 3 % 3 - 1, oz = k / 9 - 1;
          if (ix + ox >= 0 && ix + ox < NX && iy + oy >= 0 && iy + oy < NY && iz + oz >= 0 && iz + oz < NZ) {
            if (k == 13) diag = pos;
            out[pos++] = (OVW && fixed && k == 13) ? JT(1) : acc[k];
          }
        }
      }
    }
    if (DOR) r[n] = res;
  }
  if constexpr (DOJ) {
    if (OVW) {
      mrgdev::fence_to_bulk();
      __syncthreads();
      mrgdev::seg_store_bulk<JT>(J + seg0, sv, seg1 - seg0);
    } else {
      __syncthreads();
      mrgdev::seg_store<JT, true>(J + seg0, sv, seg1 - seg0);
      __syncthreads();
      if (fixed) J[row + diag] = JT(1);
    }
  }
}

inline unsigned nblk(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

struct Nl1 {
  Nl1Args A;
};

template <typename JT>
cudaError_t launch(const mrg_problem* p, const Nl1Args& A, const MrgPiece& q, const double* u, double* r, JT* J, JT* z,
                   double* rb, bool doJ, bool doR, bool ovw, cudaStream_t s) {
  const unsigned gc = nblk(q.cell1 - q.cell0, CT_), gr = nblk(q.row1 - q.row0, RT);
  if (doJ && doR) k_nl1_cell<JT, double, true, true><<<gc, CT_, 0, s>>>(A, u, z, rb);
  else if (doJ) k_nl1_cell<JT, JT, true, false><<<gc, CT_, 0, s>>>(A, u, z, rb);
  else k_nl1_cell<double, double, false, true><<<gc, CT_, 0, s>>>(A, u, nullptr, rb);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  const int smem = doJ ? (RT * 27 + 16 / (int)sizeof(JT)) * (int)sizeof(JT) : 0;
#define MRG_NL1_ROW(DJ, DR, OV) k_nl1_row<JT, DJ, DR, OV><<<gr, RT, smem, s>>>(p->g, q.row0, q.row1, z, rb, r, J)
  if (doJ && doR) { if (ovw) MRG_NL1_ROW(true, true, true); else MRG_NL1_ROW(true, true, false); }
  else if (doJ) { if (ovw) MRG_NL1_ROW(true, false, true); else MRG_NL1_ROW(true, false, false); }
  else { if (ovw) MRG_NL1_ROW(false, true, true); else MRG_NL1_ROW(false, true, false); }
#undef MRG_NL1_ROW
  return cudaGetLastError();
}

}  // namespace

int mrg_nl1_setup(mrg_problem* p) {
  Nl1* Q = new Nl1();
  p->nl1 = Q;
  Nl1Args& A = Q->A;
  A.g = p->g;
  double l[2], dl[2];
  mrg_lagrange_1d(1, p->gx1[0], l, dl);
  A.beta = l[1];
  A.alpha = l[0];
  A.slope = l[1] * (l[0] - l[1]);
  A.betaf = (float)A.beta;
  A.slopef = (float)A.slope;
  const double m[3] = {l[0] * l[0], l[0] * l[1], l[1] * l[1]};
  A.near = l[0] / l[1];
  A.far = l[1] / l[0];
  for (int k = 0; k < 3; ++k) {
    A.m32[k][0] = (float)m[k];
    A.m32[k][1] = (float)(m[k] - (double)A.m32[k][0]);
  }
  double vol = 1.0;
  for (int a = 0; a < 3; ++a) vol *= 0.5 * p->h[a] * p->gw1[0];  // both weights are 1
  for (int a = 0; a < 3; ++a) {
    A.w[a] = vol / (p->h[a] * p->h[a]);
    A.wf[a] = (float)A.w[a];
    A.wj[a] = A.w[a] * (m[1] * m[1]);
  }
  A.load = p->source_amp * vol;  // the 8 basis values at the 8 equal-weight points add up to 1 for each node
  return mrg_ws_open(p);
}

void mrg_nl1_free(mrg_problem* p) {
  delete reinterpret_cast<Nl1*>(p->nl1);
  p->nl1 = nullptr;
}

int mrg_launch_nl1(mrg_problem* p, const double* u, double* r, void* J, uint32_t flags, cudaStream_t s) {
  const Nl1Args& A = reinterpret_cast<Nl1*>(p->nl1)->A;
  const bool doJ = flags & MRG_ASM_JAC, doR = flags & MRG_ASM_RES, ovw = flags & MRG_ASM_OVERWRITE;
  const bool fp32 = flags & MRG_ASM_J_FP32;
  const size_t zblock = doJ ? (size_t)CB * NZ_ * (fp32 ? sizeof(float) : sizeof(double)) : 0;
  const size_t rblock = doR ? (size_t)CB * 8 * sizeof(double) : 0;
  return mrg_in_pieces(p, zblock + rblock, s, [&](const MrgPiece& q) {
    Nl1Args Q = A;
    Q.c0 = q.cell0;
    Q.c1 = q.cell1;
    double* rb = mrg_piece_array<double>(q.ws + q.blocks * zblock, q, 8 * CB);
    return fp32 && doJ
               ? launch<float>(p, Q, q, u, r, (float*)J, mrg_piece_array<float>(q.ws, q, NZ_ * CB), rb, doJ, doR, ovw, s)
               : launch<double>(p, Q, q, u, r, (double*)J, mrg_piece_array<double>(q.ws, q, NZ_ * CB), rb, doJ, doR, ovw, s);
  });
}
