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
// entries: about 250 operations, and 2 additions an entry when the rows gather them (the row-by-row contraction
// took about 200 operations a row and cell, 1600 a cell).  The residual shares c and d_a with it: about 150
// operations a cell against 360 with one lane per Gauss point.
//
//   k_nl1_cell   one thread a cell: the 54 numbers (and the 8 residual entries) to a workspace in blocks of 32
//                cells, so that lanes write and read consecutive addresses and every offset is an immediate; or,
//                residual only, coloured read-modify-write into r (no workspace: such calls may overlap on
//                streams)
//   k_nl1_row    one thread a CSR row: 24 loads from each of its 8 cells, the CTA's rows staged in shared memory
//                and written once
#include <cmath>

#include "mrg_device.cuh"
#include "mrg_fixmul.cuh"
#include "mrg_internal.h"

namespace {

constexpr int CT_ = 128;  // cells per CTA
constexpr int RT = 128;   // rows per CTA
constexpr int NZ_ = 54;   // numbers per cell
constexpr int CB = 32;    // cells per workspace block

// products and sums that must not be contracted differently from one instance to the next (the residual of the
// separate and of the fused call has the same bits)
__device__ __forceinline__ double mulr(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mulr(float a, float b) { return __fmul_rn(a, b); }
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
  double w[3];       // |J| w_q / h_a^2
  double load;       // f * int(phi_l) over one cell
  float betaf, wf[3];
  int color, cc0, cc1;  // coloured launch: its colour and cells per axis; color < 0: all cells
  int64_t ncl;
};

template <typename T>
__device__ __forceinline__ T beta_of(const Nl1Args& A) {
  if constexpr (sizeof(T) == 4) return A.betaf; else return A.beta;
}
template <typename T>
__device__ __forceinline__ T w_of(const Nl1Args& A, int a) {
  if constexpr (sizeof(T) == 4) return A.wf[a]; else return A.w[a];
}

// values at the two Gauss points from two nodes, or node sums from two Gauss points (the 2 x 2 table is
// symmetric); d is the difference
template <typename T>
__device__ __forceinline__ void lerp2(T beta, T a, T b, T& p0, T& p1, T& d) {
  d = addr(b, -a);
  p0 = fma(beta, d, a);
  p1 = fma(-beta, d, b);
}

// sums of two Gauss points' values against L[q][l] L[q][j]: (00, 01, 11)
template <typename T>
__device__ __forceinline__ void pair3(T aa, T bb, T ab, T v0, T v1, T& t00, T& t01, T& t11) {
  t00 = fma(bb, v1, aa * v0);
  t11 = fma(aa, v1, bb * v0);
  t01 = ab * (v0 + v1);
}

// JT: type of the 54 numbers.  CT: type of the fields at the Gauss points (double whenever the residual is
// formed; float for the FP32 Jacobian alone).
template <typename JT, typename CT, bool DOJ, bool DOR>
__global__ void __launch_bounds__(CT_) k_nl1_cell(const __grid_constant__ Nl1Args A, const double* __restrict__ u_,
                                                  double* __restrict__ r, JT* __restrict__ zbuf,
                                                  double* __restrict__ rbuf) {
  const int64_t cl = (int64_t)blockIdx.x * CT_ + threadIdx.x;
  if (cl >= A.ncl) return;
  const Grid& g = A.g;
  const unsigned c32 = (unsigned)cl;  // n_cells < n_dofs <= INT32_MAX
  int cx, cy, cz;
  if (A.color < 0) {
    const unsigned t = c32 / (unsigned)g.nc[0];
    cx = (int)(c32 - t * (unsigned)g.nc[0]);
    cz = (int)(t / (unsigned)g.nc[1]);
    cy = (int)(t - (unsigned)cz * (unsigned)g.nc[1]);
  } else {
    const unsigned t = c32 / (unsigned)A.cc0, tz = t / (unsigned)A.cc1;
    cx = 2 * (int)(c32 - t * (unsigned)A.cc0) + (A.color & 1);
    cy = 2 * (int)(t - tz * (unsigned)A.cc1) + ((A.color >> 1) & 1);
    cz = 2 * (int)tz + ((A.color >> 2) & 1);
  }
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
  CT cw[2][2][2];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const CT q = u[k >> 2][(k >> 1) & 1][k & 1];
    cw[k >> 2][(k >> 1) & 1][k & 1] = fma(q, q, CT(1));
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
      for (int p = 0; p < 2; ++p) C[q][p] = mulr(w_of<CT>(A, a), addr(at(cw, a, q, p, 0), at(cw, a, q, p, 1)));
    if constexpr (DOR) {
      CT m[2][2], unused;
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const CT f0 = mulr(C[q][0], gd[a][q][0]), f1 = mulr(C[q][1], gd[a][q][1]);
        lerp2(be, f0, f1, m[q][0], m[q][1], unused);
      }
#pragma unroll
      for (int p = 0; p < 2; ++p) lerp2(be, m[0][p], m[1][p], R[a][0][p], R[a][1][p], unused);
    }
    if constexpr (DOJ) {
      const JT bj = beta_of<JT>(A), al = JT(1) - bj, aa = al * al, bb = bj * bj, ab = al * bj;
      const JT w2 = JT(2) * w_of<JT>(A, a);
      JT* out = zbuf + ((cl >> 5) * NZ_ + a * 18) * CB + (cl & 31);
      JT Z[2][2][2];  // [j][q][p]
#pragma unroll
      for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int p = 0; p < 2; ++p) {
          JT U[2], unused;
          lerp2(bj, as<JT>(at(u, a, q, p, 0)), as<JT>(at(u, a, q, p, 1)), U[0], U[1], unused);
          const JT D = w2 * as<JT>(gd[a][q][p]), Cj = as<JT>(C[q][p]);
          Z[0][q][p] = fma(D, U[0], -Cj);
          Z[1][q][p] = fma(D, U[1], Cj);
        }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        JT P[2][3];
#pragma unroll
        for (int q = 0; q < 2; ++q) pair3(aa, bb, ab, Z[j][q][0], Z[j][q][1], P[q][0], P[q][1], P[q][2]);
#pragma unroll
        for (int t = 0; t < 3; ++t) {
          JT o[3];
          pair3(aa, bb, ab, P[0][t], P[1][t], o[0], o[1], o[2]);
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
      CT v = addr(x ? R[0][z][y] : -R[0][z][y], (CT)(-A.load));
      v = addr(v, y ? R[1][z][x] : -R[1][z][x]);
      v = addr(v, z ? R[2][y][x] : -R[2][y][x]);
      if constexpr (DOJ) {
        rbuf[((cl >> 5) * 8 + l) * CB + (cl & 31)] = v;
      } else {
        if (!node_fixed(g, cx + x, cy + y, cz + z)) {
          double* p = r + n0 + x + NX * y + plane * z;
          *p = addr(*p, -v);  // r += -res.val()
        }
      }
    }
  }
}

// 4 CTAs per SM (128 registers): 27 accumulators and a cell's 24 loads in flight
template <typename JT, bool DOR, bool OVW>
__global__ void __launch_bounds__(RT, 4) k_nl1_row(const Grid g, int64_t nrows, const JT* __restrict__ zbuf,
                                                   const double* __restrict__ rbuf, double* __restrict__ r,
                                                   JT* __restrict__ J) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int64_t s_seg[2];
  const int64_t n0 = (int64_t)blockIdx.x * RT, n = n0 + threadIdx.x;
  const int64_t nend = n0 + RT < nrows ? n0 + RT : nrows;
  const bool active = n < nrows;
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
  if (threadIdx.x == 0) s_seg[0] = row;
  if (n == nend - 1) s_seg[1] = row + cx * cy * cz;
  __syncthreads();
  const int64_t seg0 = s_seg[0], seg1 = s_seg[1];
  const int phase = (int)(((uintptr_t)(J + seg0) & 15) / sizeof(JT));
  JT* sv = reinterpret_cast<JT*>(smem_raw) + phase;
  const bool fixed = active && node_fixed(g, ix, iy, iz);
  int64_t diag = 0;
  if (active) {
    JT acc[27];
#pragma unroll
    for (int k = 0; k < 27; ++k) acc[k] = JT(0);
    if (!fixed) {
#pragma unroll
      for (int s = 0; s < 8; ++s) {
        const int sx = s & 1, sy = (s >> 1) & 1, sz = s >> 2;  // the cell on the right of the node along an axis
        const int ccx = ix - 1 + sx, ccy = iy - 1 + sy, ccz = iz - 1 + sz;
        if (ccx >= 0 && ccx < g.nc[0] && ccy >= 0 && ccy < g.nc[1] && ccz >= 0 && ccz < g.nc[2]) {
          const int64_t c = ccx + (int64_t)g.nc[0] * (ccy + (int64_t)g.nc[1] * ccz);
          const JT* z = zbuf + (c >> 5) * (NZ_ * CB) + (c & 31);
          const int l[3] = {1 - sx, 1 - sy, 1 - sz};
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int jj[3] = {j & 1, (j >> 1) & 1, j >> 2};
            const int t[3] = {l[0] + jj[0], l[1] + jj[1], l[2] + jj[2]};  // 00, 01, 11
            JT v = acc[(jj[2] - l[2] + 1) * 9 + (jj[1] - l[1] + 1) * 3 + (jj[0] - l[0] + 1)];
#pragma unroll
            for (int a = 0; a < 3; ++a) {
              const int p = a == 0 ? 1 : 0, q = a == 2 ? 1 : 2;
              const JT x = __ldg(z + (a * 18 + jj[a] * 9 + t[q] * 3 + t[p]) * CB);
              v += l[a] ? x : -x;
            }
            acc[(jj[2] - l[2] + 1) * 9 + (jj[1] - l[1] + 1) * 3 + (jj[0] - l[0] + 1)] = v;
          }
        }
      }
    }
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
    if (DOR) {
      double v = OVW ? 0.0 : r[n];
      if (!fixed) {
        // the cells in the order of the coloured launches: the same sum
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int ccx = ix - 1 + (((ix - 1) ^ k) & 1), ccy = iy - 1 + (((iy - 1) ^ (k >> 1)) & 1);
          const int ccz = iz - 1 + (((iz - 1) ^ (k >> 2)) & 1);
          if (ccx >= 0 && ccx < g.nc[0] && ccy >= 0 && ccy < g.nc[1] && ccz >= 0 && ccz < g.nc[2]) {
            const int64_t c = ccx + (int64_t)g.nc[0] * (ccy + (int64_t)g.nc[1] * ccz);
            const int l = (ix - ccx) + 2 * (iy - ccy) + 4 * (iz - ccz);
            v = addr(v, -__ldg(rbuf + ((c >> 5) * 8 + l) * CB + (c & 31)));
          }
        }
      }
      r[n] = v;
    }
  }
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

inline unsigned nblk(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

struct Nl1 {
  Nl1Args A;
  unsigned char* ws = nullptr;  // the cells' numbers, then their residual entries; grows to the largest request
  size_t ws_bytes = 0;
};

template <typename JT>
cudaError_t launch_rows(const mrg_problem* p, const JT* z, const double* rb, double* r, JT* J, bool doR, bool ovw,
                        cudaStream_t s) {
  const int smem = (RT * 27 + 16 / (int)sizeof(JT)) * (int)sizeof(JT);
  const unsigned grid = nblk(p->ndof, RT);
#define MRG_NL1_ROW(DR, OV) k_nl1_row<JT, DR, OV><<<grid, RT, smem, s>>>(p->g, p->ndof, z, rb, r, J)
  if (doR) { if (ovw) MRG_NL1_ROW(true, true); else MRG_NL1_ROW(true, false); }
  else { if (ovw) MRG_NL1_ROW(false, true); else MRG_NL1_ROW(false, false); }
#undef MRG_NL1_ROW
  return cudaGetLastError();
}

}  // namespace

bool mrg_nl1_eligible(int dim, int order, int kind, int source_kind, int points_per_axis, bool affine) {
  return affine && dim == 3 && order == 1 && kind == MRG_DIFFUSION_1PU2 && source_kind == MRG_SRC_CONST &&
         points_per_axis == 2;
}

int mrg_nl1_setup(mrg_problem* p) {
  Nl1* Q = new Nl1();
  p->nl1 = Q;
  Nl1Args& A = Q->A;
  A.g = p->g;
  double l[2], dl[2];
  mrg_lagrange_1d(1, p->gx1[0], l, dl);
  A.beta = l[1];
  A.betaf = (float)A.beta;
  double vol = 1.0;
  for (int a = 0; a < 3; ++a) vol *= 0.5 * p->h[a] * p->gw1[0];  // both weights are 1
  for (int a = 0; a < 3; ++a) {
    A.w[a] = vol / (p->h[a] * p->h[a]);
    A.wf[a] = (float)A.w[a];
  }
  A.load = p->source_amp * vol;  // the 8 basis values at the 8 equal-weight points add up to 1 for each node
  return MRG_OK;
}

void mrg_nl1_free(mrg_problem* p) {
  Nl1* Q = reinterpret_cast<Nl1*>(p->nl1);
  if (!Q) return;
  if (Q->ws) cudaFreeAsync(Q->ws, p->stream);
  delete Q;
  p->nl1 = nullptr;
}

int mrg_launch_nl1(mrg_problem* p, const double* u, double* r, void* J, uint32_t flags, cudaStream_t s) {
  Nl1& Q = *reinterpret_cast<Nl1*>(p->nl1);
  const bool doJ = flags & MRG_ASM_JAC, doR = flags & MRG_ASM_RES, ovw = flags & MRG_ASM_OVERWRITE;
  const bool fp32 = flags & MRG_ASM_J_FP32;
  Nl1Args A = Q.A;
  A.color = -1;
  A.cc0 = A.cc1 = 1;
  A.ncl = p->ncell;
  if (!doJ) {
    if (ovw) MRG_CUDA(cudaMemsetAsync(r, 0, p->ndof * sizeof(double), s));
    // 8 colours: no two cells of one launch share a node
    for (int c = 0; c < 8; ++c) {
      const int n[3] = {(p->g.nc[0] - (c & 1) + 1) / 2, (p->g.nc[1] - ((c >> 1) & 1) + 1) / 2,
                        (p->g.nc[2] - (c >> 2) + 1) / 2};
      A.color = c;
      A.cc0 = n[0];
      A.cc1 = n[1];
      A.ncl = (int64_t)n[0] * n[1] * n[2];
      if (A.ncl == 0) continue;
      k_nl1_cell<double, double, false, true><<<nblk(A.ncl, CT_), CT_, 0, s>>>(A, u, r, nullptr, nullptr);
      MRG_CUDA(cudaGetLastError());
    }
    return MRG_OK;
  }
  const int64_t blocks = (p->ncell + CB - 1) / CB;
  const size_t zbytes = (size_t)blocks * CB * NZ_ * (fp32 ? sizeof(float) : sizeof(double));
  const size_t need = zbytes + (doR ? (size_t)blocks * CB * 8 * sizeof(double) : 0);
  if (Q.ws_bytes < need) {
    if (Q.ws) cudaFreeAsync(Q.ws, s);
    Q.ws = nullptr;
    Q.ws_bytes = 0;
    MRG_CUDA(cudaMallocAsync(&Q.ws, need, s));
    Q.ws_bytes = need;
  }
  double* rb = reinterpret_cast<double*>(Q.ws + zbytes);
  const unsigned grid = nblk(p->ncell, CT_);
  if (fp32) {
    float* z = reinterpret_cast<float*>(Q.ws);
    if (doR) k_nl1_cell<float, double, true, true><<<grid, CT_, 0, s>>>(A, u, r, z, rb);
    else k_nl1_cell<float, float, true, false><<<grid, CT_, 0, s>>>(A, u, r, z, rb);
    MRG_CUDA(cudaGetLastError());
    MRG_CUDA(launch_rows<float>(p, z, rb, r, (float*)J, doR, ovw, s));
  } else {
    double* z = reinterpret_cast<double*>(Q.ws);
    if (doR) k_nl1_cell<double, double, true, true><<<grid, CT_, 0, s>>>(A, u, r, z, rb);
    else k_nl1_cell<double, double, true, false><<<grid, CT_, 0, s>>>(A, u, r, z, rb);
    MRG_CUDA(cudaGetLastError());
    MRG_CUDA(launch_rows<double>(p, z, rb, r, (double*)J, doR, ovw, s));
  }
  return MRG_OK;
}
