// Assembly from cell matrices with stored geometry: 1 + u^2 on Q1 hexahedra of general shape (or with a source that
// varies), 1 + u^2 on Q1 and Q2 quadrilaterals, and thermal Q2 quadrilaterals of general shape (reference:
// src/physics/thermal.cpp:71-165, src/managers/assembly/assemblyManager_jacres.hpp:121-630,
// assemblyManager_scatter.hpp:164-278; the geometry kept from setup is the reference's stored basis data,
// assemblyManager_groups.hpp:396-398, :476-513).
//
// Of a cell's geometry the residual needs, at each Gauss point q, only the symmetric metric
//     M_ab = w_q / |det J| (C^T C)_ab      (C the cofactors of the geometric Jacobian)
// and the node loads; both are computed once at creation.  With k = kappa_c or 1 + u^2 and reference gradients,
//     res_i  = sum_q k sum_ab M_ab d_a phi_i d_b u - load_i
//     J_ij   = sum_q k sum_ab M_ab d_a phi_i d_b phi_j  +  sum_q 2 u (sum_ab M_ab d_b u d_a phi_i) phi_j .
// FP64 arithmetic bounds these passes (1/64 of the FP32 rate), so the sums over the tensor-product points are taken
// axis by axis, one thread a cell (small meshes of quadrilaterals: one thread a cell and l_x): about 1000 operations for
// a Q1 hexahedron and 1500 for a Q2 quadrilateral, where forward differentiation row by row took about 7000 and 8500.
//
//   k_metric      (setup) one thread a Gauss point
//   k_cell_hex1,  one thread a cell: the cell matrix and residual to a workspace in blocks of 32 cells, so that
//   k_cell_quad   lanes write and read consecutive addresses
//   k_gather      one thread a CSR row: adds its cells' entries in a fixed order; rows staged in shared memory and
//                 written once
// Measured, FP64 Jacobian and residual: 47 x 45 x 50 hexahedra with every vertex moved 1783 -> 246 us (cells 220, FP64
// pipe 87 % active, rows 27).
// The workspace is taken from the device's pool in stream order for each call, so calls of one handle may overlap
// on several streams and may be captured; a mesh that would need more than MRG_PIECE_BYTES is worked on in pieces.
#include <cmath>
#include <type_traits>

#include "mrg_device.cuh"
#include "mrg_fixmul.cuh"
#include "mrg_internal.h"

namespace {

constexpr int CB = MRG_CELL_BLOCK;  // cells per workspace block
constexpr int CT_ = 64;    // cells per CTA (up to 255 registers a thread)
constexpr int RT = 128;    // rows per CTA of the gather

struct GenTab {  // 1-D tables at the Gauss points: values, derivatives, weights
  double l[3][3], d[3][3], w[3];
};

struct HexTab {  // Q1 hexahedra: weights of the pairs of nodes 00, 01, 11 at a Gauss point
  double near, far;  // 00 / 01, 11 / 01
  double scale;      // 2 (01)^2
};

struct GenArgs {
  Grid g;
  GenTab t;
  HexTab hex;
  const double* metric;  // [cell / 32][components * points][32]
  const double* bnode;   // node loads
  const double* kap;
  int thermal;
  int64_t c0, c1;        // cells of the launch
};

__host__ __device__ constexpr int ipow(int b, int e) { return e == 0 ? 1 : b * ipow(b, e - 1); }

template <int DIM, int P>
struct Gen {
  static constexpr int N1 = P + 1, NL = ipow(N1, DIM), NM = DIM * (DIM + 1) / 2;
  static constexpr int MROW = NM * NL;   // metric values per cell
};

__device__ __forceinline__ void cell_of(const Grid& g, int64_t c, int& cx, int& cy, int& cz) {
  const unsigned c32 = (unsigned)c, t = c32 / (unsigned)g.nc[0];
  cx = (int)(c32 - t * (unsigned)g.nc[0]);
  cz = (int)(t / (unsigned)g.nc[1]);
  cy = (int)(t - (unsigned)cz * (unsigned)g.nc[1]);
}

template <typename T>
__device__ __forceinline__ T as(double v) {
  if constexpr (sizeof(T) == 4) return mrgfix::f64_to_f32_rn(v);  // on the integer pipes
  else return v;
}

// ---- setup ----------------------------------------------------------------------------------------
struct MetricArgs {
  Grid g;
  GenTab t;
  double gx[3];          // 1-D Gauss points
  const double* vcoord;  // [vertex][dim], or null: uniform box
  double lo[3], h[3];
  int src_sin;
  double amp, freq;
  int64_t ncell;
  double* metric;
  double* fw;            // [point][cell]: source times w |det J|
};

template <int DIM, int P>
__global__ void __launch_bounds__(128) k_metric(const __grid_constant__ MetricArgs A) {
  constexpr int N1 = P + 1, NL = Gen<DIM, P>::NL, NV = 1 << DIM;
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t c = e % A.ncell;
  const int q = (int)(e / A.ncell);
  if (q >= NL) return;
  int cc[3];
  cell_of(A.g, c, cc[0], cc[1], cc[2]);
  const int qi[3] = {q % N1, q / N1 % N1, DIM == 3 ? q / (N1 * N1) : 0};
  double wq = 1.0;
#pragma unroll
  for (int k = 0; k < DIM; ++k) wq *= A.t.w[qi[k]];
  double Jm[DIM][DIM], xq[DIM];  // Jm[k][m] = dx_k / dxi_m
#pragma unroll
  for (int k = 0; k < DIM; ++k) {
    xq[k] = 0.0;
#pragma unroll
    for (int m = 0; m < DIM; ++m) Jm[k][m] = 0.0;
  }
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const int iv[3] = {v & 1, (v >> 1) & 1, v >> 2};
    double f[DIM], ps = 1.0;
#pragma unroll
    for (int k = 0; k < DIM; ++k) {
      f[k] = 0.5 * (iv[k] ? 1.0 + A.gx[qi[k]] : 1.0 - A.gx[qi[k]]);
      ps *= f[k];
    }
    const int64_t vid = (cc[0] + iv[0]) + (int64_t)(A.g.nc[0] + 1) * ((cc[1] + iv[1]) + (int64_t)(A.g.nc[1] + 1) * (cc[2] + iv[2]));
#pragma unroll
    for (int k = 0; k < DIM; ++k) {
      const double x = A.vcoord ? __ldg(A.vcoord + vid * DIM + k) : A.lo[k] + A.h[k] * (cc[k] + iv[k]);
      xq[k] = fma(x, ps, xq[k]);
#pragma unroll
      for (int m = 0; m < DIM; ++m) {
        double dp = iv[m] ? 0.5 : -0.5;
#pragma unroll
        for (int j = 0; j < DIM; ++j)
          if (j != m) dp *= f[j];
        Jm[k][m] = fma(x, dp, Jm[k][m]);
      }
    }
  }
  double C[DIM][DIM], det;
  if constexpr (DIM == 3) {
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        const int k1 = (k + 1) % 3, k2 = (k + 2) % 3, m1 = (m + 1) % 3, m2 = (m + 2) % 3;
        C[k][m] = Jm[k1][m1] * Jm[k2][m2] - Jm[k1][m2] * Jm[k2][m1];
      }
    det = Jm[0][0] * C[0][0] + Jm[0][1] * C[0][1] + Jm[0][2] * C[0][2];
  } else {
    C[0][0] = Jm[1][1];
    C[0][1] = -Jm[1][0];
    C[1][0] = -Jm[0][1];
    C[1][1] = Jm[0][0];
    det = Jm[0][0] * Jm[1][1] - Jm[0][1] * Jm[1][0];
  }
  const double ad = fabs(det), sc = (DIM == 3 ? 0.25 : 1.0) * (wq / ad);  // k_cell_hex1 uses a quarter of M
  double* out = A.metric + ((c >> 5) * Gen<DIM, P>::MROW + q) * CB + (c & 31);
  int k = 0;
#pragma unroll
  for (int a = 0; a < DIM; ++a)
#pragma unroll
    for (int b = a; b < DIM; ++b) {
      double s = 0.0;
#pragma unroll
      for (int i = 0; i < DIM; ++i) s = fma(C[i][a], C[i][b], s);
      out[(k++ * NL) * CB] = s * sc;  // 2-D: 00 01 11; 3-D: 00 01 02 11 12 22
    }
  double f = A.amp;
  if (A.src_sin) {
#pragma unroll
    for (int i = 0; i < DIM; ++i) f *= sin(A.freq * xq[i]);
  }
  A.fw[(int64_t)q * A.ncell + c] = f * wq * ad;
}

// b_i = sum over the node's cells (fixed order) of sum_q f w |det| phi_i
template <int DIM, int P>
__global__ void __launch_bounds__(128) k_loads(const __grid_constant__ MetricArgs A, int64_t nrows, double* __restrict__ b) {
  constexpr int N1 = P + 1, NL = Gen<DIM, P>::NL;
  const int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= nrows) return;
  int i[3], cf[3] = {0, 0, 0}, nc[3] = {1, 1, 1};
  mrgdev::decompose(A.g, n, i[0], i[1], i[2]);
#pragma unroll
  for (int k = 0; k < DIM; ++k) axis_cells(i[k], A.g.nn[k], P, cf[k], nc[k]);
  double s = 0.0;
  for (int z = cf[2]; z < cf[2] + nc[2]; ++z)
    for (int y = cf[1]; y < cf[1] + nc[1]; ++y)
      for (int x = cf[0]; x < cf[0] + nc[0]; ++x) {
        const int64_t c = x + (int64_t)A.g.nc[0] * (y + (int64_t)A.g.nc[1] * z);
        const int lx = i[0] - P * x, ly = i[1] - P * y, lz = DIM == 3 ? i[2] - P * z : 0;
        for (int q = 0; q < NL; ++q) {
          double ph = A.t.l[q % N1][lx] * A.t.l[q / N1 % N1][ly];
          if (DIM == 3) ph *= A.t.l[q / (N1 * N1)][lz];
          s = fma(ph, A.fw[(int64_t)q * A.ncell + c], s);
        }
      }
  b[n] = s;
}

// ---- Q1 hexahedra ----------------------------------------------------------------------------------
// A linear node's reference gradient along its own axis is the constant +-1/2, so with differences d_b in place of
// reference gradients a quarter of M is used (stored so), sigma = -1 or +1 stands for the derivative, and the
// weights of a pair of nodes at a Gauss point depend on the unordered pair alone (00, 01 or 11).
__device__ __forceinline__ void lerp2(double be, double a, double b, double& p0, double& p1, double& d) {
  d = __dadd_rn(b, -a);
  p0 = fma(be, d, a);
  p1 = fma(-be, d, b);
}
// the same of the values c0 g0 and c1 g1, al = 1 - be: an operation less
__device__ __forceinline__ void lerp2(double be, double al, double c0, double g0, double c1, double g1, double& p0, double& p1) {
  const double f0 = __dmul_rn(c0, g0), d = fma(c1, g1, -f0);
  p0 = fma(be, d, f0);
  p1 = fma(al, d, f0);
}
// Sums of two Gauss points' values against L[q][l] L[q][j]: (00, 01, 11), the pairs' weights w; and in units of the pair 01's
// weight (near = 00 / 01, far = 11 / 01), an operation less.
__device__ __forceinline__ void pair3(const double (&w)[3], double v0, double v1, double* t) {
  t[0] = fma(w[2], v1, w[0] * v0);
  t[1] = w[1] * (v0 + v1);
  t[2] = fma(w[2], v0, w[0] * v1);
}
__device__ __forceinline__ void pair3(double near, double far, double v0, double v1, double* t) {
  t[0] = fma(far, v1, near * v0);
  t[1] = v0 + v1;
  t[2] = fma(far, v0, near * v1);
}

template <typename JT, bool DOJ, bool DOR>
__global__ void __launch_bounds__(CT_) k_cell_hex1(const __grid_constant__ GenArgs A, const double* __restrict__ u_,
                                                   JT* __restrict__ ebuf, double* __restrict__ rbuf) {
  const int64_t c = A.c0 + (int64_t)blockIdx.x * CT_ + threadIdx.x;
  if (c >= A.c1) return;
  const Grid& g = A.g;
  int cx, cy, cz;
  cell_of(g, c, cx, cy, cz);
  const int64_t NX = g.nn[0], plane = NX * g.nn[1], n0 = cx + NX * cy + plane * cz;
  const double be = A.t.l[0][1], al = A.t.l[0][0];
  double u[8], gd[3][4];  // u at the points q = qx + 2 qy + 4 qz; differences at the points of the other two axes
  {
    double v[8], X[8], Y[8], dx[4], dy[4], t[4], unused;
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = __ldg(u_ + n0 + (k & 1) + NX * ((k >> 1) & 1) + plane * (k >> 2));
#pragma unroll
    for (int k = 0; k < 4; ++k) lerp2(be, v[2 * k], v[2 * k + 1], X[2 * k], X[2 * k + 1], dx[k]);  // k = y + 2 z
#pragma unroll
    for (int z = 0; z < 2; ++z)
#pragma unroll
      for (int x = 0; x < 2; ++x)
        lerp2(be, X[4 * z + x], X[4 * z + 2 + x], Y[4 * z + x], Y[4 * z + 2 + x], dy[x + 2 * z]);
#pragma unroll
    for (int k = 0; k < 4; ++k) lerp2(be, Y[k], Y[4 + k], u[k], u[4 + k], gd[2][k]);  // k = qx + 2 qy
#pragma unroll
    for (int z = 0; z < 2; ++z) lerp2(be, dx[2 * z], dx[2 * z + 1], t[2 * z], t[2 * z + 1], unused);
#pragma unroll
    for (int y = 0; y < 2; ++y) lerp2(be, t[y], t[2 + y], gd[0][y], gd[0][2 + y], unused);  // qy + 2 qz
#pragma unroll
    for (int x = 0; x < 2; ++x) lerp2(be, dy[x], dy[2 + x], gd[1][x], gd[1][2 + x], unused);  // qx + 2 qz
  }
  double k[8], h[3][8];
  const double* M = A.metric + (c >> 5) * (48 * CB) + (c & 31);
  auto m = [&](int comp, int q) { return __ldg(M + (comp * 8 + q) * CB); };  // 00 01 02 11 12 22
  auto comp = [](int a, int b) { return a == 0 ? b : a + b + 1; };  // a <= b
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int x = q & 1, y = (q >> 1) & 1, z = q >> 2;
    k[q] = fma(u[q], u[q], 1.0);
    const double d0 = gd[0][y + 2 * z], d1 = gd[1][x + 2 * z], d2 = gd[2][x + 2 * y];
    const double m01 = m(1, q), m02 = m(2, q), m12 = m(4, q);
    h[0][q] = fma(m(0, q), d0, fma(m01, d1, m02 * d2));
    h[1][q] = fma(m01, d0, fma(m(3, q), d1, m12 * d2));
    h[2][q] = fma(m02, d0, fma(m12, d1, m(5, q) * d2));
  }
  // the point with index o along axis a, p along the first and q along the second other axis
  auto pt = [](int a, int q, int p, int o) { return a == 0 ? o + 2 * p + 4 * q : (a == 1 ? p + 2 * o + 4 * q : p + 2 * q + 4 * o); };
  if constexpr (DOR) {
    double R[3][4];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      double s[2][2], unused;
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        double f[2];
#pragma unroll
        for (int p = 0; p < 2; ++p)
          f[p] = fma(k[pt(a, q, p, 1)], h[a][pt(a, q, p, 1)], __dmul_rn(k[pt(a, q, p, 0)], h[a][pt(a, q, p, 0)]));
        lerp2(be, f[0], f[1], s[q][0], s[q][1], unused);
      }
#pragma unroll
      for (int p = 0; p < 2; ++p) lerp2(be, s[0][p], s[1][p], R[a][p], R[a][2 + p], unused);
    }
    double* out = rbuf + (c >> 5) * (8 * CB) + (c & 31);
#pragma unroll
    for (int l = 0; l < 8; ++l) {
      const int x = l & 1, y = (l >> 1) & 1, z = l >> 2;
      const double a = x ? R[0][y + 2 * z] : -R[0][y + 2 * z], b = y ? R[1][x + 2 * z] : -R[1][x + 2 * z];
      const double d = z ? R[2][x + 2 * y] : -R[2][x + 2 * y];
      out[l * CB] = __dadd_rn(__dadd_rn(a, b), d);
    }
  }
  if constexpr (DOJ) {
    const double w[3] = {al * al, al * be, be * be};  // of the pairs 00, 01, 11
    // the same-axis parts' two sums over pairs leave the square of the pair 01's weight out (48 multiplications)
    const double near = A.hex.near, far = A.hex.far, sc = A.hex.scale, hs = 0.5 * sc;
    double E[64], su[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) su[q] = sc * u[q];
    // same-axis and advective parts: E[l][j] gets sigma(l_a) Z[j_a][pair b][pair c]
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      double Z[2][2][2];  // [j][q][p]
#pragma unroll
      for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int p = 0; p < 2; ++p) {
          const int q0 = pt(a, q, p, 0), q1 = pt(a, q, p, 1), ca = a == 0 ? 0 : (a == 1 ? 3 : 5);
          const double C = fma(k[q1], m(ca, q1), k[q0] * m(ca, q0));
          const double f0 = su[q0] * h[a][q0], d = fma(su[q1], h[a][q1], -f0);  // 2 u h
          Z[0][q][p] = fma(be, d, fma(-hs, C, f0));
          Z[1][q][p] = fma(al, d, fma(hs, C, f0));
        }
#pragma unroll
      for (int ja = 0; ja < 2; ++ja) {
        double Pq[2][3], T[3][3];  // T[pair of the first other axis][pair of the second]
        pair3(near, far, Z[ja][0][0], Z[ja][0][1], Pq[0]);
        pair3(near, far, Z[ja][1][0], Z[ja][1][1], Pq[1]);
#pragma unroll
        for (int t = 0; t < 3; ++t) pair3(near, far, Pq[0][t], Pq[1][t], T[t]);
        const int p = a == 0 ? 1 : 0, q = a == 2 ? 1 : 2;
#pragma unroll
        for (int l = 0; l < 8; ++l)
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            if (((j >> a) & 1) != ja) continue;
            const double t = T[((l >> p) & 1) + ((j >> p) & 1)][((l >> q) & 1) + ((j >> q) & 1)];
            const double v = ((l >> a) & 1) ? t : -t;
            E[l * 8 + j] = a == 0 ? v : E[l * 8 + j] + v;
          }
      }
    }
    // mixed-axis parts: X[i][j][pair c] = sum_q k M_ab L_i(q_a) L_j(q_b) (pair c); E[l][j] gets
    // sigma(l_a) sigma(j_b) X[j_a][l_b] + sigma(l_b) sigma(j_a) X[l_a][j_b]
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int b = a + 1; b < 3; ++b) {
        const int o = 3 - a - b;
        double V[2][2][2];  // [point of o][node of a][node of b]
#pragma unroll
        for (int qo = 0; qo < 2; ++qo) {
          double W[2][2], unused;  // [node of a][point of b]
#pragma unroll
          for (int qb = 0; qb < 2; ++qb) {
            const int q0 = (qb << b) | (qo << o), q1 = q0 | (1 << a);
            lerp2(be, al, k[q0], m(comp(a, b), q0), k[q1], m(comp(a, b), q1), W[0][qb], W[1][qb]);
          }
#pragma unroll
          for (int i = 0; i < 2; ++i) lerp2(be, W[i][0], W[i][1], V[qo][i][0], V[qo][i][1], unused);
        }
        double X[2][2][3];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int j = 0; j < 2; ++j) pair3(w, V[0][i][j], V[1][i][j], X[i][j]);
        // the 16 combinations of (l_a, j_a, l_b, j_b), each with its mirror (l and j exchanged) at once
#pragma unroll
        for (int s = 0; s < 16; ++s) {
          const int la = s & 1, ja = (s >> 1) & 1, lb = (s >> 2) & 1, jb = s >> 3;
          const int mir = ja | (la << 1) | (jb << 2) | (lb << 3);
          if (mir < s) continue;
#pragma unroll
          for (int t = 0; t < 3; ++t) {
            const double x1 = (la == jb) ? X[ja][lb][t] : -X[ja][lb][t], x2 = (lb == ja) ? X[la][jb][t] : -X[la][jb][t];
            const double y = x1 + x2;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int lo = e & 1, jo = e >> 1;
              if (lo + jo != t) continue;
              const int l = (la << a) | (lb << b) | (lo << o), j = (ja << a) | (jb << b) | (jo << o);
              E[l * 8 + j] += y;
              if (mir != s) {
                const int l2 = (ja << a) | (jb << b) | (lo << o), j2 = (la << a) | (lb << b) | (jo << o);
                E[l2 * 8 + j2] += y;
              }
            }
          }
        }
      }
    JT* out = ebuf + (c >> 5) * (64 * CB) + (c & 31);
#pragma unroll
    for (int e = 0; e < 64; ++e) out[e * CB] = as<JT>(E[e]);
  }
}

// ---- quadrilaterals --------------------------------------------------------------------------------
// Sums over q_x for each pair of x indices, then over q_y: an entry's terms have four kinds of factor along y
// (value or derivative of either function), so with a, b the combinations for the row's function
//     E[l][j] = sum_qy a(qy) L_{jy}(qy) + b(qy) D_{jy}(qy).
// SPLIT (small meshes): a thread forms the rows of one l_x, blockIdx.y.
template <int P, typename JT, bool DOJ, bool DOR, bool SPLIT>
__global__ void __launch_bounds__(CT_) k_cell_quad(const __grid_constant__ GenArgs A, const double* __restrict__ u_,
                                                   JT* __restrict__ ebuf, double* __restrict__ rbuf) {
  constexpr int N1 = P + 1, NL = N1 * N1;
  const int64_t c = A.c0 + (int64_t)blockIdx.x * CT_ + threadIdx.x;
  if (c >= A.c1) return;
  const Grid& g = A.g;
  const GenTab& T = A.t;
  int cx, cy, cz;
  cell_of(g, c, cx, cy, cz);
  const int64_t NX = g.nn[0], n0 = P * cx + NX * (P * cy);
  double k00[N1][N1], k01[N1][N1], k11[N1][N1], v0[N1][N1], v1[N1][N1];  // [qy][qx]
  double F0[N1][N1], F1[N1][N1];
  {
    double ux[N1][N1], dx[N1][N1];  // [node y][qx]
#pragma unroll
    for (int b = 0; b < N1; ++b) {
      double v[N1];
#pragma unroll
      for (int a = 0; a < N1; ++a) v[a] = __ldg(u_ + n0 + a + NX * b);
#pragma unroll
      for (int q = 0; q < N1; ++q) {
        double s = __dmul_rn(T.l[q][0], v[0]), d = __dmul_rn(T.d[q][0], v[0]);
#pragma unroll
        for (int a = 1; a < N1; ++a) {
          s = fma(T.l[q][a], v[a], s);
          d = fma(T.d[q][a], v[a], d);
        }
        ux[b][q] = s;
        dx[b][q] = d;
      }
    }
    const double kc = A.thermal ? __ldg(A.kap + c) : 0.0;
    const double* M = A.metric + (c >> 5) * (Gen<2, P>::MROW * CB) + (c & 31);
#pragma unroll
    for (int qy = 0; qy < N1; ++qy)
#pragma unroll
      for (int qx = 0; qx < N1; ++qx) {
        double uq = __dmul_rn(T.l[qy][0], ux[0][qx]), g0 = __dmul_rn(T.l[qy][0], dx[0][qx]), g1 = __dmul_rn(T.d[qy][0], ux[0][qx]);
#pragma unroll
        for (int b = 1; b < N1; ++b) {
          uq = fma(T.l[qy][b], ux[b][qx], uq);
          g0 = fma(T.l[qy][b], dx[b][qx], g0);
          g1 = fma(T.d[qy][b], ux[b][qx], g1);
        }
        const int q = qx + N1 * qy;
        const double m00 = __ldg(M + q * CB), m01 = __ldg(M + (NL + q) * CB), m11 = __ldg(M + (2 * NL + q) * CB);
        const double k = A.thermal ? kc : fma(uq, uq, 1.0);
        const double h0 = fma(m00, g0, __dmul_rn(m01, g1)), h1 = fma(m01, g0, __dmul_rn(m11, g1));
        F0[qy][qx] = __dmul_rn(k, h0);
        F1[qy][qx] = __dmul_rn(k, h1);
        k00[qy][qx] = k * m00;
        k01[qy][qx] = k * m01;
        k11[qy][qx] = k * m11;
        const double u2 = A.thermal ? 0.0 : 2.0 * uq;
        v0[qy][qx] = u2 * h0;
        v1[qy][qx] = u2 * h1;
      }
  }
  if (DOR && (!SPLIT || blockIdx.y == 0)) {
    double* out = rbuf + (c >> 5) * (NL * CB) + (c & 31);
#pragma unroll
    for (int lx = 0; lx < N1; ++lx) {
      double s0[N1], s1[N1];  // sums over q_x
#pragma unroll
      for (int qy = 0; qy < N1; ++qy) {
        s0[qy] = __dmul_rn(T.d[0][lx], F0[qy][0]);
        s1[qy] = __dmul_rn(T.l[0][lx], F1[qy][0]);
#pragma unroll
        for (int qx = 1; qx < N1; ++qx) {
          s0[qy] = fma(T.d[qx][lx], F0[qy][qx], s0[qy]);
          s1[qy] = fma(T.l[qx][lx], F1[qy][qx], s1[qy]);
        }
      }
#pragma unroll
      for (int ly = 0; ly < N1; ++ly) {
        double r = __dmul_rn(T.l[0][ly], s0[0]);
        r = fma(T.d[0][ly], s1[0], r);
#pragma unroll
        for (int qy = 1; qy < N1; ++qy) r = fma(T.d[qy][ly], s1[qy], fma(T.l[qy][ly], s0[qy], r));
        out[(lx + N1 * ly) * CB] = r;
      }
    }
  }
  if constexpr (DOJ) {
    JT* out = ebuf + (c >> 5) * (NL * NL * CB) + (c & 31);
    // not unrolled: the code of one (l_x, j_x) is already some hundred operations
    for (int lx = SPLIT ? (int)blockIdx.y : 0; lx < (SPLIT ? (int)blockIdx.y + 1 : N1); ++lx)
#pragma unroll 1
      for (int jx = 0; jx < N1; ++jx) {
        double LL[N1], DD[N1], LD[N1], DL[N1];  // factors along y: row's function first
#pragma unroll
        for (int qy = 0; qy < N1; ++qy) LL[qy] = DD[qy] = LD[qy] = DL[qy] = 0.0;
#pragma unroll
        for (int qx = 0; qx < N1; ++qx) {
          const double ll = T.l[qx][lx], dl = T.d[qx][lx], lj = T.l[qx][jx], dj = T.d[qx][jx];
          const double wdd = dl * dj, wdl = dl * lj, wld = ll * dj, wll = ll * lj;
#pragma unroll
          for (int qy = 0; qy < N1; ++qy) {
            LL[qy] = fma(wdl, v0[qy][qx], fma(wdd, k00[qy][qx], LL[qy]));
            DD[qy] = fma(wll, k11[qy][qx], DD[qy]);
            LD[qy] = fma(wdl, k01[qy][qx], LD[qy]);
            DL[qy] = fma(wll, v1[qy][qx], fma(wld, k01[qy][qx], DL[qy]));
          }
        }
#pragma unroll
        for (int ly = 0; ly < N1; ++ly) {
          double e[N1];
#pragma unroll
          for (int jy = 0; jy < N1; ++jy) e[jy] = 0.0;
#pragma unroll
          for (int qy = 0; qy < N1; ++qy) {
            const double a = fma(T.l[qy][ly], LL[qy], T.d[qy][ly] * DL[qy]);
            const double b = fma(T.l[qy][ly], LD[qy], T.d[qy][ly] * DD[qy]);
#pragma unroll
            for (int jy = 0; jy < N1; ++jy) e[jy] = fma(T.l[qy][jy], a, fma(T.d[qy][jy], b, e[jy]));
          }
#pragma unroll
          for (int jy = 0; jy < N1; ++jy)
            out[((lx + N1 * ly) * NL + jx + N1 * jy) * CB] = as<JT>(e[jy]);
        }
      }
  }
}

// ---- rows ------------------------------------------------------------------------------------------
// Row lengths of a CTA's 128 rows fit the staged segment; entries are added cell by cell (cz, cy, cx order) at
// positions computed from the row's extents.
// With entries, 64 registers for 8 CTAs per SM (as many as their staged rows leave room for): left to itself the compiler
// took 32 to 48 and loaded an element row in parts (300 x 400 Q2 quadrilaterals, FP64 Jacobian and residual, 504 us -> 500;
// with the bounds of a piece among the arguments and 32 registers 522).
template <int DIM, int P, typename JT, bool DOJ, bool DOR, bool OVW>
__global__ void __launch_bounds__(RT, DOJ ? 8 : 0) k_gather(const Grid g, int64_t row0, int64_t row1, const JT* __restrict__ ebuf,
                                               const double* __restrict__ rbuf, const double* __restrict__ bnode,
                                               double* __restrict__ r, JT* __restrict__ J) {
  constexpr int N1 = P + 1, NL = Gen<DIM, P>::NL;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int64_t s_seg[2];
  const int64_t n0 = row0 + (int64_t)blockIdx.x * RT, n = n0 + threadIdx.x;
  const int64_t nend = n0 + RT < row1 ? n0 + RT : row1;
  const bool active = n < row1;
  int ix = 0, iy = 0, iz = 0;
  mrgdev::RowInfo R{0, 0, 0, 1, 1, 1, 0};
  if (active) {
    mrgdev::decompose(g, n, ix, iy, iz);
    R = mrgdev::row_info<P>(g, ix, iy, iz);
  }
  const int len = R.cx * R.cy * R.cz;
  const bool fixed = active && node_fixed(g, ix, iy, iz);
  int64_t seg0 = 0, seg1 = 0;
  JT* sv = nullptr;
  JT* row = nullptr;
  if constexpr (DOJ) {
    if (threadIdx.x == 0) s_seg[0] = R.rp;
    if (n == nend - 1) s_seg[1] = R.rp + len;
    __syncthreads();
    seg0 = s_seg[0];
    seg1 = s_seg[1];
    sv = reinterpret_cast<JT*>(smem_raw) + (int)(((uintptr_t)(J + seg0) & 15) / sizeof(JT));
    row = sv + (R.rp - seg0);
  }
  const int diag = ((iz - R.lz) * R.cy + (iy - R.ly)) * R.cx + (ix - R.lx);
  if (active) {
    if constexpr (DOJ) {
      for (int k = 0; k < len; ++k) row[k] = JT(0);
      if (OVW && fixed) row[diag] = JT(1);
    }
    if (!fixed) {
      int cf[3] = {0, 0, 0}, nc[3] = {1, 1, 1};
      axis_cells(ix, g.nn[0], P, cf[0], nc[0]);
      axis_cells(iy, g.nn[1], P, cf[1], nc[1]);
      if (DIM == 3) axis_cells(iz, g.nn[2], P, cf[2], nc[2]);
      double acc = DOR ? __ldg(bnode + n) : 0.0;
      for (int z = cf[2]; z < cf[2] + nc[2]; ++z)
        for (int y = cf[1]; y < cf[1] + nc[1]; ++y)
          for (int x = cf[0]; x < cf[0] + nc[0]; ++x) {
            const int64_t c = x + (int64_t)g.nc[0] * (y + (int64_t)g.nc[1] * z);
            const int l = (ix - P * x) + N1 * (iy - P * y) + (DIM == 3 ? N1 * N1 * (iz - P * z) : 0);
            if constexpr (DOR) acc = __dadd_rn(acc, -__ldg(rbuf + ((c >> 5) * NL + l) * CB + (c & 31)));
            if constexpr (DOJ) {
              const JT* e = ebuf + ((c >> 5) * (NL * NL) + l * NL) * CB + (c & 31);
              JT v[NL];
#pragma unroll
              for (int j = 0; j < NL; ++j) v[j] = __ldg(e + j * CB);
              JT* at = row + ((DIM == 3 ? P * z - R.lz : 0) * R.cy + (P * y - R.ly)) * R.cx + (P * x - R.lx);
#pragma unroll
              for (int j = 0; j < NL; ++j)
                at[((DIM == 3 ? j / (N1 * N1) : 0) * R.cy + j / N1 % N1) * R.cx + j % N1] += v[j];
            }
          }
      if constexpr (DOR) {
        if (OVW) r[n] = acc; else r[n] += acc;
      }
    } else if (DOR && OVW) {
      r[n] = 0.0;
    }
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
      if (fixed) J[R.rp + diag] = JT(1);
    }
  }
}

inline unsigned nblk(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

struct General {
  GenArgs A;
  double* d_metric = nullptr;
  double* d_bnode = nullptr;
};

template <int DIM, int P>
int setup_t(mrg_problem* p, General* Q, MetricArgs& M, cudaStream_t s) {
  using K = Gen<DIM, P>;
  const int64_t blocks = (p->ncell + CB - 1) / CB;
  double* fw = nullptr;
  MRG_CUDA(cudaMallocAsync(&Q->d_metric, (size_t)blocks * CB * K::MROW * sizeof(double), s));
  MRG_CUDA(cudaMallocAsync(&Q->d_bnode, (size_t)p->ndof * sizeof(double), s));
  MRG_CUDA(cudaMallocAsync(&fw, (size_t)p->ncell * K::NL * sizeof(double), s));
  M.metric = Q->d_metric;
  M.fw = fw;
  k_metric<DIM, P><<<nblk(p->ncell * K::NL, 128), 128, 0, s>>>(M);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) {
    k_loads<DIM, P><<<nblk(p->ndof, 128), 128, 0, s>>>(M, p->ndof, Q->d_bnode);
    e = cudaGetLastError();
  }
  cudaFreeAsync(fw, s);
  return e == cudaSuccess ? MRG_OK : mrg_cuda_check(e, "cell geometry launch");
}

// FP64 work issues at 64 cycles a warp instruction on each of an SM's four schedulers, so a mesh with fewer cells than
// 32 lanes on all of them (19456 on 152 SMs) leaves schedulers idle and takes a cell's whole chain.  A quadrilateral's
// matrix is then split by its rows over P + 1 threads, each forming the fields again, as long as that gives a scheduler
// two warps at most (Q2).  FP64 Jacobian and residual, whole -> split: Q2, 60 x 60 cells 86 -> 57 us, 100 x 100 94 -> 85,
// 120 x 120 95 -> 104; Q1, 60 x 60 36 -> 31, 120 x 120 37.7 -> 36.8, 139 x 139 38 -> 42.  A hexahedron's rows share too
// much: one axis's and one mixed part a thread with the parts added by the gather took 62 us against 50 on 20 x 22 x 19.
constexpr int64_t FILL = 32 * 4 * 2 / 3 - 1;  // cells per SM

template <int DIM, int P, typename JT, bool SPLIT>
cudaError_t launch_t(const mrg_problem* p, const General& Q, const MrgPiece& q, const double* u, double* r, JT* J, JT* ebuf,
                     double* rbuf, bool doJ, bool doR, bool ovw, cudaStream_t s) {
  const dim3 gc(nblk(q.cell1 - q.cell0, CT_), SPLIT && doJ ? P + 1 : 1);
  const unsigned gr = nblk(q.row1 - q.row0, RT);
  GenArgs A = Q.A;
  A.c0 = q.cell0;
  A.c1 = q.cell1;
#define MRG_GEN_CELL(DJ, DR, SP)                                                              \
  if constexpr (DIM == 3) k_cell_hex1<JT, DJ, DR><<<gc, CT_, 0, s>>>(A, u, ebuf, rbuf);     \
  else k_cell_quad<P, JT, DJ, DR, SP><<<gc, CT_, 0, s>>>(A, u, ebuf, rbuf)
  if (doJ && doR) { MRG_GEN_CELL(true, true, SPLIT); }
  else if (doJ) { MRG_GEN_CELL(true, false, SPLIT); }
  else { MRG_GEN_CELL(false, true, false); }
#undef MRG_GEN_CELL
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  const int smem = doJ ? (RT * ipow(2 * P + 1, DIM) + 16 / (int)sizeof(JT)) * (int)sizeof(JT) : 0;
  static_assert((RT * ipow(2 * P + 1, DIM) + 2) * (int)sizeof(JT) <= 48 * 1024, "staged rows fit the default shared memory");
#define MRG_GEN_ROW(DJ, DR, OV) \
  k_gather<DIM, P, JT, DJ, DR, OV><<<gr, RT, smem, s>>>(p->g, q.row0, q.row1, ebuf, rbuf, Q.d_bnode, r, J)
  if (doJ && doR) { if (ovw) MRG_GEN_ROW(true, true, true); else MRG_GEN_ROW(true, true, false); }
  else if (doJ) { if (ovw) MRG_GEN_ROW(true, false, true); else MRG_GEN_ROW(true, false, false); }
  else { if (ovw) MRG_GEN_ROW(false, true, true); else MRG_GEN_ROW(false, true, false); }
#undef MRG_GEN_ROW
  return cudaGetLastError();
}

}  // namespace

bool mrg_general_eligible(const mrg_problem* p, int points_per_axis) {
  if (p->path != MRG_PATH_CELL || points_per_axis != p->g.p + 1) return false;
  return p->g.dim == 2 || p->g.p == 1;
}

int mrg_general_setup(mrg_problem* p, cudaStream_t s) {
  // a metric of more than a quarter of the device's memory (hexahedra: 384 bytes a cell) is left to the per-cell kernels,
  // which form it anew: the caller's matrix is to fit as it would without it
  const size_t bytes = (size_t)p->ncell * (p->g.dim == 3 ? 6 : 3) * p->npe * sizeof(double);
  if (bytes > (size_t)1 << 30) {
    size_t avail = 0, total = 0;
    MRG_CUDA(cudaMemGetInfo(&avail, &total));
    if (bytes > total / 4) return MRG_OK;
  }
  General* Q = new General();
  p->general = Q;
  GenTab& t = Q->A.t;
  MetricArgs M{};
  for (int q = 0; q <= p->g.p; ++q) {
    mrg_lagrange_1d(p->g.p, p->gx1[q], t.l[q], t.d[q]);
    t.w[q] = p->gw1[q];
    M.gx[q] = p->gx1[q];
  }
  const double l0 = t.l[0][0], l1 = t.l[0][1];
  HexTab& x = Q->A.hex;
  x.near = l0 / l1;
  x.far = l1 / l0;
  x.scale = 2.0 * (l0 * l1) * (l0 * l1);
  M.g = p->g;
  M.t = t;
  M.vcoord = p->d_vcoord;
  for (int k = 0; k < 3; ++k) {
    M.lo[k] = p->lo[k];
    M.h[k] = p->h[k];
  }
  M.src_sin = p->source_kind == MRG_SRC_SINPROD;
  M.amp = p->source_amp;
  M.freq = p->source_freq;
  M.ncell = p->ncell;
  const int st = p->g.dim == 3 ? setup_t<3, 1>(p, Q, M, s) : (p->g.p == 1 ? setup_t<2, 1>(p, Q, M, s) : setup_t<2, 2>(p, Q, M, s));
  if (st == MRG_ENOMEM) {  // likewise
    cudaGetLastError();
    mrg_general_free(p);
    return MRG_OK;
  }
  if (st) return st;
  Q->A.g = p->g;
  Q->A.metric = Q->d_metric;
  Q->A.bnode = Q->d_bnode;
  Q->A.kap = p->d_kappa;
  Q->A.thermal = p->kind == MRG_THERMAL;
  return mrg_ws_open(p);
}

void mrg_general_free(mrg_problem* p) {
  General* Q = reinterpret_cast<General*>(p->general);
  if (!Q) return;
  if (Q->d_metric) cudaFreeAsync(Q->d_metric, p->stream);
  if (Q->d_bnode) cudaFreeAsync(Q->d_bnode, p->stream);
  delete Q;
  p->general = nullptr;
}

int mrg_launch_general(mrg_problem* p, const double* u, double* r, void* J, uint32_t flags, cudaStream_t s) {
  const General& Q = *reinterpret_cast<General*>(p->general);
  const bool doJ = flags & MRG_ASM_JAC, doR = flags & MRG_ASM_RES, ovw = flags & MRG_ASM_OVERWRITE;
  const bool fp32 = flags & MRG_ASM_J_FP32;
  const size_t ent = (size_t)CB * p->npe * p->npe, eblock = doJ ? ent * (fp32 ? sizeof(float) : sizeof(double)) : 0;
  const size_t rblock = doR ? (size_t)CB * p->npe * sizeof(double) : 0;
  return mrg_in_pieces(p, eblock + rblock, s, [&](const MrgPiece& q) {
    double* rb = mrg_piece_array<double>(q.ws + q.blocks * eblock, q, (size_t)CB * p->npe);
    auto go = [&](auto* Jt) {
      using JT = std::remove_pointer_t<decltype(Jt)>;
      JT* eb = mrg_piece_array<JT>(q.ws, q, ent);
      if (p->g.dim == 3) return launch_t<3, 1, JT, false>(p, Q, q, u, r, Jt, eb, rb, doJ, doR, ovw, s);
      const bool split = p->ncell < FILL * mrg_device_sms();
      if (p->g.p == 1)
        return split ? launch_t<2, 1, JT, true>(p, Q, q, u, r, Jt, eb, rb, doJ, doR, ovw, s)
                     : launch_t<2, 1, JT, false>(p, Q, q, u, r, Jt, eb, rb, doJ, doR, ovw, s);
      return split ? launch_t<2, 2, JT, true>(p, Q, q, u, r, Jt, eb, rb, doJ, doR, ovw, s)
                   : launch_t<2, 2, JT, false>(p, Q, q, u, r, Jt, eb, rb, doJ, doR, ovw, s);
    };
    return fp32 ? go(reinterpret_cast<float*>(J)) : go(reinterpret_cast<double*>(J));
  });
}
