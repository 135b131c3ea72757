// Thermal Q2 quadrilaterals and hexahedra on identical affine cells (reference: src/physics/thermal.cpp:71-165,
// src/managers/assembly/assemblyManager_jacres.hpp:121-630, assemblyManager_scatter.hpp:164-278; the
// identical-element reuse is assemblyManager_database.hpp:12-80).
//
// kappa is constant on a cell, so every cell matrix is kappa_c K_ref.  K_ref is a sum of products of 1-D
// stiffness and mass matrices, which are mirror symmetric, so the entry of a node pair depends along each axis
// on the kind of the row's node (vertex or mid-side) and the distance of the two nodes alone:
//     J(i, i+off) = K[kind(i)][|off|] S(off),   S(off) = sum of kappa over the cells that hold both nodes.
// One thread owns one CSR row: at most 19 additions form its S(off) and one multiplication each entry, where
// the contraction over the Gauss points takes 27 * 81 operations per row and cell.  The residual is
// r_i = b_i - sum over the distance classes of K[class] * (sum of S(off) u(i+off) over the class).
//
// FP32 Jacobians: FP32 sums and products in 3-D; in 2-D, where a row has 16 entries on average, the FP64 products
// rounded once.
//
// What bounds it: the FP64 pipe (16 SM cycles a warp instruction), with about 64 multiplications and 87 FMAs a
// row in 3-D; so warps are filled with rows of one kind (mrg_q2_rows.cuh), which keeps all 32 lanes on the same
// unrolled code whatever the mesh size.  Measured, FP64 Jacobian and residual:
// 33 x 30 x 27 cells 6081 -> 78 us (FP64 floor 66), 300 x 211 cells with two flux sides 1146 -> 33 us.
#include <cmath>
#include <type_traits>
#include <vector>

#include "mrg_fixmul.cuh"
#include "mrg_q2_rows.cuh"

namespace {

using mrgq2::cells;
using mrgq2::half;
using mrgq2::PLANE;

constexpr int BT = 128;  // threads per CTA: 4 warps of 32 rows of one kind

struct BoxArgs {
  Grid g;
  mrgq2::Kinds kinds;
  double K[125];  // class coefficients of the 8 node kinds, kind by kind, z slowest
  float K32[125];
  int koff[8];    // first coefficient of a kind
  const double* B[3];  // per-axis load factors
  double amp;
};

__host__ __device__ constexpr int classes(int P) { return P ? 2 : 3; }  // distances along an axis
__host__ __device__ constexpr int sums(int P) { return P ? 1 : 3; }     // distinct sets of cells: left, both, right
__host__ __device__ constexpr int cls_of(int P, int e) { return e < half(P) ? half(P) - e : e - half(P); }
__host__ __device__ constexpr int sum_of(int P, int e) { return P ? 0 : (e < 2 ? 0 : (e == 2 ? 1 : 2)); }

// S over one axis: (left, left + right, right) of the cells' values, or the one cell's value
template <int P, typename T>
__device__ __forceinline__ T axis_sum(const T* v, int stride, int s) {
  if constexpr (P) return v[0];
  else return s == 0 ? v[0] : (s == 2 ? v[stride] : v[0] + v[stride]);
}

template <int PX, int PY, int PZ, typename T>
__device__ __forceinline__ void kappa_sums(const T (&k)[cells(PZ)][cells(PY)][cells(PX)],
                                           T (&S)[sums(PZ)][sums(PY)][sums(PX)]) {
  T a[cells(PZ)][cells(PY)][sums(PX)], b[cells(PZ)][sums(PY)][sums(PX)];
#pragma unroll
  for (int z = 0; z < cells(PZ); ++z)
#pragma unroll
    for (int y = 0; y < cells(PY); ++y)
#pragma unroll
      for (int x = 0; x < sums(PX); ++x) a[z][y][x] = axis_sum<PX>(&k[z][y][0], 1, x);
#pragma unroll
  for (int z = 0; z < cells(PZ); ++z)
#pragma unroll
    for (int y = 0; y < sums(PY); ++y)
#pragma unroll
      for (int x = 0; x < sums(PX); ++x) b[z][y][x] = axis_sum<PY>(&a[z][0][x], sums(PX), y);
#pragma unroll
  for (int z = 0; z < sums(PZ); ++z)
#pragma unroll
    for (int y = 0; y < sums(PY); ++y)
#pragma unroll
      for (int x = 0; x < sums(PX); ++x) S[z][y][x] = axis_sum<PZ>(&b[0][y][x], sums(PY) * sums(PX), z);
}

// The rows of one warp: kind (PX, PY, PZ), row number `at` of the kind.  2-D problems run as one z plane (PZ = 1,
// D3 = false).
template <bool D3, int PX, int PY, int PZ, typename JT, bool DOJ, bool DOR, bool OVW>
__device__ __forceinline__ void box_rows(const BoxArgs& A, int kind, int64_t at, const double* __restrict__ u,
                                         const double* __restrict__ kap, const float* __restrict__ kap32,
                                         double* __restrict__ r, JT* __restrict__ J, JT* stage) {
  constexpr bool F32 = sizeof(JT) == 4 && D3;  // FP32 products
  constexpr bool K64 = !F32 || DOR;            // FP64 sums of kappa
  using R = mrgq2::Row<D3, PX, PY, PZ>;
  const Grid& g = A.g;
  const R row(g, A.kinds, kind, at);
  const int NX = g.nn[0], NY = g.nn[1];
  // kappa of the row's cells, 0 outside the mesh
  double k[cells(PZ)][cells(PY)][cells(PX)];
  float k32[cells(PZ)][cells(PY)][cells(PX)];
#pragma unroll
  for (int z = 0; z < cells(PZ); ++z)
#pragma unroll
    for (int y = 0; y < cells(PY); ++y)
#pragma unroll
      for (int x = 0; x < cells(PX); ++x) {
        int64_t c;
        const bool ok = row.cell(g, x, y, z, c);
        if (K64) k[z][y][x] = ok ? __ldg(kap + c) : 0.0;
        if (F32 && DOJ) k32[z][y][x] = ok ? __ldg(kap32 + c) : 0.0f;
      }
  double S[sums(PZ)][sums(PY)][sums(PX)];
  float S32[sums(PZ)][sums(PY)][sums(PX)];
  if constexpr (K64) kappa_sums<PX, PY, PZ, double>(k, S);
  if constexpr (F32 && DOJ) kappa_sums<PX, PY, PZ, float>(k32, S32);
  const double* K = A.K + A.koff[kind];
  const float* K32 = A.K32 + A.koff[kind];
  double acc = 0.0;
  if (DOR && row.on) {
    acc = A.amp * __ldg(A.B[0] + row.ix) * __ldg(A.B[1] + row.iy);
    if (D3) acc *= __ldg(A.B[2] + row.iz);
  }
  const double* un = u + row.n;
#pragma unroll
  for (int ez = 0; ez < R::LZ; ++ez) {
    const int oz = D3 ? ez - half(PZ) : 0;
    const int sz = D3 ? sum_of(PZ, ez) : 0, kz = D3 ? cls_of(PZ, ez) : 0;
#pragma unroll
    for (int ky = 0; ky < classes(PY); ++ky)
#pragma unroll
      for (int kx = 0; kx < classes(PX); ++kx) {
        double t = 0.0;
        const int kc = (kz * classes(PY) + ky) * classes(PX) + kx;
#pragma unroll
        for (int ey = 0; ey < R::LY; ++ey) {
          if (cls_of(PY, ey) != ky) continue;
#pragma unroll
          for (int ex = 0; ex < R::LX; ++ex) {
            if (cls_of(PX, ex) != kx) continue;
            const int oy = ey - half(PY), ox = ex - half(PX);
            if (DOJ) {
              JT val;
              if constexpr (F32) val = K32[kc] * S32[sz][sum_of(PY, ey)][sum_of(PX, ex)];
              else if constexpr (sizeof(JT) == 4) val = mrgfix::f64_to_f32_rn(K[kc] * S[sz][sum_of(PY, ey)][sum_of(PX, ex)]);
              else val = K[kc] * S[sz][sum_of(PY, ey)][sum_of(PX, ex)];
              if (row.fixed) val = (OVW && ox == 0 && oy == 0 && oz == 0) ? JT(1) : JT(0);
              row.put(stage, ez, ey, ex, val);
            }
            if (DOR && row.on && row.has_z(oz) && row.has_y(oy) && row.has_x(ox))
              t = fma(S[sz][sum_of(PY, ey)][sum_of(PX, ex)], __ldg(un + ox + (int64_t)NX * (oy + (int64_t)NY * oz)), t);
          }
        }
        if (DOR) acc = fma(-K[kc], t, acc);
      }
    if (DOJ) row.template store_plane<OVW, true>(J, stage, ez);
  }
  if (DOJ && !OVW) row.fix_diagonal(J);
  if (DOR && row.on) {
    if (row.fixed) {
      if (OVW) r[row.n] = 0.0;
    } else {
      if (OVW) r[row.n] = acc; else r[row.n] += acc;
    }
  }
}

template <bool D3, typename JT, bool DOJ, bool DOR, bool OVW>
__global__ void __launch_bounds__(BT) k_box_q2(const __grid_constant__ BoxArgs A, const double* __restrict__ u,
                                               const double* __restrict__ kap, const float* __restrict__ kap32,
                                               double* __restrict__ r, JT* __restrict__ J) {
  __shared__ JT stage_all[DOJ ? (BT / 32) * 32 * PLANE : 1];
  JT* stage = stage_all + (DOJ ? (threadIdx.x >> 5) * 32 * PLANE : 0);
  const int kind = mrgq2::kind_of(A.kinds, blockIdx.x);
  const int64_t at = ((int64_t)blockIdx.x - A.kinds.block0[kind]) * BT + threadIdx.x;
  mrgq2::with_kind<D3>(kind, [&](auto px, auto py, auto pz) {
    box_rows<D3, decltype(px)::value, decltype(py)::value, decltype(pz)::value, JT, DOJ, DOR, OVW>(A, kind, at, u, kap,
                                                                                                  kap32, r, J, stage);
  });
}

struct BoxQ2 {
  BoxArgs A;
  double* d_B = nullptr;
};

template <bool D3, typename JT>
cudaError_t launch(const mrg_problem* p, const BoxQ2& Q, const double* u, double* r, JT* J, bool doJ, bool doR, bool ovw,
                   cudaStream_t s) {
  const unsigned grid = (unsigned)Q.A.kinds.block0[8];
#define MRG_BOX_LAUNCH(DJ, DR, OV) \
  k_box_q2<D3, JT, DJ, DR, OV><<<grid, BT, 0, s>>>(Q.A, u, p->d_kappa, p->d_kappa32, r, J)
  if (doJ && doR) { if (ovw) MRG_BOX_LAUNCH(true, true, true); else MRG_BOX_LAUNCH(true, true, false); }
  else if (doJ) { if (ovw) MRG_BOX_LAUNCH(true, false, true); else MRG_BOX_LAUNCH(true, false, false); }
  else { if (ovw) MRG_BOX_LAUNCH(false, true, true); else MRG_BOX_LAUNCH(false, true, false); }
#undef MRG_BOX_LAUNCH
  return cudaGetLastError();
}

}  // namespace

bool mrg_box_q2_eligible(int order, int kind, int points_per_axis, bool affine) {
  return affine && order == 2 && kind == MRG_THERMAL && points_per_axis == 3;
}

int mrg_box_q2_setup(mrg_problem* p, cudaStream_t s) {
  BoxQ2* Q = new BoxQ2();
  p->box_q2 = Q;
  BoxArgs& A = Q->A;
  A.g = p->g;
  A.amp = p->source_amp;
  const int d = p->g.dim;
  // 1-D mass and stiffness of one cell by the problem's rule; the rows of the left vertex and the mid-side node
  // (the right vertex mirrors the left)
  double M[3][2][3] = {}, D[3][2][3] = {}, l[3][3], dl[3][3];
  for (int q = 0; q < 3; ++q) mrg_lagrange_1d(2, p->gx1[q], l[q], dl[q]);
  for (int k = 0; k < d; ++k)
    for (int a = 0; a < 2; ++a)
      for (int b = 0; b < 3; ++b)
        for (int q = 0; q < 3; ++q) {
          M[k][a][b] += p->gw1[q] * l[q][a] * l[q][b] * 0.5 * p->h[k];
          D[k][a][b] += p->gw1[q] * dl[q][a] * dl[q][b] * 2.0 / p->h[k];
        }
  // distance c from a vertex: its own row [0][c]; from a mid-side node: [1][1] and [1][0]
  auto at = [](const double (&m)[2][3], int mid, int c) { return mid ? m[1][1 - c] : m[0][c]; };
  int off = 0;
  for (int t = 0; t < (d == 3 ? 8 : 4); ++t) {
    const int P[3] = {t & 1, (t >> 1) & 1, d == 3 ? (t >> 2) & 1 : 1};
    A.koff[t] = off;
    for (int c2 = 0; c2 < (d == 3 ? classes(P[2]) : 1); ++c2)
      for (int c1 = 0; c1 < classes(P[1]); ++c1)
        for (int c0 = 0; c0 < classes(P[0]); ++c0) {
          const int c[3] = {c0, c1, c2};
          double v = 0.0;
          for (int a = 0; a < d; ++a) {
            double f = 1.0;
            for (int k = 0; k < d; ++k) f *= (k == a) ? at(D[k], P[k], c[k]) : at(M[k], P[k], c[k]);
            v += f;
          }
          A.K[off] = v;
          A.K32[off++] = (float)v;
        }
  }
  A.kinds = mrgq2::make_kinds(p->g, BT);
  // load factors: b_i = amp * prod_k B_k[i_k], B_k[i] the 1-D integral of f_k phi_i over the node's cells with
  // f_k = 1 or sin(freq x)
  std::vector<double> B;
  for (int k = 0; k < d; ++k)
    for (int i = 0; i < p->g.nn[k]; ++i) {
      int cf, nc;
      axis_cells(i, p->g.nn[k], 2, cf, nc);
      double v = 0.0;
      for (int c = cf; c < cf + nc; ++c)
        for (int q = 0; q < 3; ++q) {
          const double x = p->lo[k] + p->h[k] * (c + 0.5 * (1.0 + p->gx1[q]));
          const double f = p->source_kind == MRG_SRC_SINPROD ? std::sin(p->source_freq * x) : 1.0;
          v += f * l[q][i - 2 * c] * p->gw1[q] * 0.5 * p->h[k];
        }
      B.push_back(v);
    }
  MRG_CUDA(cudaMallocAsync(&Q->d_B, B.size() * sizeof(double), s));
  MRG_CUDA(cudaMemcpyAsync(Q->d_B, B.data(), B.size() * sizeof(double), cudaMemcpyHostToDevice, s));
  MRG_CUDA(cudaStreamSynchronize(s));  // B is a host temporary
  A.B[0] = Q->d_B;
  A.B[1] = Q->d_B + p->g.nn[0];
  A.B[2] = d == 3 ? Q->d_B + p->g.nn[0] + p->g.nn[1] : nullptr;
  return MRG_OK;
}

void mrg_box_q2_free(mrg_problem* p) {
  BoxQ2* Q = reinterpret_cast<BoxQ2*>(p->box_q2);
  if (!Q) return;
  cudaFreeAsync(Q->d_B, p->stream);
  delete Q;
  p->box_q2 = nullptr;
}

int mrg_launch_box_q2(mrg_problem* p, const double* u, double* r, void* J, uint32_t flags, cudaStream_t s) {
  BoxQ2& Q = *reinterpret_cast<BoxQ2*>(p->box_q2);
  const bool doJ = flags & MRG_ASM_JAC, doR = flags & MRG_ASM_RES, ovw = flags & MRG_ASM_OVERWRITE;
  const bool fp32 = flags & MRG_ASM_J_FP32;
  cudaError_t e;
  if (p->g.dim == 3)
    e = fp32 ? launch<true, float>(p, Q, u, r, (float*)J, doJ, doR, ovw, s)
             : launch<true, double>(p, Q, u, r, (double*)J, doJ, doR, ovw, s);
  else
    e = fp32 ? launch<false, float>(p, Q, u, r, (float*)J, doJ, doR, ovw, s)
             : launch<false, double>(p, Q, u, r, (double*)J, doJ, doR, ovw, s);
  return e == cudaSuccess ? MRG_OK : mrg_cuda_check(e, "box Q2 assembly launch");
}
