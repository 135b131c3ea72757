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
// What bounds it: the FP64 pipe (16 SM cycles a warp instruction), with about 64 multiplications and 87 FMAs a
// row in 3-D; so warps are filled with rows of one kind (8 kinds in 3-D, 4 in 2-D, each a grid of its own,
// flattened), which keeps all 32 lanes on the same unrolled code whatever the mesh size.  Rows of a kind are
// not neighbours in CSR: each warp stages one z plane of its 32 rows (25, 15 or 9 values each) in shared memory
// and writes it with consecutive lanes on consecutive addresses.  Measured, FP64 Jacobian and residual:
// 33 x 30 x 27 cells 6081 -> 78 us (FP64 floor 66), 300 x 211 cells with two flux sides 1146 -> 39 us.
#include <cmath>
#include <vector>

#include "mrg_device.cuh"
#include "mrg_internal.h"

namespace {

constexpr int BT = 128;   // threads per CTA: 4 warps of 32 rows of one kind
constexpr int PLANE = 25;  // most entries of a row in one z plane

struct BoxArgs {
  Grid g;
  double K[125];    // class coefficients of the 8 node kinds, kind by kind, z slowest
  float K32[125];
  int koff[8];      // first coefficient of a kind
  int m[8][3];      // nodes of a kind per axis
  int64_t block0[9];  // first CTA of a kind
  const double* B[3];  // per-axis load factors
  double amp;
};

// Along one axis a row of kind PX (0: vertex, 1: mid-side) has up to len(PX) couplings from up to 2 - PX cells
__host__ __device__ constexpr int len(int P) { return P ? 3 : 5; }
__host__ __device__ constexpr int half(int P) { return P ? 1 : 2; }
__host__ __device__ constexpr int classes(int P) { return P ? 2 : 3; }
__host__ __device__ constexpr int sums(int P) { return P ? 1 : 3; }  // distinct sets of cells: left, both, right
__host__ __device__ constexpr int cells(int P) { return P ? 1 : 2; }
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

// The rows of one warp: kind (PX, PY, PZ), row number `at` of the kind (x fastest).  2-D problems run as one
// z plane (PZ = 1, D3 = false).
template <bool D3, int PX, int PY, int PZ, typename JT, bool DOJ, bool DOR, bool OVW>
__device__ __forceinline__ void box_rows(const BoxArgs& A, int kind, int64_t at, const double* __restrict__ u,
                                         const double* __restrict__ kap, const float* __restrict__ kap32,
                                         double* __restrict__ r, JT* __restrict__ J, JT* stage) {
  constexpr bool MIXED = sizeof(JT) == 4;
  constexpr int LX = len(PX), LY = len(PY), LZ = D3 ? len(PZ) : 1, N = LX * LY;
  const Grid& g = A.g;
  const int lane = threadIdx.x & 31;
  const int mx = A.m[kind][0], my = A.m[kind][1];
  const bool on = at < (int64_t)mx * my * A.m[kind][2];
  int ix = PX, iy = PY, iz = D3 ? PZ : 0;
  if (on) {
    const unsigned a = (unsigned)at, t = a / (unsigned)mx;
    ix += 2 * (int)(a - t * (unsigned)mx);
    iy += 2 * (int)(t % (unsigned)my);
    if (D3) iz += 2 * (int)(t / (unsigned)my);
  }
  const int NX = g.nn[0], NY = g.nn[1], NZ = g.nn[2];
  // couplings that exist: a vertex at an end of its axis has one cell only
  const bool xl = PX || ix > 0, xr = PX || ix < NX - 1, yl = PY || iy > 0, yr = PY || iy < NY - 1;
  const bool zl = !D3 || PZ || iz > 0, zr = !D3 || PZ || iz < NZ - 1;
  const int cx = (xl && xr) ? LX : 3, cy = (yl && yr) ? LY : 3, cz = D3 ? ((zl && zr) ? LZ : 3) : 1;
  const bool fixed = on && node_fixed(g, ix, iy, iz);
  const int64_t n = ix + (int64_t)NX * (iy + (int64_t)NY * iz);
  int64_t rp = 0;
  if (DOJ && on) rp = g.P[2][iz] * g.T[1] * g.T[0] + (int64_t)cz * (g.P[1][iy] * g.T[0] + (int64_t)cy * g.P[0][ix]);
  // kappa of the row's cells, 0 outside the mesh
  double k[cells(PZ)][cells(PY)][cells(PX)];
  float k32[cells(PZ)][cells(PY)][cells(PX)];
#pragma unroll
  for (int z = 0; z < cells(PZ); ++z)
#pragma unroll
    for (int y = 0; y < cells(PY); ++y)
#pragma unroll
      for (int x = 0; x < cells(PX); ++x) {
        const int ccx = PX ? ix / 2 : ix / 2 - 1 + x, ccy = PY ? iy / 2 : iy / 2 - 1 + y;
        const int ccz = !D3 ? 0 : (PZ ? iz / 2 : iz / 2 - 1 + z);
        const bool ok = on && ccx >= 0 && ccx < g.nc[0] && ccy >= 0 && ccy < g.nc[1] && ccz >= 0 && ccz < g.nc[2];
        const int64_t c = ccx + (int64_t)g.nc[0] * (ccy + (int64_t)g.nc[1] * ccz);
        if (!MIXED || DOR) k[z][y][x] = ok ? __ldg(kap + c) : 0.0;
        if (MIXED && DOJ) k32[z][y][x] = ok ? __ldg(kap32 + c) : 0.0f;
      }
  double S[sums(PZ)][sums(PY)][sums(PX)];
  float S32[sums(PZ)][sums(PY)][sums(PX)];
  if constexpr (!MIXED || DOR) kappa_sums<PX, PY, PZ, double>(k, S);
  if constexpr (MIXED && DOJ) kappa_sums<PX, PY, PZ, float>(k32, S32);
  const double* K = A.K + A.koff[kind];
  const float* K32 = A.K32 + A.koff[kind];
  double acc = 0.0;
  if (DOR) {
    acc = on ? A.amp * __ldg(A.B[0] + ix) * __ldg(A.B[1] + iy) : 0.0;
    if (D3 && on) acc *= __ldg(A.B[2] + iz);
  }
  const bool whole = cx == LX && cy == LY && cz == LZ && on;
  const bool all_whole = __all_sync(0xffffffffu, whole);
  const double* un = u + n;
#pragma unroll
  for (int ez = 0; ez < LZ; ++ez) {
    const int oz = D3 ? ez - half(PZ) : 0;
    const int sz = D3 ? sum_of(PZ, ez) : 0, kz = D3 ? cls_of(PZ, ez) : 0;
    const bool vz = !D3 || PZ || oz == 0 || (oz < 0 ? zl : zr);
    const int xmin = xl ? 0 : half(PX), ymin = yl ? 0 : half(PY);
#pragma unroll
    for (int ky = 0; ky < classes(PY); ++ky)
#pragma unroll
      for (int kx = 0; kx < classes(PX); ++kx) {
        double t = 0.0;
        const int kc = (kz * classes(PY) + ky) * classes(PX) + kx;
#pragma unroll
        for (int ey = 0; ey < LY; ++ey) {
          if (cls_of(PY, ey) != ky) continue;
#pragma unroll
          for (int ex = 0; ex < LX; ++ex) {
            if (cls_of(PX, ex) != kx) continue;
            const int oy = ey - half(PY), ox = ex - half(PX);
            const bool v = vz && (PY || oy == 0 || (oy < 0 ? yl : yr)) && (PX || ox == 0 || (ox < 0 ? xl : xr));
            if (DOJ) {
              JT val;
              if constexpr (MIXED) val = K32[kc] * S32[sz][sum_of(PY, ey)][sum_of(PX, ex)];
              else val = K[kc] * S[sz][sum_of(PY, ey)][sum_of(PX, ex)];
              if (fixed) val = (OVW && ox == 0 && oy == 0 && oz == 0) ? JT(1) : JT(0);
              if (all_whole) stage[lane * N + ey * LX + ex] = val;
              else if (v) stage[lane * PLANE + (ey - ymin) * cx + (ex - xmin)] = val;
            }
            if (DOR && v && on) t = fma(S[sz][sum_of(PY, ey)][sum_of(PX, ex)], __ldg(un + ox + (int64_t)NX * (oy + (int64_t)NY * oz)), t);
          }
        }
        if (DOR) acc = fma(-K[kc], t, acc);
      }
    if (DOJ) {
      __syncwarp();
      if (all_whole) {
        // 32 rows of N values, value by value: consecutive lanes on consecutive addresses
        const int64_t base = rp + (int64_t)ez * N;
#pragma unroll 5
        for (int i = 0; i < N; ++i) {
          const int e = i * 32 + lane, row = e / N;
          const int64_t d = __shfl_sync(0xffffffffu, base, row) + (e - row * N);
          if (OVW) __stcs(J + d, stage[e]); else J[d] += stage[e];
        }
      } else {
        const int64_t base = rp + (int64_t)(ez - (zl ? 0 : half(PZ))) * cx * cy;
        const int count = (on && vz) ? cx * cy : 0;
        for (int row = 0; row < 32; ++row) {
          const int64_t d = __shfl_sync(0xffffffffu, base, row);
          const int c = __shfl_sync(0xffffffffu, count, row);
          if (lane < c) {
            if (OVW) J[d + lane] = stage[row * PLANE + lane]; else J[d + lane] += stage[row * PLANE + lane];
          }
        }
      }
      __syncwarp();
    }
  }
  if (DOJ && !OVW && fixed) {
    // the row's values were left as they were; its diagonal is 1 (written after this warp's additions)
    const int dx = xl ? half(PX) : 0, dy = yl ? half(PY) : 0, dz = !D3 ? 0 : (zl ? half(PZ) : 0);
    J[rp + ((int64_t)dz * cy + dy) * cx + dx] = JT(1);
  }
  if (DOR && on) {
    if (fixed) {
      if (OVW) r[n] = 0.0;
    } else {
      if (OVW) r[n] = acc; else r[n] += acc;
    }
  }
}

template <bool D3, typename JT, bool DOJ, bool DOR, bool OVW>
__global__ void __launch_bounds__(BT) k_box_q2(const __grid_constant__ BoxArgs A, const double* __restrict__ u,
                                               const double* __restrict__ kap, const float* __restrict__ kap32,
                                               double* __restrict__ r, JT* __restrict__ J) {
  __shared__ JT stage_all[DOJ ? (BT / 32) * 32 * PLANE : 1];
  JT* stage = stage_all + (DOJ ? (threadIdx.x >> 5) * 32 * PLANE : 0);
  constexpr int KINDS = D3 ? 8 : 4;
  int kind = 0;
#pragma unroll
  for (int t = 1; t < KINDS; ++t)
    if ((int64_t)blockIdx.x >= A.block0[t]) kind = t;
  const int64_t at = ((int64_t)blockIdx.x - A.block0[kind]) * BT + threadIdx.x;
#define MRG_BOX_KIND(T)                                                                                           \
  case T:                                                                                                         \
    box_rows<D3, (T) & 1, ((T) >> 1) & 1, D3 ? ((T) >> 2) & 1 : 1, JT, DOJ, DOR, OVW>(A, T, at, u, kap, kap32, r, \
                                                                                     J, stage);                  \
    break;
  switch (kind) {
    MRG_BOX_KIND(0)
    MRG_BOX_KIND(1)
    MRG_BOX_KIND(2)
    MRG_BOX_KIND(3)
    default:
      if constexpr (D3) {
        switch (kind) {
          MRG_BOX_KIND(4)
          MRG_BOX_KIND(5)
          MRG_BOX_KIND(6)
          MRG_BOX_KIND(7)
        }
      }
  }
#undef MRG_BOX_KIND
}

struct BoxQ2 {
  BoxArgs A;
  int64_t blocks = 0;
  double* d_B = nullptr;
};

template <bool D3, typename JT>
cudaError_t launch(const mrg_problem* p, const BoxQ2& Q, const double* u, double* r, JT* J, bool doJ, bool doR, bool ovw,
                   cudaStream_t s) {
  const unsigned grid = (unsigned)Q.blocks;
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
  int64_t blocks = 0;
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
    int64_t rows = 1;
    for (int k = 0; k < 3; ++k) {
      A.m[t][k] = k < d ? (P[k] ? p->g.nc[k] : p->g.nc[k] + 1) : 1;
      rows *= A.m[t][k];
    }
    A.block0[t] = blocks;
    blocks += (rows + BT - 1) / BT;
  }
  for (int t = (d == 3 ? 8 : 4); t <= 8; ++t) A.block0[t] = blocks;
  Q->blocks = blocks;
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
