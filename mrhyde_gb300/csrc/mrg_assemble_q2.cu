// 1 + u^2 diffusion on Q2 hexahedra of identical affine cells (configuration C3: -div((1+u^2) grad u) = f, 27 nodes
// and 3 x 3 x 3 Gauss points a cell).  Reference: src/physics/thermal.cpp:71-165 (residual form),
// src/managers/assembly/assemblyManager_jacres.hpp:121-630 (workset loop), assemblyManager_scatter.hpp:164-278.
//
// k_q2_cell works on 32 cells a CTA: lane = cell, warp = line, so that every table entry is a warp-uniform constant and
// every shared-memory access 32 consecutive values.
//   Fields and residual (FP64).  u and its scaled reference gradient at the Gauss points by sum factorisation, a warp
//   for each of the 9 lines of a direction; the middle Gauss point is the middle node, and the outer two are mirror
//   images, so a line takes 9 operations for values and derivatives (18 by the 3 x 3 tables) and 13 back for a pair of
//   fluxes.  1,060 FP64 operations a cell (1,300, and 1025 us for the call below, with the products of the fluxes formed by
//   themselves and the doublings and constants left in the lines) against 1,650 with one lane per Gauss point, and all
//   32 lanes work instead of 27: the FP64 pipe bounds this part.
//   Element matrix (FP64 or FP32, the Jacobian's type).  Warp w owns the pair (l_x, j_x) = (w % 3, w / 3).  With the
//   coefficients c = W (1 + u^2) and e_a = W 2 u s_a^2 d_a u at the points, sums over q_x, q_y and q_z in turn give
//       J[l][j] = sum_q c sum_a s_a^2 d_a phi_l d_a phi_j + sum_q sum_a e_a d_a phi_l phi_j
//   in about 11,400 multiply-adds a cell, where the dense contraction with the constant operand takes 2 * 27 * 27 * 108
//   (three times that as 3xTF32 products on the tensor cores): in FP32 that is less time than the tensor cores take,
//   and it runs on the FP32 pipe while other CTAs' fields keep the FP64 pipe busy.
//   Results go to a workspace in blocks of 32 cells, entry by entry, so that lanes write consecutive addresses.
// k_q2_row: one thread a CSR row, rows of one kind per warp (mrg_q2_rows.cuh): its 1, 2, 4 or 8 cells' entries, lane by
// lane consecutive, added in a fixed order and written once.
//
// Measured on 64^3 cells, FP32 Jacobian and FP64 residual: 1818 -> 933 us (the tensor-core path with eight coloured
// residual launches before), and the FP32 matrix's error fell from 2.4e-7 to 2.1e-8.  Cells take 600 us of it (FP64 pipe),
// rows 390 (memory); the rows of a slab run beside the next slab's cells.
// MRG_ASM_TENSOR_CORES takes the FP32 element matrices from the tcgen05 kernel instead (mrg_tc_q2.cu), for which
// k_q2_cell writes the coefficients as TF32 operand images.
#include <algorithm>
#include <cmath>
#include <mutex>
#include <vector>

#include "mrg_fixmul.cuh"
#include "mrg_q2_rows.cuh"

namespace {

constexpr int CB = MRG_CELL_BLOCK;  // cells per CTA and per workspace block
constexpr int LINES = 9;     // warps: lines of one direction, pairs (l_x, j_x)
constexpr int ET = LINES * 32;
constexpr int ENT = 729;     // entries of an element matrix
constexpr int QRT = 128;     // threads per CTA of the row kernel
// Slabs of cell layers (64^3 cells, FP32 Jacobian and FP64 residual, with 1,300 operations a cell: one slab 1151 us,
// 4 1074, 8 1050, 12 1059, 16 1086).
// A slab of 16384 cells is 512 CTAs, a little more than the GPU holds at 3 CTAs per SM: below that the launches' ends cost
// more than the overlap gives.
constexpr int MAXSLAB = 8;
constexpr int64_t SLAB_CELLS = 16384;

// k_q2_cell hands over e_a / E_SCALE (half the derivatives, and W u for 2 W u)
constexpr double E_SCALE = 4.0;

// Tables in the arithmetic type.  Gauss points -s, 0, s; node values l(q, a), derivatives d(q, a).
template <typename T>
struct Tab {
  T ea, oa, w;         // l(q, outer) = ea -+ oa, l(outer q, middle) = w = 1 - 2 ea, l(middle q, middle) = 1
  T hc[3], zc[3];      // c / 4 and c s / 2 with c = (2 / h_a)^2: half the scaled derivative
  T s2, s4;            // 2 s and -4 s: twice the transposed derivative
  T W[27];             // w_q |det J|
  T load[27];          // f * sum_q W_q phi_l(q)
  T LL[3][9], DL[3][9];  // [q][l + 3 j]: l_l l_j, E_SCALE d_l l_j
  T DD[3][3][9];       // [axis][q][l + 3 j]: sc d_l d_j
};

struct Q2Args {
  Grid g;
  int64_t ncell;
  int64_t blk0;        // first block of 32 cells of the launch
  Tab<double> t64;
  Tab<float> t32;
};

template <typename T>
__device__ __forceinline__ const Tab<T>& tab(const Q2Args& A) {
  if constexpr (sizeof(T) == 4) return A.t32; else return A.t64;
}

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

// round to the nearest TF32 value (10 explicit mantissa bits, ties away from zero)
__device__ __forceinline__ float tf32_rn(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;\n" : "=r"(r) : "f"(x));
  return __uint_as_float(r);
}

// Line operations, with explicit operations throughout.  Powers of two go where they cost nothing: derivatives are taken at
// half and their transposes at twice their size, exactly.
// values at the three Gauss points of a line: with z = v0 - 2 v1 + v2 the even part is v1 + ea z
template <typename T>
__device__ __forceinline__ T even_odd(const T v[3], T& o) {
  o = addr(v[2], -v[0]);
  return fma(T(-2), v[1], addr(v[0], v[2]));
}
template <typename T>
__device__ __forceinline__ void values(const Tab<T>& t, const T v[3], T q[3]) {
  T o;
  const T z = even_odd(v, o), m = fma(t.ea, z, v[1]);
  q[0] = fma(-t.oa, o, m);
  q[1] = v[1];
  q[2] = fma(t.oa, o, m);
}
// values, and half the derivatives along axis a
template <typename T>
__device__ __forceinline__ void values_derivs(const Tab<T>& t, int a, const T v[3], T q[3], T d[3]) {
  T o;
  const T z = even_odd(v, o), m = fma(t.ea, z, v[1]), h = mulr(t.hc[a], o);
  q[0] = fma(-t.oa, o, m);
  q[1] = v[1];
  q[2] = fma(t.oa, o, m);
  d[0] = fma(-t.zc[a], z, h);
  d[1] = h;
  d[2] = fma(t.zc[a], z, h);
}
// the transposes: node sums of Gauss-point values against node values
template <typename T>
__device__ __forceinline__ void values_t(const Tab<T>& t, T f1, T e, T o, T v[3]) {  // e = f0 + f2, o = f2 - f0
  const T m = mulr(t.ea, e);
  v[0] = fma(-t.oa, o, m);
  v[1] = fma(t.w, e, f1);
  v[2] = fma(t.oa, o, m);
}
template <typename T>
__device__ __forceinline__ void values_t(const Tab<T>& t, const T f[3], T v[3]) {
  values_t<T>(t, f[1], addr(f[0], f[2]), addr(f[2], -f[0]), v);
}
// of the products c g
template <typename T>
__device__ __forceinline__ void values_t(const Tab<T>& t, const T c[3], const T g[3], T v[3]) {
  const T f0 = mulr(c[0], g[0]);
  values_t<T>(t, mulr(c[1], g[1]), fma(c[2], g[2], f0), fma(c[2], g[2], -f0), v);
}
// twice the sums against node derivatives, of the products c g
template <typename T>
__device__ __forceinline__ void derivs_t(const Tab<T>& t, const T c[3], const T g[3], T v[3]) {
  const T f0 = mulr(c[0], g[0]), o = fma(c[2], g[2], -f0), m = fma(c[1], g[1], fma(c[2], g[2], f0));
  v[0] = fma(t.s2, o, -m);
  v[1] = mulr(t.s4, o);
  v[2] = fma(t.s2, o, m);
}
// twice the sums of fd against derivatives plus the sums of fv against values
template <typename T>
__device__ __forceinline__ void derivs_values_t(const Tab<T>& t, const T fd[3], const T fv[3], T v[3]) {
  const T o = addr(fd[2], -fd[0]), m = addr(addr(fd[0], fd[2]), fd[1]);
  const T e = addr(fv[0], fv[2]), ov = addr(fv[2], -fv[0]);
  v[0] = fma(t.s2, o, fma(-t.oa, ov, fma(t.ea, e, -m)));
  v[1] = fma(t.s4, o, fma(t.w, e, fv[1]));
  v[2] = fma(t.s2, o, fma(t.oa, ov, fma(t.ea, e, m)));
}

// What k_q2_cell leaves behind besides the residual entries
enum { OUT_NONE = 0, OUT_MATRIX = 1, OUT_TF32 = 2 };

template <typename JT, typename CT, int OUT>
constexpr int cell_smem() {
  return 2 * 3 * 27 * CB * (int)sizeof(CT) + (OUT == OUT_NONE ? 0 : 108 * CB * (int)sizeof(JT));
}

// JT: type of the element matrix.  CT: type of the fields (double whenever the residual is formed; float for the FP32
// Jacobian alone).  out: element matrices [cell / 32][27 l + j][32], or the operand image
// [cell / 128][hi, lo][k / 4][128][4].  rbuf: residual entries [cell / 32][27][32].
template <typename JT, typename CT, int OUT, bool DOR>
__global__ void __launch_bounds__(ET, sizeof(JT) == 4 ? 3 : 2)  // FP32: 1106 -> 1074 us against 2 CTAs per SM
    k_q2_cell(const __grid_constant__ Q2Args A, const double* __restrict__ u, JT* __restrict__ out,
              double* __restrict__ rbuf) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  CT* const a0 = reinterpret_cast<CT*>(smem_raw) + (threadIdx.x & 31);  // three fields of 27 values a cell
  CT* const b0 = a0 + 3 * 27 * CB;
  JT* const co = reinterpret_cast<JT*>(smem_raw + 2 * 3 * 27 * CB * sizeof(CT)) + (threadIdx.x & 31);  // c, e_x, e_y, e_z
  constexpr int F = 27 * CB;  // stride between fields
  const Tab<CT>& t = tab<CT>(A);
  const Grid& g = A.g;
  const int line = threadIdx.x >> 5, lane = threadIdx.x & 31, i = line % 3, k = line / 3;
  const int64_t blk = A.blk0 + blockIdx.x, slot = blk * CB + lane;
  const int64_t c = slot < A.ncell ? slot : A.ncell - 1;  // the last block's spare lanes repeat a cell
  {
    const unsigned c32 = (unsigned)c, r = c32 / (unsigned)g.nc[0];
    const int cx = (int)(c32 - r * (unsigned)g.nc[0]), cz = (int)(r / (unsigned)g.nc[1]);
    const int cy = (int)(r - (unsigned)cz * (unsigned)g.nc[1]);
    const double* un = u + 2 * cx + (int64_t)g.nn[0] * ((2 * cy + i) + (int64_t)g.nn[1] * (2 * cz + k));
    CT v[3], q[3], d[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) v[a] = (CT)__ldg(un + a);
    values_derivs<CT>(t, 0, v, q, d);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      a0[(3 * line + a) * CB] = q[a];
      a0[F + (3 * line + a) * CB] = d[a];
    }
  }
  __syncthreads();
  {  // y: line (q_x, node z)
    const int at = (i + 9 * k) * CB;
    CT v[3], q[3], d[3];
#pragma unroll
    for (int b = 0; b < 3; ++b) v[b] = a0[at + 3 * b * CB];
    values_derivs<CT>(t, 1, v, q, d);
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      b0[at + 3 * b * CB] = q[b];
      b0[2 * F + at + 3 * b * CB] = d[b];
      v[b] = a0[F + at + 3 * b * CB];
    }
    values<CT>(t, v, q);
#pragma unroll
    for (int b = 0; b < 3; ++b) b0[F + at + 3 * b * CB] = q[b];
  }
  __syncthreads();
  {  // z: line (q_x, q_y); the flux at its three points and back
    const int at = line * CB;
    CT v[3], uq[3], gx[3], gy[3], gz[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) v[q] = b0[at + 9 * q * CB];
    values_derivs<CT>(t, 2, v, uq, gz);
#pragma unroll
    for (int q = 0; q < 3; ++q) v[q] = b0[F + at + 9 * q * CB];
    values<CT>(t, v, gx);
#pragma unroll
    for (int q = 0; q < 3; ++q) v[q] = b0[2 * F + at + 9 * q * CB];
    values<CT>(t, v, gy);
    CT cw[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const CT W = t.W[line + 9 * q], e = mulr(W, uq[q]);
      cw[q] = fma(e, uq[q], W);
      if constexpr (OUT != OUT_NONE) {
        co[(line + 9 * q) * CB] = as<JT>(cw[q]);
        co[(27 + line + 9 * q) * CB] = as<JT>(mulr(e, gx[q]));
        co[(54 + line + 9 * q) * CB] = as<JT>(mulr(e, gy[q]));
        co[(81 + line + 9 * q) * CB] = as<JT>(mulr(e, gz[q]));
      }
    }
    if constexpr (DOR) {
      values_t<CT>(t, cw, gx, v);
#pragma unroll
      for (int q = 0; q < 3; ++q) a0[at + 9 * q * CB] = v[q];
      values_t<CT>(t, cw, gy, v);
#pragma unroll
      for (int q = 0; q < 3; ++q) a0[F + at + 9 * q * CB] = v[q];
      derivs_t<CT>(t, cw, gz, v);
#pragma unroll
      for (int q = 0; q < 3; ++q) a0[2 * F + at + 9 * q * CB] = v[q];
    }
  }
  __syncthreads();
  if constexpr (DOR) {
    // the x and y fluxes come at half their size and are doubled by their transposed derivatives; the z flux is whole
    {  // back along y: line (q_x, node z)
      const int at = (i + 9 * k) * CB;
      CT f[3], w[3], v[3];
#pragma unroll
      for (int b = 0; b < 3; ++b) f[b] = a0[at + 3 * b * CB];
      values_t<CT>(t, f, v);
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        b0[at + 3 * b * CB] = v[b];
        f[b] = a0[F + at + 3 * b * CB];
        w[b] = a0[2 * F + at + 3 * b * CB];
      }
      derivs_values_t<CT>(t, f, w, v);
#pragma unroll
      for (int b = 0; b < 3; ++b) b0[F + at + 3 * b * CB] = v[b];
    }
    __syncthreads();
    {  // back along x: line (node y, node z)
      CT f[3], w[3], v[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        f[a] = b0[(3 * line + a) * CB];
        w[a] = b0[F + (3 * line + a) * CB];
      }
      derivs_values_t<CT>(t, f, w, v);
#pragma unroll
      for (int a = 0; a < 3; ++a) rbuf[(blk * 27 + 3 * line + a) * CB + lane] = addr(v[a], -t.load[3 * line + a]);
    }
  }
  if constexpr (OUT == OUT_TF32) {
    // four consecutive coefficients of a cell, split x = hi + lo (hi = x rounded to TF32, lo = the remainder rounded
    // to TF32), to the operand image
    if (slot < A.ncell) {
#pragma unroll
      for (int n = 0; n < 3; ++n) {
        const int ch = line + 9 * n;  // 27 chunks
        float h[4], l[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float v = co[(4 * ch + e) * CB];
          h[e] = tf32_rn(v);
          l[e] = tf32_rn(v - h[e]);
        }
        float* w = out + (c >> 7) * (2 * 128 * 112) + ch * 512 + (c & 127) * 4;
        *reinterpret_cast<float4*>(w) = make_float4(h[0], h[1], h[2], h[3]);
        *reinterpret_cast<float4*>(w + 128 * 112) = make_float4(l[0], l[1], l[2], l[3]);
      }
    }
  }
  if constexpr (OUT == OUT_MATRIX) {
    const Tab<JT>& tj = tab<JT>(A);
    const int lx = line % 3, jx = line / 3;
    // sums over q_x at (q_y, q_z): what multiplies L L along y and z (P), D D along one of them (Q), D L along y (Y) and
    // along z (Z)
    JT P[9], Q[9], Y[9], Z[9];
    {
      JT ll[3], dl[3], dd[3];
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        ll[q] = tj.LL[q][line];
        dl[q] = tj.DL[q][line];
        dd[q] = tj.DD[0][q][line];
      }
#pragma unroll
      for (int m = 0; m < 9; ++m) {
        P[m] = Q[m] = Y[m] = Z[m] = JT(0);
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          const JT cq = co[(q + 3 * m) * CB];
          P[m] = fma(dl[q], co[(27 + q + 3 * m) * CB], fma(dd[q], cq, P[m]));
          Q[m] = fma(ll[q], cq, Q[m]);
          Y[m] = fma(ll[q], co[(54 + q + 3 * m) * CB], Y[m]);
          Z[m] = fma(ll[q], co[(81 + q + 3 * m) * CB], Z[m]);
        }
      }
    }
    JT* eo = out + (blk * ENT + 27 * lx + jx) * CB + lane;
#pragma unroll 1
    for (int y = 0; y < 9; ++y) {  // (l_y, j_y) = (y % 3, y / 3)
      JT p[3], d[3], z[3];
#pragma unroll
      for (int qz = 0; qz < 3; ++qz) {
        p[qz] = d[qz] = z[qz] = JT(0);
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          const int m = q + 3 * qz;
          p[qz] = fma(tj.LL[q][y], P[m], fma(tj.DD[1][q][y], Q[m], fma(tj.DL[q][y], Y[m], p[qz])));
          d[qz] = fma(tj.LL[q][y], Q[m], d[qz]);
          z[qz] = fma(tj.LL[q][y], Z[m], z[qz]);
        }
      }
      JT* ey = eo + (81 * (y % 3) + 3 * (y / 3)) * CB;  // 27 (l_x + 3 l_y) + j_x + 3 j_y
#pragma unroll
      for (int w = 0; w < 9; ++w) {  // (l_z, j_z) = (w % 3, w / 3)
        JT e = JT(0);
#pragma unroll
        for (int q = 0; q < 3; ++q) e = fma(tj.LL[q][w], p[q], fma(tj.DD[2][q][w], d[q], fma(tj.DL[q][w], z[q], e)));
        ey[(243 * (w % 3) + 9 * (w / 3)) * CB] = e;
      }
    }
  }
}

// One row of kind (PX, PY, PZ)
template <int PX, int PY, int PZ, typename JT, bool DOJ, bool DOR, bool OVW>
__device__ __forceinline__ void q2_row(const Grid& g, const mrgq2::Kinds& K, int kind, int64_t at, const JT* __restrict__ ebuf,
                                       const double* __restrict__ rbuf, double* __restrict__ r, JT* __restrict__ J,
                                       JT* stage) {
  using mrgq2::cells;
  using mrgq2::half;
  using R = mrgq2::Row<true, PX, PY, PZ>;
  const R row(g, K, kind, at);
  // local index along an axis: a mid-side node is 1; a vertex is 2 in the cell on its left, 0 in the one on its right
  auto local = [](int P, int s) { return P ? 1 : (s ? 0 : 2); };
  const JT* e[cells(PZ)][cells(PY)][cells(PX)];
  bool ok[cells(PZ)][cells(PY)][cells(PX)];
  double res = 0.0;
  if (DOR && row.on && !OVW) res = r[row.n];
#pragma unroll
  for (int z = 0; z < cells(PZ); ++z)
#pragma unroll
    for (int y = 0; y < cells(PY); ++y)
#pragma unroll
      for (int x = 0; x < cells(PX); ++x) {
        int64_t c;
        ok[z][y][x] = row.cell(g, x, y, z, c) && !row.fixed;
        const int l = local(PX, x) + 3 * local(PY, y) + 9 * local(PZ, z);
        if (DOJ) e[z][y][x] = ebuf + ((c >> 5) * ENT + 27 * l) * CB + (c & 31);
        if (DOR && ok[z][y][x]) res = addr(res, -__ldg(rbuf + ((c >> 5) * 27 + l) * CB + (c & 31)));
      }
  if (DOR && row.on) r[row.n] = res;  // a Dirichlet row is left alone (overwrite: 0)
  if constexpr (DOJ) {
    // Rows with all their cells: no predicates and no branches, so that a plane's loads are in flight together (the
    // kernel waits on memory: with a branch at every entry it took 623 us on 64^3 cells)
    const bool fast = row.all_whole && !__any_sync(0xffffffffu, row.fixed);
    auto plane = [&](int ez, auto fast_tag) {
      constexpr bool FAST = decltype(fast_tag)::value;
      JT v[R::N];
#pragma unroll
      for (int n = 0; n < R::N; ++n) {
        const int oz = ez - half(PZ), oy = n / R::LX - half(PY), ox = n % R::LX - half(PX);
        v[n] = JT(0);
#pragma unroll
        for (int z = 0; z < cells(PZ); ++z)
#pragma unroll
          for (int y = 0; y < cells(PY); ++y)
#pragma unroll
            for (int x = 0; x < cells(PX); ++x) {
              const int jx = local(PX, x) + ox, jy = local(PY, y) + oy, jz = local(PZ, z) + oz;
              if (jx < 0 || jx > 2 || jy < 0 || jy > 2 || jz < 0 || jz > 2) continue;
              if (FAST || ok[z][y][x]) v[n] += __ldg(e[z][y][x] + (jx + 3 * jy + 9 * jz) * CB);
            }
        if (!FAST && OVW && row.fixed && ox == 0 && oy == 0 && oz == 0) v[n] = JT(1);
      }
#pragma unroll
      for (int n = 0; n < R::N; ++n) {
        if (FAST) stage[(threadIdx.x & 31) * R::N + n] = v[n];
        else row.put(stage, ez, n / R::LX, n % R::LX, v[n]);
      }
    };
#pragma unroll
    for (int ez = 0; ez < R::LZ; ++ez) {
      if (fast) plane(ez, std::true_type{});
      else plane(ez, std::false_type{});
      row.template store_plane<OVW, false>(J, stage, ez);
    }
    if (!OVW) row.fix_diagonal(J);
  }
}

template <typename JT, bool DOJ, bool DOR, bool OVW>
__global__ void __launch_bounds__(QRT) k_q2_row(const Grid g, const __grid_constant__ mrgq2::Kinds K,
                                                const JT* __restrict__ ebuf, const double* __restrict__ rbuf,
                                                double* __restrict__ r, JT* __restrict__ J) {
  __shared__ JT stage_all[DOJ ? QRT * mrgq2::PLANE : 1];
  JT* stage = stage_all + (DOJ ? (threadIdx.x >> 5) * 32 * mrgq2::PLANE : 0);
  const int kind = mrgq2::kind_of(K, blockIdx.x);
  const int64_t at = ((int64_t)blockIdx.x - K.block0[kind]) * QRT + threadIdx.x;
  mrgq2::with_kind<true>(kind, [&](auto px, auto py, auto pz) {
    q2_row<decltype(px)::value, decltype(py)::value, decltype(pz)::value, JT, DOJ, DOR, OVW>(g, K, kind, at, ebuf, rbuf,
                                                                                             r, J, stage);
  });
}

}  // namespace

// ------------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------------
struct Q2Data {
  Q2Args A;
  std::mutex side_use;              // held by the call that launches on the side stream
  cudaStream_t side = nullptr;      // rows of a slab while the next slab's cells are worked on (several slabs only)
  std::vector<cudaEvent_t> ev;      // MAXSLAB: a slab's cells are done; the last: all rows are
  int* d_err = nullptr;          // tensor-core kernel status (bounded waits), sticky until reported
  int* h_err = nullptr;          // pinned mirror, refreshed asynchronously after every tensor-core launch
  cudaEvent_t err_ev = nullptr;  // recorded after the refresh
  bool err_pending = false;
  Q2Tc* tc = nullptr;            // tensor-core element-matrix plan, built on its first use
};

// slabs of a piece of the mesh
static int slabs_of(const mrg_problem* p, int layers) {
  const int64_t cells = (int64_t)p->g.nc[0] * p->g.nc[1] * layers;
  return (int)std::max<int64_t>(1, std::min<int64_t>(std::min(layers, MAXSLAB), cells / SLAB_CELLS));
}

static Q2Data* q2data(mrg_problem* p) { return reinterpret_cast<Q2Data*>(p->q2); }

int mrg_q2_setup(mrg_problem* p) {
  Q2Data* Q = new Q2Data();
  p->q2 = Q;
  Q->A.g = p->g;
  Q->A.ncell = p->ncell;
  Q->A.blk0 = 0;
  Tab<double>& t = Q->A.t64;
  double l[3][3], d[3][3], sc[3], detJ = 1.0;
  for (int q = 0; q < 3; ++q) mrg_lagrange_1d(2, p->gx1[q], l[q], d[q]);
  const double gs = p->gx1[2];
  t.s2 = 2.0 * gs;
  t.s4 = -4.0 * gs;
  t.ea = 0.5 * (l[0][0] + l[0][2]);
  t.oa = 0.5 * (l[0][0] - l[0][2]);
  t.w = l[0][1];
  for (int a = 0; a < 3; ++a) {
    detJ *= 0.5 * p->h[a];
    sc[a] = (2.0 / p->h[a]) * (2.0 / p->h[a]);
    t.hc[a] = 0.25 * sc[a];
    t.zc[a] = 0.5 * gs * sc[a];
  }
  const double* tw = p->qtab_host.data();
  const double* tphi = tw + p->nq;
  for (int q = 0; q < 27; ++q) t.W[q] = tw[q] * detJ;
  for (int n = 0; n < 27; ++n) {
    double s = 0.0;
    for (int q = 0; q < 27; ++q) s += t.W[q] * tphi[n * 27 + q];
    t.load[n] = p->source_amp * s;
  }
  for (int q = 0; q < 3; ++q)
    for (int n = 0; n < 9; ++n) {
      t.LL[q][n] = l[q][n % 3] * l[q][n / 3];
      t.DL[q][n] = E_SCALE * (d[q][n % 3] * l[q][n / 3]);
      for (int a = 0; a < 3; ++a) t.DD[a][q][n] = sc[a] * d[q][n % 3] * d[q][n / 3];
    }
  static_assert(sizeof(Tab<double>) == 2 * sizeof(Tab<float>), "the two tables hold the same values");
  const double* src = reinterpret_cast<const double*>(&t);
  float* dst = reinterpret_cast<float*>(&Q->A.t32);
  for (size_t k = 0; k < sizeof(t) / sizeof(double); ++k) dst[k] = (float)src[k];
  if (slabs_of(p, p->g.nc[2]) > 1) {
    MRG_CUDA(cudaStreamCreateWithFlags(&Q->side, cudaStreamNonBlocking));
    for (int k = 0; k <= MAXSLAB; ++k) {
      cudaEvent_t e = nullptr;
      MRG_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
      Q->ev.push_back(e);
    }
  }
  cudaStream_t s = p->stream;
  MRG_CUDA(cudaMallocAsync(&Q->d_err, sizeof(int), s));
  MRG_CUDA(cudaMemsetAsync(Q->d_err, 0, sizeof(int), s));
  return mrg_ws_open(p);
}

void mrg_q2_free(mrg_problem* p) {
  Q2Data* Q = q2data(p);
  if (!Q) return;
  if (Q->side) cudaStreamDestroy(Q->side);
  for (cudaEvent_t e : Q->ev) cudaEventDestroy(e);
  cudaFreeAsync(Q->d_err, p->stream);
  if (Q->err_ev) cudaEventDestroy(Q->err_ev);
  mrg_pinned_release(Q->h_err);
  mrg_q2tc_free(Q->tc, p->stream);
  delete Q;
  p->q2 = nullptr;
}

template <typename JT, typename CT, int OUT, bool DOR>
static cudaError_t launch_cell(const Q2Data& Q, const double* u, JT* out, double* rbuf, cudaStream_t s, int64_t b0,
                               int64_t b1) {
  constexpr int smem = cell_smem<JT, CT, OUT>();
  auto kern = k_q2_cell<JT, CT, OUT, DOR>;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  Q2Args A = Q.A;
  A.blk0 = b0;
  if (b1 > b0) kern<<<(unsigned)(b1 - b0), ET, smem, s>>>(A, u, out, rbuf);
  return cudaGetLastError();
}

template <typename JT>
static cudaError_t launch_rows(const mrg_problem* p, const mrgq2::Kinds& K, const JT* ebuf, const double* rbuf, double* r, JT* J,
                               bool doJ, bool doR, bool ovw, cudaStream_t s) {
  const unsigned grid = (unsigned)K.block0[8];
#define MRG_Q2_ROW(DJ, DR, OV) k_q2_row<JT, DJ, DR, OV><<<grid, QRT, 0, s>>>(p->g, K, ebuf, rbuf, r, J)
  if (doJ && doR) { if (ovw) MRG_Q2_ROW(true, true, true); else MRG_Q2_ROW(true, true, false); }
  else if (doJ) { if (ovw) MRG_Q2_ROW(true, false, true); else MRG_Q2_ROW(true, false, false); }
  else { if (ovw) MRG_Q2_ROW(false, true, true); else MRG_Q2_ROW(false, true, false); }
#undef MRG_Q2_ROW
  return cudaGetLastError();
}

// Cells, then rows; in slabs of cell layers on a large mesh, the rows of a slab on the side stream while the next slab's
// cells are worked on: the cells are bound by arithmetic and the rows by memory, so the two overlap.  The bits are the
// same either way.  The side stream and its events serve one call at a time: a call that finds them taken by another
// thread's, or that is being captured (its graph would hold on to the stream until the capture ends), goes without.
template <typename JT, typename CT, bool DOR>
static cudaError_t launch_slabs(const mrg_problem* p, Q2Data& Q, const MrgPiece& q, const double* u, JT* eb, double* rb,
                                double* r, JT* J, bool ovw, cudaStream_t s) {
  const int slabs = slabs_of(p, q.b - q.a);
  std::unique_lock<std::mutex> use(Q.side_use, std::defer_lock);
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (slabs > 1) {
    const cudaError_t e = cudaStreamIsCapturing(s, &cap);
    if (e != cudaSuccess) return e;
  }
  if (slabs == 1 || cap != cudaStreamCaptureStatusNone || !use.try_lock()) {
    const cudaError_t e = launch_cell<JT, CT, OUT_MATRIX, DOR>(Q, u, eb, rb, s, q.block0, q.block1);
    const mrgq2::Kinds K = mrgq2::make_kinds(p->g, QRT, q.a, q.b);
    return e != cudaSuccess ? e : launch_rows<JT>(p, K, eb, rb, r, J, true, DOR, ovw, s);
  }
  const int64_t layer = (int64_t)p->g.nc[0] * p->g.nc[1];
  cudaError_t e = cudaSuccess;
  int64_t b0 = q.block0;
  for (int k = 0; k < slabs && e == cudaSuccess; ++k) {
    const int64_t n = q.b - q.a;
    const int z0 = q.a + (int)(n * k / slabs), z1 = q.a + (int)(n * (k + 1) / slabs);
    // blocks of 32 cells up to the slab's last cell (they may reach into the next layer)
    const int64_t b1 = (layer * z1 + CB - 1) / CB;
    e = launch_cell<JT, CT, OUT_MATRIX, DOR>(Q, u, eb, rb, s, b0, b1);
    b0 = b1;
    if (e == cudaSuccess) e = cudaEventRecord(Q.ev[k], s);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(Q.side, Q.ev[k], 0);
    if (e == cudaSuccess)
      e = launch_rows<JT>(p, mrgq2::make_kinds(p->g, QRT, z0, z1), eb, rb, r, J, true, DOR, ovw, Q.side);
  }
  // the caller's stream goes on when the rows are written, whatever was launched
  cudaError_t j = cudaEventRecord(Q.ev[MAXSLAB], Q.side);
  if (j == cudaSuccess) j = cudaStreamWaitEvent(s, Q.ev[MAXSLAB], 0);
  return e != cudaSuccess ? e : j;
}

// FP32 Jacobian with the element matrices from the tensor cores; rbuf is null when no residual is asked for.
static int launch_tensor_cores(mrg_problem* p, const double* u, double* r, float* J, double* rbuf, bool ovw, cudaStream_t s) {
  Q2Data& Q = *q2data(p);
  // A time-out inside a previous tensor-core launch is reported here, without synchronising: the status word is
  // copied to pinned memory behind an event after every launch and read once that event has completed, so the
  // assembly stays free of host synchronisation (graph-capturable once the plan exists).
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  MRG_CUDA(cudaStreamIsCapturing(s, &cap));
  const bool capturing = cap != cudaStreamCaptureStatusNone;
  if (!capturing && Q.err_pending && cudaEventQuery(Q.err_ev) == cudaSuccess) {
    Q.err_pending = false;
    if (*Q.h_err) {
      *Q.h_err = 0;
      MRG_CUDA(cudaMemsetAsync(Q.d_err, 0, sizeof(int), s));
      return mrg_fail(MRG_ETIMEOUT, "tensor-core element kernel: an mbarrier wait timed out in a previous launch");
    }
  }
  // The first call allocates the plan (element matrices, operand images) and uploads the constant operand: make it
  // outside stream capture.
  if (!Q.tc) {
    const int st = mrg_q2tc_create(p, &Q.tc, s);
    if (st) return st;
    Q.h_err = (int*)mrg_pinned_slot();
    if (!Q.h_err) return mrg_fail(MRG_ENOMEM, "pinned error word");
    *Q.h_err = 0;
    MRG_CUDA(cudaEventCreateWithFlags(&Q.err_ev, cudaEventDisableTiming));
  }
  float* w = mrg_q2tc_w_image(Q.tc);
  const int64_t blocks = (p->ncell + CB - 1) / CB;
  if (rbuf) {
    MRG_CUDA((launch_cell<float, double, OUT_TF32, true>(Q, u, w, rbuf, s, 0, blocks)));
    MRG_CUDA(launch_rows<float>(p, mrgq2::make_kinds(p->g, QRT), nullptr, rbuf, r, nullptr, false, true, ovw, s));
  } else {
    MRG_CUDA((launch_cell<float, float, OUT_TF32, false>(Q, u, w, nullptr, s, 0, blocks)));
  }
  const int st = mrg_q2tc_launch(p, Q.tc, J, ovw, Q.d_err, s);
  if (st) return st;
  MRG_CUDA(cudaMemcpyAsync(Q.h_err, Q.d_err, sizeof(int), cudaMemcpyDeviceToHost, s));
  if (!capturing) {
    MRG_CUDA(cudaEventRecord(Q.err_ev, s));
    Q.err_pending = true;
  }
  return MRG_OK;
}

int mrg_launch_q2(mrg_problem* p, const double* u, double* r, void* J, uint32_t flags, cudaStream_t s) {
  Q2Data& Q = *q2data(p);
  const bool doJ = flags & MRG_ASM_JAC, doR = flags & MRG_ASM_RES, ovw = flags & MRG_ASM_OVERWRITE;
  const bool fp32 = (flags & MRG_ASM_J_FP32) && doJ;
  const bool tc = fp32 && (flags & MRG_ASM_TENSOR_CORES) && !(flags & MRG_ASM_CUDA_CORES);
  const size_t rblock = doR ? (size_t)CB * 27 * sizeof(double) : 0;
  if (tc) {  // the plan holds all cells' coefficients and matrices, and so does the call
    MrgWs ws;
    if (doR) {
      const cudaError_t e = mrg_ws_take(p, (size_t)((p->ncell + CB - 1) / CB) * rblock, s, &ws);
      if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        return MRG_NO_WORKSPACE;
      }
      MRG_CUDA(e);
    }
    const int st = launch_tensor_cores(p, u, r, (float*)J, reinterpret_cast<double*>(ws.p), ovw, s);
    if (ws.p) MRG_CUDA(mrg_ws_give(ws, s));
    return st;
  }
  const size_t eblock = doJ ? (size_t)CB * ENT * (fp32 ? sizeof(float) : sizeof(double)) : 0;
  return mrg_in_pieces(p, eblock + rblock, s, [&](const MrgPiece& q) {
    double* rb = doR ? mrg_piece_array<double>(q.ws + q.blocks * eblock, q, 27 * CB) : nullptr;
    if (!doJ) {
      const cudaError_t e = launch_cell<double, double, OUT_NONE, true>(Q, u, nullptr, rb, s, q.block0, q.block1);
      const mrgq2::Kinds K = mrgq2::make_kinds(p->g, QRT, q.a, q.b);
      return e != cudaSuccess ? e : launch_rows<double>(p, K, nullptr, rb, r, nullptr, false, true, ovw, s);
    }
    float* ef = mrg_piece_array<float>(q.ws, q, ENT * CB);
    double* ed = mrg_piece_array<double>(q.ws, q, ENT * CB);
    if (fp32)
      return doR ? launch_slabs<float, double, true>(p, Q, q, u, ef, rb, r, (float*)J, ovw, s)
                 : launch_slabs<float, float, false>(p, Q, q, u, ef, nullptr, r, (float*)J, ovw, s);
    return doR ? launch_slabs<double, double, true>(p, Q, q, u, ed, rb, r, (double*)J, ovw, s)
               : launch_slabs<double, double, false>(p, Q, q, u, ed, nullptr, r, (double*)J, ovw, s);
  });
}
