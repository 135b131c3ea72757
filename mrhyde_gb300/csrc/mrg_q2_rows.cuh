// CSR rows of Q2 graphs by kind of node.  Along each axis a node is a vertex (up to 5 couplings, 2 cells) or a
// mid-side node (3 couplings, 1 cell); the 8 (2-D: 4) kinds are grids of their own, flattened one after the other
// over the CTAs, so that the lanes of a warp run the same unrolled code on rows of one length.  Rows of a kind are
// not neighbours in CSR: a warp stages one z plane of its 32 rows in shared memory and writes it with consecutive
// lanes on consecutive addresses.
#pragma once

#include <type_traits>

#include "mrg_device.cuh"
#include "mrg_internal.h"

namespace mrgq2 {

constexpr int PLANE = 25;  // most entries of a row in one z plane

__host__ __device__ constexpr int len(int P) { return P ? 3 : 5; }    // couplings along an axis (P: mid-side)
__host__ __device__ constexpr int half(int P) { return P ? 1 : 2; }
__host__ __device__ constexpr int cells(int P) { return P ? 1 : 2; }

struct Kinds {
  int m[8][3];        // nodes of a kind per axis
  int z0;             // first cell layer
  int64_t block0[9];  // first block of a kind; block0[8]: all blocks
};

// the rows of all nodes, or of the node planes 2 c0 .. 2 c1 - 1 (with the last plane when c1 is the last layer)
inline Kinds make_kinds(const Grid& g, int rows_per_block, int c0 = 0, int c1 = -1) {
  Kinds K;
  int64_t blocks = 0;
  if (c1 < 0) c1 = g.nc[2];
  K.z0 = c0;
  for (int t = 0; t < 8; ++t) {
    int64_t rows = 1;
    for (int k = 0; k < 3; ++k) {
      const int mid = (t >> k) & 1;
      const int n = k == 2 ? c1 - c0 : g.nc[k];
      const bool end = k != 2 || c1 == g.nc[2];
      K.m[t][k] = k < g.dim ? (mid || !end ? n : n + 1) : (mid ? 0 : 1);  // 2-D: kinds 0 to 3 only
      rows *= K.m[t][k];
    }
    K.block0[t] = blocks;
    blocks += (rows + rows_per_block - 1) / rows_per_block;
  }
  K.block0[8] = blocks;
  return K;
}

__device__ __forceinline__ int kind_of(const Kinds& K, int64_t block) {
  int kind = 0;
#pragma unroll
  for (int t = 1; t < 8; ++t)
    if (block >= K.block0[t]) kind = t;
  return kind;
}

// One thread's row: number `at` of its kind (x fastest)
template <bool D3, int PX, int PY, int PZ>
struct Row {
  static constexpr int LX = len(PX), LY = len(PY), LZ = D3 ? len(PZ) : 1, N = LX * LY;
  int ix, iy, iz, cx, cy, cz;
  bool on, fixed, all_whole;            // a row; a Dirichlet row; every lane's row has all its couplings
  bool xl, xr, yl, yr, zl, zr;          // cells on either side of a vertex
  int64_t n, rp;

  __device__ __forceinline__ Row(const Grid& g, const Kinds& K, int kind, int64_t at) {
    const int (&m)[3] = K.m[kind];
    on = at < (int64_t)m[0] * m[1] * m[2];
    ix = PX;
    iy = PY;
    iz = D3 ? PZ : 0;
    if (on) {
      const unsigned a = (unsigned)at, t = a / (unsigned)m[0];
      ix += 2 * (int)(a - t * (unsigned)m[0]);
      iy += 2 * (int)(t % (unsigned)m[1]);
      if (D3) iz += 2 * (K.z0 + (int)(t / (unsigned)m[1]));
    }
    xl = PX || ix > 0;
    xr = PX || ix < g.nn[0] - 1;
    yl = PY || iy > 0;
    yr = PY || iy < g.nn[1] - 1;
    zl = !D3 || PZ || iz > 0;
    zr = !D3 || PZ || iz < g.nn[2] - 1;
    cx = (xl && xr) ? LX : 3;
    cy = (yl && yr) ? LY : 3;
    cz = D3 ? ((zl && zr) ? LZ : 3) : 1;
    fixed = on && node_fixed(g, ix, iy, iz);
    n = ix + (int64_t)g.nn[0] * (iy + (int64_t)g.nn[1] * iz);
    rp = on ? g.P[2][iz] * g.T[1] * g.T[0] + (int64_t)cz * (g.P[1][iy] * g.T[0] + (int64_t)cy * g.P[0][ix]) : 0;
    all_whole = __all_sync(0xffffffffu, on && cx == LX && cy == LY && cz == LZ);
  }
  // whether the coupling at offset o along an axis exists (l, r: the sides' cells)
  __device__ __forceinline__ bool has_z(int o) const { return !D3 || PZ || o == 0 || (o < 0 ? zl : zr); }
  __device__ __forceinline__ bool has_y(int o) const { return PY || o == 0 || (o < 0 ? yl : yr); }
  __device__ __forceinline__ bool has_x(int o) const { return PX || o == 0 || (o < 0 ? xl : xr); }
  // the cell on side s of the node (mid-side node: its cell)
  __device__ __forceinline__ bool cell(const Grid& g, int sx, int sy, int sz, int64_t& c) const {
    const int x = PX ? ix / 2 : ix / 2 - 1 + sx, y = PY ? iy / 2 : iy / 2 - 1 + sy;
    const int z = !D3 ? 0 : (PZ ? iz / 2 : iz / 2 - 1 + sz);
    c = x + (int64_t)g.nc[0] * (y + (int64_t)g.nc[1] * z);
    return on && x >= 0 && x < g.nc[0] && y >= 0 && y < g.nc[1] && z >= 0 && z < g.nc[2];
  }
  // the entry (ey, ex) of the staged plane
  template <typename JT>
  __device__ __forceinline__ void put(JT* stage, int ez, int ey, int ex, JT v) const {
    const int lane = threadIdx.x & 31;
    if (all_whole) stage[lane * N + ey * LX + ex] = v;
    else if (has_z(D3 ? ez - half(PZ) : 0) && has_y(ey - half(PY)) && has_x(ex - half(PX)))
      stage[lane * PLANE + (ey - (yl ? 0 : half(PY))) * cx + (ex - (xl ? 0 : half(PX)))] = v;
  }
  // write (or add) the staged plane ez of the warp's rows; STREAM: past the caches (thermal rows, 33 x 30 x 27 cells:
  // 80.0 -> 78.3 us; rows gathered from element matrices, 64^3 cells: 1050 -> 1061, so not there)
  template <bool OVW, bool STREAM, typename JT>
  __device__ __forceinline__ void store_plane(JT* __restrict__ J, const JT* stage, int ez) const {
    const int lane = threadIdx.x & 31;
    __syncwarp();
    if (all_whole) {
      const int64_t base = rp + (int64_t)ez * N;
#pragma unroll 5
      for (int i = 0; i < N; ++i) {
        const int e = i * 32 + lane, row = e / N;
        const int64_t d = __shfl_sync(0xffffffffu, base, row) + (e - row * N);
        if constexpr (!OVW) J[d] += stage[e];
        else if constexpr (STREAM) __stcs(J + d, stage[e]);
        else J[d] = stage[e];
      }
    } else {
      const int64_t base = rp + (int64_t)(ez - (zl ? 0 : half(PZ))) * cx * cy;
      const int count = (on && has_z(D3 ? ez - half(PZ) : 0)) ? cx * cy : 0;
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
  // a Dirichlet row's diagonal after the warp's additions of zeros (overwrite: staged with the row)
  template <typename JT>
  __device__ __forceinline__ void fix_diagonal(JT* __restrict__ J) const {
    const int dx = xl ? half(PX) : 0, dy = yl ? half(PY) : 0, dz = !D3 ? 0 : (zl ? half(PZ) : 0);
    if (fixed) J[rp + ((int64_t)dz * cy + dy) * cx + dx] = JT(1);
  }
};

// f(kind constants) for the block's kind
template <bool D3, typename F>
__device__ __forceinline__ void with_kind(int kind, F&& f) {
#define MRG_Q2_KIND(T)                                                                                          \
  case T:                                                                                                       \
    f(std::integral_constant<int, (T) & 1>{}, std::integral_constant<int, ((T) >> 1) & 1>{},                    \
      std::integral_constant<int, D3 ? ((T) >> 2) & 1 : 1>{});                                                  \
    break;
  if constexpr (D3) {
    switch (kind) {
      MRG_Q2_KIND(0) MRG_Q2_KIND(1) MRG_Q2_KIND(2) MRG_Q2_KIND(3)
      MRG_Q2_KIND(4) MRG_Q2_KIND(5) MRG_Q2_KIND(6) MRG_Q2_KIND(7)
    }
  } else {
    switch (kind) { MRG_Q2_KIND(0) MRG_Q2_KIND(1) MRG_Q2_KIND(2) MRG_Q2_KIND(3) }
  }
#undef MRG_Q2_KIND
}

}  // namespace mrgq2
