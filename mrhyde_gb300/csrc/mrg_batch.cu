// Batched multiscale-subgrid solves (configuration C4): thousands of independent steady-thermal Q1
// hexahedral problems of uneven size, assembled and solved in one persistent launch.
//
// Reference: the multiscale manager solves each macro element's local problem one at a time on the
// host (src/managers/multiscale/multiscaleManager.cpp:866 -> src/subgrid/subgridDtN.cpp:985 ->
// src/subgrid/subgridDtN_solver.cpp:136, assembly :681, nonlinear solve :903), each with its own
// workset assembly and linear solve.  Here one CTA owns one local problem at a time, taken from an
// atomic work queue ordered largest-first; everything a problem needs happens inside that CTA:
//
//   1. u = Dirichlet data on the boundary, 0 inside (setDirichlet);
//   2. FP32 Jacobian of the problem written to its canonical CSR (factored form kappa_c * K_ref of
//      identical box cells, consistent diagonal), 1/diag kept in registers;
//   3. FP64 residual r = b - A(u) (matrix-free factored form, FP64 kappa);
//   4. refinement loop: FP32 Jacobi-PCG on A32 d = r (the FP32 operator) to the inner tolerance, u += d (FP64),
//      FP64 residual again, until ||r||_inf / ||r_0||_inf <= tol (the reference's Newton test).
//
// Interior rows only are worked on (every boundary node is a Dirichlet node).  A thread owns up to R rows of one
// (x, y) column and marches up it: each cell layer's kappa sums meet the node planes below and above once, so a row
// of the FP32 operator takes about 40 operations and 13 shared-memory reads, where reading its 27 stored entries
// touched 27 lines a load instruction (the stored rows are written once and not read again).  Columns of a large
// problem fill the CTA; those of a small one are cut into segments.  r, q and p of the rows stay in registers,
// x and 1/diag in the thread's own shared-memory slots, p also in shared memory for the neighbours, with kappa.  Reductions are block
// reductions in a fixed order, so a problem's result does not depend on which CTA ran it or on what else was
// running: the same bits alone or in the mix.  No grid-wide synchronisation, no spinning.
// Measured (per-axis cells 4 to 16, 256 threads, 2 CTAs per SM): 700 problems 1938 -> 622 us, 4096 problems 6.32 ->
// 2.28 ms a launch; one 16^3 problem 1264 -> 395 us.
#include <algorithm>
#include <cmath>
#include <numeric>
#include <vector>

#include "mrg_internal.h"

struct BatchProb {
  int nx, ny, nz, pad;
  int64_t cell_off, node_off, nnz_off;
  double Kp[8];
  float Kp32[8];
  float Kc32[8];  // classes of the FP32 operator; class 0 balances the others
  float Kc0_lo;   // and what it lacks
  double load;  // f * vol / 8
};

struct mrg_batch {
  int nprob = 0;
  int64_t ncell = 0, nnode = 0, nnz = 0;
  int max_nodes = 0, max_cells = 0;
  BatchProb* d_probs = nullptr;
  int32_t* d_order = nullptr;
  double* d_kappa = nullptr;
  float* d_kappa32 = nullptr;
  double* d_g = nullptr;
  int* d_counter = nullptr;
  mrg_batch_stat* d_stats = nullptr;
  std::vector<BatchProb> probs;
  // tuned launch configuration
  int threads = 256;
  int ctas_per_sm = 2;
  double f = 1.0;
  cudaGraphExec_t graph = nullptr;
  const void* graph_key[4] = {nullptr, nullptr, nullptr, nullptr};
  int graph_threads = 0, graph_ctas = 0;
  cudaStream_t graph_stream = nullptr;
  double graph_tol[2] = {0, 0};
  int graph_iters[2] = {0, 0};
};

namespace {

struct BatchArgs {
  const BatchProb* probs;
  const int32_t* order;
  int nprob;
  const double* kappa;
  const float* kappa32;
  const double* g;
  double* u;
  float* J;
  int* counter;
  mrg_batch_stat* stats;
  double tol, inner_tol;
  int max_outer, max_inner;
  int max_nodes, max_cells;  // of the largest problem: lengths of the shared-memory arrays
};

// Block sums of FP32 per-thread partials (the inner solve is FP32): warp tree, one partial per warp in
// shared memory, one barrier, then every thread adds the warp partials in the same fixed order (same
// value everywhere, independent of scheduling).  The partial buffers alternate between two halves, so a
// reduction never overwrites partials that a slower thread may still be reading from the previous one:
// between a write to a half and the previous reads of that half lies the barrier of the reduction in
// between.
template <int T>
__device__ __forceinline__ float2 bsum2(float a, float b, float* red, int& half) {
  constexpr int NW = T / 32;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_down_sync(0xffffffffu, a, o);
    b += __shfl_down_sync(0xffffffffu, b, o);
  }
  float* buf = red + half * (2 * NW);
  if ((threadIdx.x & 31) == 0) {
    buf[threadIdx.x >> 5] = a;
    buf[NW + (threadIdx.x >> 5)] = b;
  }
  __syncthreads();
  float sa = 0.0f, sb = 0.0f;
#pragma unroll
  for (int w = 0; w < NW; ++w) {
    sa += buf[w];
    sb += buf[NW + w];
  }
  half ^= 1;
  return make_float2(sa, sb);
}

template <int T>
__device__ __forceinline__ double bmax(double v, double* sh) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  double s = 0.0;
#pragma unroll
  for (int i = 0; i < T / 32; ++i) s = fmax(s, sh[i]);
  return s;
}

__device__ __forceinline__ int axis_count(int i, int N) { return (i == 0 || i == N - 1) ? 2 : 3; }
__device__ __forceinline__ int64_t axis_prefix(int i, int N) { return i == 0 ? 0 : (i >= N ? 3LL * N - 2 : 3LL * i - 1); }

__device__ __forceinline__ void nstep_add(float& sum, float& comp, float v) {
  const float t = sum + v;
  comp += (fabsf(sum) >= fabsf(v)) ? (sum - t) + v : (v - t) + sum;
  sum = t;
}

// Sums of one cell layer's kappa over the cells that a node (x, y) of the plane below or above shares with the
// node at (dx, dy): single cells at the corners, pairs, all four.
template <typename T>
struct Layer {
  T k00, k10, k01, k11, xm, xp, ym, yp, all;
  __device__ __forceinline__ void load(const T* k, int nx) {
    k00 = k[0];
    k10 = k[1];
    k01 = k[nx];
    k11 = k[nx + 1];
    ym = k00 + k10;
    yp = k01 + k11;
    xm = k00 + k01;
    xp = k10 + k11;
    all = ym + yp;
  }
};

// The 3 x 3 values of a node plane around a column
template <typename T>
struct Plane {
  T v[9];
  __device__ __forceinline__ void load(const T* p, int NX) {
#pragma unroll
    for (int k = 0; k < 9; ++k) v[k] = p[(k % 3 - 1) + NX * (k / 3 - 1)];
  }
};

// Sums over the classes (own column, x neighbours, y neighbours, diagonal neighbours) of S * value
template <typename T>
__device__ __forceinline__ void class_sums(const Layer<T>& L, const Plane<T>& P, T c[4]) {
  c[0] = L.all * P.v[4];
  c[1] = fma(L.xp, P.v[5], L.xm * P.v[3]);
  c[2] = fma(L.yp, P.v[7], L.ym * P.v[1]);
  c[3] = fma(L.k11, P.v[8], fma(L.k01, P.v[6], fma(L.k10, P.v[2], L.k00 * P.v[0])));
}

// f(k, (A v)_k, v_k) for the rows z0 .. z0 + n - 1 of a column: kap at the column's first cell of layer 0, v at the
// column's node of plane 0.  A row takes the layer below and the layer above; each layer meets the planes below and
// above it once.  FP32: class 0 has a second part K0_lo.
template <int U, int R, typename T, typename F>  // U: steps unrolled
__device__ __forceinline__ void march(const T* K, T K0_lo, const T* kap, int nx, int nxy, const T* v, int NX, int NXY, int z0, int n,
                                      F&& f) {
  Layer<T> L;
  Plane<T> lo, hi;
  T a[4], b[4];  // the lower layer's sums with the plane below it (dz = -1) and above it (dz = 0)
  lo.load(v + (z0 - 1) * NXY, NX);
  hi.load(v + z0 * NXY, NX);
  L.load(kap + (z0 - 1) * nxy, nx);
  class_sums(L, lo, a);
  class_sums(L, hi, b);
#pragma unroll U
  for (int k = 0; k < R; ++k) {
    if (k >= n) break;
    const int z = z0 + k;
    const T own = hi.v[4];
    T a1[4], b1[4];
    L.load(kap + z * nxy, nx);
    class_sums(L, hi, a1);
    hi.load(v + (z + 1) * NXY, NX);
    class_sums(L, hi, b1);
    const T c0 = b[0] + a1[0];
    T q = K[0] * c0;
    if constexpr (sizeof(T) == 4) q = fma(K0_lo, c0, q);
    q = fma(K[4], a[0] + b1[0], q);
#pragma unroll
    for (int c = 1; c < 4; ++c) {
      q = fma(K[c], b[c] + a1[c], q);
      q = fma(K[4 + c], a[c] + b1[c], q);
    }
    f(k, q, own);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      a[c] = a1[c];
      b[c] = b1[c];
    }
  }
}

// T threads, up to R rows of one column a thread.  Dynamic shared memory: p and kappa of the largest problem, x and
// 1/diag of every thread's rows.
template <int T, int R>
__global__ void __launch_bounds__(T, T == 256 ? 2 : 1) k_batch(const BatchArgs A) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float* x_own = reinterpret_cast<float*>(smem_raw) + threadIdx.x;  // row k at [k T]
  float* mi_own = x_own + R * T;
  float* p_sh = reinterpret_cast<float*>(smem_raw) + 2 * R * T;
  float* k_sh = p_sh + A.max_nodes;
  __shared__ float red[2 * 2 * (T / 32)];
  __shared__ double redd[T / 32];
  __shared__ int s_idx;
  int half = 0;
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) s_idx = atomicAdd(A.counter, 1);
    __syncthreads();
    const int idx = s_idx;
    if (idx >= A.nprob) break;
    const int pid = A.order[idx];
    const BatchProb& P = A.probs[pid];
    const int nx = P.nx, ny = P.ny, nz = P.nz, NX = nx + 1, NY = ny + 1, NZ = nz + 1, NXY = NX * NY, nxy = nx * ny;
    const int nn = NXY * NZ;
    const double* kap = A.kappa + P.cell_off;
    const float* kap32 = A.kappa32 + P.cell_off;
    double* u = A.u + P.node_off;
    float* J = A.J + P.nnz_off;
    const double* gv = A.g + P.node_off;
    const int Tx = 3 * NX - 2, Ty = 3 * NY - 2, Tz = 3 * NZ - 2;
    // this thread's rows: column (cx, cy) of the interior, planes z0 .. z0 + n - 1
    const int ncol = (nx - 1) * (ny - 1), nseg = max(1, min(nz - 1, T / ncol)), per = (nz - 2 + nseg) / nseg;
    const int col = (int)threadIdx.x % ncol, seg = (int)threadIdx.x / ncol;
    const int cx = col % (nx - 1) + 1, cy = col / (nx - 1) + 1, z0 = 1 + seg * per;
    const int n = max(0, min(per, nz - z0));
    const int at = cx + NX * cy;           // node of plane 0
    const int ct = (cx - 1) + nx * (cy - 1);  // first of the column's four cells in layer 0
    // ---- 1. Dirichlet data, kappa; 2. FP32 Jacobian ----
    // identity rows first: zeros everywhere, 1 on the boundary rows' diagonals, then the interior rows
    const int nnz = Tx * Ty * Tz;
    for (int k = threadIdx.x; k < nnz; k += T) J[k] = 0.0f;
    for (int k = threadIdx.x; k < nx * ny * nz; k += T) k_sh[k] = kap32[k];
    __syncthreads();
    for (int i = threadIdx.x; i < nn; i += T) {
      const int ix = i % NX, t = i / NX, iy = t % NY, iz = t / NY;
      const bool inside = ix > 0 && ix < NX - 1 && iy > 0 && iy < NY - 1 && iz > 0 && iz < NZ - 1;
      const double g0 = inside ? 0.0 : gv[i];
      u[i] = g0;
      p_sh[i] = 0.0f;
      if (!inside) {
        const int cxn = axis_count(ix, NX), cyn = axis_count(iy, NY), czn = axis_count(iz, NZ);
        const int rp = (int)(axis_prefix(iz, NZ) * Ty * Tx + (int64_t)czn * (axis_prefix(iy, NY) * Tx + (int64_t)cyn * axis_prefix(ix, NX)));
        J[rp + ((iz > 0) * cyn + (iy > 0)) * cxn + (ix > 0)] = 1.0f;
      }
    }
    for (int k = 0; k < n; ++k) {
      const int iz = z0 + k;
      float* row = J + (3 * iz - 1) * Ty * Tx + 3 * ((3 * cy - 1) * Tx + 3 * (3 * cx - 1));
      float k32[2][2][2];
#pragma unroll
      for (int c = 0; c < 8; ++c) k32[c >> 2][(c >> 1) & 1][c & 1] = k_sh[ct + (c & 1) + nx * ((c >> 1) & 1) + nxy * (iz - 1 + (c >> 2))];
      float osum = 0.0f, ocomp = 0.0f;
#pragma unroll
      for (int e = 0; e < 27; ++e) {
        const int dx = e % 3 - 1, dy = e / 3 % 3 - 1, dz = e / 9 - 1;
        const int cls = (dx != 0) + 2 * (dy != 0) + 4 * (dz != 0);
        if (cls == 0) continue;
        float s = 0.0f;
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
          for (int b = 0; b < 2; ++b)
#pragma unroll
            for (int a = 0; a < 2; ++a) {
              const bool incl = (dx == 0 || dx == 2 * a - 1) && (dy == 0 || dy == 2 * b - 1) && (dz == 0 || dz == 2 * c - 1);
              if (incl) s += k32[c][b][a];
            }
        const float v = P.Kp32[cls] * s;
        row[e] = v;
        nstep_add(osum, ocomp, v);
      }
      const float dg = -(osum + ocomp);
      row[13] = dg;
      mi_own[k * T] = 1.0f / dg;
    }
    __syncthreads();
    // ---- 3./4. refinement loop ----
    double r0 = 0.0, rnorm = 0.0;
    int outer = 0, inner_tot = 0, status = MRG_OK;
    float Kc[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) Kc[c] = P.Kc32[c];
    const float Kc0_lo = P.Kc0_lo;
    for (;;) {
      // FP64 residual at u: b - A u, matrix-free
      double amax = 0.0;
      {
        double Kd[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) Kd[c] = P.Kp[c];
        const double b = P.load * 8.0;
        if (n > 0)
          march<1, R, double>(Kd, 0.0, kap + ct, nx, nxy, u + at, NX, NXY, z0, n, [&](int k, double q, double) {
            const double acc = b - q;
            x_own[k * T] = (float)acc;  // scaled below, once the max is known
            amax = fmax(amax, fabs(acc));
          });
      }
      rnorm = bmax<T>(amax, redd);
      if (outer == 0) r0 = rnorm;
      if (!isfinite(rnorm)) { status = MRG_ENUMERIC; break; }
      if (rnorm == 0.0 || rnorm <= A.tol * r0 || outer >= A.max_outer) break;
      // FP32 Jacobi PCG on A32 d = r / ||r||_inf (x0 = 0): the scaled residual is O(1), so FP32 squares and
      // dot products stay far from the FP32 range limits whatever the refinement level (r itself is held
      // in FP32 from here on, as the inner solve is)
      const float sc = (float)(1.0 / rnorm);
      float r[R], pr[R];
      float rrf = 0.0f, rzf = 0.0f;
#pragma unroll
      for (int k = 0; k < R; ++k) {
        if (k >= n) break;
        r[k] = x_own[k * T] * sc;
        x_own[k * T] = 0.0f;
        pr[k] = r[k] * mi_own[k * T];
        p_sh[at + (z0 + k) * NXY] = pr[k];
        rrf = fmaf(r[k], r[k], rrf);
        rzf = fmaf(r[k], pr[k], rzf);
      }
      float2 d2 = bsum2<T>(rrf, rzf, red, half);
      float rr = d2.x, rho = d2.y;
      const float stop2 = (float)A.inner_tol * (float)A.inner_tol * rr;  // ||r||^2 threshold of the inner solve
      int it = 0;
      while (it < A.max_inner && rr > stop2 && stop2 > 0.0f) {
        float q[R];
        float pqf = 0.0f;
        if (n > 0)
          march<R, R, float>(Kc, Kc0_lo, k_sh + ct, nx, nxy, p_sh + at, NX, NXY, z0, n, [&](int k, float v, float own) {
            q[k] = v;
            pqf = fmaf(v, own, pqf);
          });
        const float pq = bsum2<T>(pqf, 0.0f, red, half).x;
        if (!(pq > 0.0f)) { status = MRG_ENUMERIC; break; }
        const float alpha = rho / pq;
        rrf = 0.0f;
        rzf = 0.0f;
#pragma unroll
        for (int k = 0; k < R; ++k) {
          if (k >= n) break;
          x_own[k * T] = fmaf(alpha, pr[k], x_own[k * T]);
          r[k] = fmaf(-alpha, q[k], r[k]);
          const float z = r[k] * mi_own[k * T];
          rrf = fmaf(r[k], r[k], rrf);
          rzf = fmaf(r[k], z, rzf);
        }
        d2 = bsum2<T>(rrf, rzf, red, half);
        rr = d2.x;
        const float beta = d2.y / rho;
        rho = d2.y;
#pragma unroll
        for (int k = 0; k < R; ++k) {
          if (k >= n) break;
          pr[k] = fmaf(beta, pr[k], r[k] * mi_own[k * T]);
          p_sh[at + (z0 + k) * NXY] = pr[k];
        }
        __syncthreads();
        ++it;
      }
      if (status != MRG_OK) break;
      inner_tot += it;
      // u += ||r|| x  (FP64)
#pragma unroll
      for (int k = 0; k < R; ++k) {
        if (k >= n) break;
        u[at + (z0 + k) * NXY] = fma((double)x_own[k * T], rnorm, u[at + (z0 + k) * NXY]);
      }
      __syncthreads();
      ++outer;
    }
    if (threadIdx.x == 0) {
      mrg_batch_stat st;
      st.outer_iterations = outer;
      st.inner_iterations = inner_tot;
      st.rel_residual = (r0 > 0.0) ? rnorm / r0 : 0.0;
      st.status = (status == MRG_OK && !(rnorm <= A.tol * r0 || rnorm == 0.0)) ? MRG_ENOCONV : status;
      A.stats[pid] = st;
    }
  }
}

// Classes of the FP32 operator: the rounded classes of the matrix, and minus their sum for class 0, in two parts, so that a
// row adds up to 0 (its kappa sums have the same total in every class) as a stiffness matrix's does, up to the rounding of
// the sums themselves.
void balanced_classes(const double* Kp, float* Kc, float* Kc0_lo) {
  double total = 0.0;
  for (int c = 1; c < 8; ++c) {
    Kc[c] = (float)Kp[c];
    total += Kc[c];
  }
  Kc[0] = (float)-total;
  *Kc0_lo = (float)(-total - Kc[0]);
}

// box-cell stiffness classes K(|dx|,|dy|,|dz|) (exact integration of the trilinear element):
// K = kx (x) my (x) mz + mx (x) ky (x) mz + mx (x) my (x) kz with 1-D k = [1,-1]/h, m = h [1/3, 1/6]
void box_classes(double hx, double hy, double hz, double* Kp) {
  const double k1[2] = {1.0, -1.0}, m1[2] = {1.0 / 3.0, 1.0 / 6.0};
  for (int c = 0; c < 8; ++c) {
    const int a = c & 1, b = (c >> 1) & 1, d = (c >> 2) & 1;
    Kp[c] = (k1[a] / hx) * (hy * m1[b]) * (hz * m1[d]) + (hx * m1[a]) * (k1[b] / hy) * (hz * m1[d]) +
            (hx * m1[a]) * (hy * m1[b]) * (k1[d] / hz);
  }
}

typedef void (*BatchKernel)(const BatchArgs);

struct KCfg {
  int threads, rows;
  BatchKernel k;
};

// rows per thread: a column of the largest problem (15 x 15 columns of 15 rows for 16^3 cells) is cut into
// floor(threads / columns) segments; with T < 2 * columns the whole column of at most 15 rows is one thread's
const KCfg kCfgs[] = {
    {256, 15, k_batch<256, 15>},
    {512, 8, k_batch<512, 8>},
    {1024, 4, k_batch<1024, 4>},
};

int batch_smem(const KCfg& c, int nodes, int cells) {
  return (2 * c.threads * c.rows + nodes + cells) * (int)sizeof(float);  // x, 1/diag; p; kappa
}
// of the largest problem that a batch may hold
constexpr int MAX_EDGE = 16;
int batch_smem_most(const KCfg& c) {
  return batch_smem(c, (MAX_EDGE + 1) * (MAX_EDGE + 1) * (MAX_EDGE + 1), MAX_EDGE * MAX_EDGE * MAX_EDGE);
}

}  // namespace

extern "C" int mrg_batch_create(const mrg_batch_desc* d, mrg_batch** out) {
  if (!d || !out || !d->sizes || !d->kappa || !d->dirichlet) return mrg_fail(MRG_EINVAL, "mrg_batch_create: null argument");
  *out = nullptr;
  if (d->n_problems < 1) return mrg_fail(MRG_EINVAL, "mrg_batch_create: n_problems must be >= 1");
  mrg_batch* B = new mrg_batch();
  B->nprob = d->n_problems;
  B->f = d->source;
  B->probs.resize(B->nprob);
  for (int k = 0; k < B->nprob; ++k) {
    BatchProb& P = B->probs[k];
    P.nx = d->sizes[3 * k];
    P.ny = d->sizes[3 * k + 1];
    P.nz = d->sizes[3 * k + 2];
    P.pad = 0;
    if (P.nx < 2 || P.ny < 2 || P.nz < 2 || P.nx > MAX_EDGE || P.ny > MAX_EDGE || P.nz > MAX_EDGE) {
      delete B;
      return mrg_fail(MRG_EINVAL, "mrg_batch_create: local problem cells per axis must be in [2, 16]");
    }
    const int64_t nc = (int64_t)P.nx * P.ny * P.nz, nnode = (int64_t)(P.nx + 1) * (P.ny + 1) * (P.nz + 1);
    P.cell_off = B->ncell;
    P.node_off = B->nnode;
    P.nnz_off = B->nnz;
    B->ncell += nc;
    B->nnode += nnode;
    B->nnz += (3LL * (P.nx + 1) - 2) * (3LL * (P.ny + 1) - 2) * (3LL * (P.nz + 1) - 2);
    B->max_nodes = std::max<int>(B->max_nodes, (int)nnode);
    B->max_cells = std::max<int>(B->max_cells, (int)nc);
    const double hx = 1.0 / P.nx, hy = 1.0 / P.ny, hz = 1.0 / P.nz;
    box_classes(hx, hy, hz, P.Kp);
    for (int c = 0; c < 8; ++c) P.Kp32[c] = (float)P.Kp[c];
    balanced_classes(P.Kp, P.Kc32, &P.Kc0_lo);
    P.load = d->source * hx * hy * hz / 8.0;
  }
  for (int64_t c = 0; c < B->ncell; ++c)
    if (!std::isfinite(d->kappa[c])) {
      delete B;
      return mrg_fail(MRG_ENUMERIC, "mrg_batch_create: kappa contains NaN or Inf");
    }
  // CTAs per SM: two share an SM's issue slots and FP64 pipe, so each runs slower but more is in flight.  While the
  // batch is little more than its largest problem for every SM, that problem's own time is the batch's: one.  Work is
  // taken as interior rows times the longest axis (the inner iterations grow with it); the line lies where both measured
  // the same.  Per-axis cells 4 to 16, one / two CTAs: 300 problems (0.35 of the largest one's work per SM) 343 / 532 us,
  // 700 (0.8) 637 / 622, 2000 (2.3) 1677 / 1129; cells 4 to 8: 700 (1.5) 211 / 153.
  double total = 0.0, largest = 0.0;
  for (const BatchProb& P : B->probs) {
    const double w = (double)(P.nx - 1) * (P.ny - 1) * (P.nz - 1) * std::max(P.nx, std::max(P.ny, P.nz));
    total += w;
    largest = std::max(largest, w);
  }
  if (total < 0.75 * largest * mrg_device_sms()) B->ctas_per_sm = 1;
  // largest problems first (longest-processing-time order for the work queue)
  std::vector<int32_t> order(B->nprob);
  std::iota(order.begin(), order.end(), 0);
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
    const BatchProb &A = B->probs[a], &C = B->probs[b];
    return (int64_t)A.nx * A.ny * A.nz > (int64_t)C.nx * C.ny * C.nz;
  });
  std::vector<float> k32(B->ncell);
  for (int64_t c = 0; c < B->ncell; ++c) k32[c] = (float)d->kappa[c];
  auto fail = [&](cudaError_t e, const char* w) {
    int st = mrg_cuda_check(e, w);
    mrg_batch_destroy(B);
    return st;
  };
  cudaError_t e;
  if ((e = cudaMalloc(&B->d_probs, B->nprob * sizeof(BatchProb))) != cudaSuccess) return fail(e, "cudaMalloc probs");
  if ((e = cudaMalloc(&B->d_order, B->nprob * sizeof(int32_t))) != cudaSuccess) return fail(e, "cudaMalloc order");
  if ((e = cudaMalloc(&B->d_kappa, B->ncell * sizeof(double))) != cudaSuccess) return fail(e, "cudaMalloc kappa");
  if ((e = cudaMalloc(&B->d_kappa32, B->ncell * sizeof(float))) != cudaSuccess) return fail(e, "cudaMalloc kappa32");
  if ((e = cudaMalloc(&B->d_g, B->nnode * sizeof(double))) != cudaSuccess) return fail(e, "cudaMalloc dirichlet");
  if ((e = cudaMalloc(&B->d_counter, sizeof(int))) != cudaSuccess) return fail(e, "cudaMalloc counter");
  if ((e = cudaMalloc(&B->d_stats, B->nprob * sizeof(mrg_batch_stat))) != cudaSuccess) return fail(e, "cudaMalloc stats");
  if ((e = cudaMemcpy(B->d_probs, B->probs.data(), B->nprob * sizeof(BatchProb), cudaMemcpyHostToDevice)) != cudaSuccess)
    return fail(e, "upload probs");
  if ((e = cudaMemcpy(B->d_order, order.data(), B->nprob * sizeof(int32_t), cudaMemcpyHostToDevice)) != cudaSuccess)
    return fail(e, "upload order");
  if ((e = cudaMemcpy(B->d_kappa, d->kappa, B->ncell * sizeof(double), cudaMemcpyHostToDevice)) != cudaSuccess)
    return fail(e, "upload kappa");
  if ((e = cudaMemcpy(B->d_kappa32, k32.data(), B->ncell * sizeof(float), cudaMemcpyHostToDevice)) != cudaSuccess)
    return fail(e, "upload kappa32");
  if ((e = cudaMemcpy(B->d_g, d->dirichlet, B->nnode * sizeof(double), cudaMemcpyHostToDevice)) != cudaSuccess)
    return fail(e, "upload dirichlet");
  // the limit belongs to the kernel, not to the batch: always the same, so that no batch takes it from another
  for (const KCfg& c : kCfgs)
    if ((e = cudaFuncSetAttribute(c.k, cudaFuncAttributeMaxDynamicSharedMemorySize, batch_smem_most(c))) != cudaSuccess)
      return fail(e, "batch kernel shared memory");
  *out = B;
  return MRG_OK;
}

extern "C" int mrg_batch_destroy(mrg_batch* B) {
  if (!B) return MRG_EINVAL;
  if (B->graph) cudaGraphExecDestroy(B->graph);
  cudaFree(B->d_probs);
  cudaFree(B->d_order);
  cudaFree(B->d_kappa);
  cudaFree(B->d_kappa32);
  cudaFree(B->d_g);
  cudaFree(B->d_counter);
  cudaFree(B->d_stats);
  delete B;
  return MRG_OK;
}

extern "C" int mrg_batch_get_info(const mrg_batch* B, mrg_batch_info* info, int64_t* node_off, int64_t* nnz_off) {
  if (!B || !info) return mrg_fail(MRG_EINVAL, "mrg_batch_get_info: null argument");
  info->n_problems = B->nprob;
  info->n_cells = B->ncell;
  info->n_nodes = B->nnode;
  info->nnz = B->nnz;
  info->threads = B->threads;
  info->ctas_per_sm = B->ctas_per_sm;
  for (int k = 0; k < B->nprob; ++k) {
    if (node_off) node_off[k] = B->probs[k].node_off;
    if (nnz_off) nnz_off[k] = B->probs[k].nnz_off;
  }
  return MRG_OK;
}

static int launch_batch(mrg_batch* B, double* u, float* J, const mrg_batch_opts* o, int threads, int ctas_per_sm,
                        cudaStream_t s) {
  int dev = 0, nsm = 0;
  MRG_CUDA(cudaGetDevice(&dev));
  MRG_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  const KCfg* cfg = nullptr;
  for (const KCfg& c : kCfgs)
    if (c.threads == threads) cfg = &c;
  if (!cfg) return mrg_fail(MRG_EINVAL, "mrg_batch: unsupported thread count");
  BatchArgs A{B->d_probs, B->d_order, B->nprob, B->d_kappa, B->d_kappa32, B->d_g, u, J, B->d_counter, B->d_stats,
              o->tol, o->inner_tol, o->max_outer, o->max_inner, B->max_nodes, B->max_cells};
  const int smem = batch_smem(*cfg, B->max_nodes, B->max_cells);
  const int grid = std::max(1, std::min(B->nprob, nsm * ctas_per_sm));
  MRG_CUDA(cudaMemsetAsync(B->d_counter, 0, sizeof(int), s));
  cfg->k<<<grid, cfg->threads, smem, s>>>(A);
  MRG_CUDA(cudaGetLastError());
  return MRG_OK;
}

extern "C" int mrg_batch_solve(mrg_batch* B, double* u, float* J, const mrg_batch_opts* o, mrg_batch_stat* stats,
                               mrg_stream_t stream) {
  if (!B || !u || !J || !o) return mrg_fail(MRG_EINVAL, "mrg_batch_solve: null argument");
  if (!(o->tol > 0.0) || !(o->inner_tol > 0.0) || o->max_outer < 1 || o->max_inner < 1)
    return mrg_fail(MRG_EINVAL, "mrg_batch_solve: bad options");
  cudaStream_t s = (cudaStream_t)stream;
  // one captured graph per (buffers, options, configuration, stream): counter reset + persistent launch
  const bool same = B->graph && B->graph_key[0] == u && B->graph_key[1] == J && B->graph_threads == B->threads &&
                    B->graph_ctas == B->ctas_per_sm && B->graph_stream == s && B->graph_tol[0] == o->tol &&
                    B->graph_tol[1] == o->inner_tol && B->graph_iters[0] == o->max_outer &&
                    B->graph_iters[1] == o->max_inner;
  if (!same) {
    if (B->graph) cudaGraphExecDestroy(B->graph);
    B->graph = nullptr;
    cudaStream_t cs = s;
    bool own = false;
    if (!s) {
      MRG_CUDA(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
      own = true;
    }
    cudaGraph_t gph;
    MRG_CUDA(cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal));
    int rc = launch_batch(B, u, J, o, B->threads, B->ctas_per_sm, cs);
    cudaError_t e = cudaStreamEndCapture(cs, &gph);
    if (own) cudaStreamDestroy(cs);
    if (rc) return rc;
    if (e != cudaSuccess) return mrg_cuda_check(e, "capture batch solve");
    e = cudaGraphInstantiate(&B->graph, gph, 0);
    cudaGraphDestroy(gph);
    if (e != cudaSuccess) return mrg_cuda_check(e, "instantiate batch solve");
    B->graph_key[0] = u;
    B->graph_key[1] = J;
    B->graph_threads = B->threads;
    B->graph_ctas = B->ctas_per_sm;
    B->graph_stream = s;
    B->graph_tol[0] = o->tol;
    B->graph_tol[1] = o->inner_tol;
    B->graph_iters[0] = o->max_outer;
    B->graph_iters[1] = o->max_inner;
  }
  MRG_CUDA(cudaGraphLaunch(B->graph, s));
  if (stats) {
    MRG_CUDA(cudaMemcpyAsync(stats, B->d_stats, B->nprob * sizeof(mrg_batch_stat), cudaMemcpyDeviceToHost, s));
    MRG_CUDA(cudaStreamSynchronize(s));
    for (int k = 0; k < B->nprob; ++k)
      if (stats[k].status != MRG_OK) return mrg_fail(stats[k].status, "mrg_batch_solve: a local problem did not converge");
  }
  return MRG_OK;
}

// Autotuner: times the whole batch for each (threads, CTAs per SM) configuration that fits and keeps
// the fastest.  The buffers are scratch for the trials (their contents are overwritten).
extern "C" int mrg_batch_autotune(mrg_batch* B, double* u, float* J, const mrg_batch_opts* o, mrg_stream_t stream) {
  if (!B || !u || !J || !o) return mrg_fail(MRG_EINVAL, "mrg_batch_autotune: null argument");
  cudaStream_t s = (cudaStream_t)stream;
  cudaEvent_t e0, e1;
  MRG_CUDA(cudaEventCreate(&e0));
  MRG_CUDA(cudaEventCreate(&e1));
  float best = 1e30f;
  int bt = B->threads, bc = B->ctas_per_sm;
  for (const KCfg& c : kCfgs) {
    for (int cps : {1, 2, 4, 8}) {
      if (c.threads * cps > 2048) continue;
      int rc = launch_batch(B, u, J, o, c.threads, cps, s);  // warm
      if (rc) continue;
      MRG_CUDA(cudaEventRecord(e0, s));
      rc = launch_batch(B, u, J, o, c.threads, cps, s);
      MRG_CUDA(cudaEventRecord(e1, s));
      MRG_CUDA(cudaEventSynchronize(e1));
      float ms = 0.f;
      MRG_CUDA(cudaEventElapsedTime(&ms, e0, e1));
      if (rc == MRG_OK && ms < best) {
        best = ms;
        bt = c.threads;
        bc = cps;
      }
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  B->threads = bt;
  B->ctas_per_sm = bc;
  return MRG_OK;
}

extern "C" int mrg_batch_set_config(mrg_batch* B, int32_t threads, int32_t ctas_per_sm) {
  if (!B) return mrg_fail(MRG_EINVAL, "mrg_batch_set_config: null batch");
  bool ok = false;
  for (const KCfg& c : kCfgs)
    if (c.threads == threads) ok = true;
  if (!ok || ctas_per_sm < 1 || ctas_per_sm > 16) return mrg_fail(MRG_EINVAL, "mrg_batch_set_config: unsupported");
  B->threads = threads;
  B->ctas_per_sm = ctas_per_sm;
  return MRG_OK;
}
