// Pressure projection (projection_3d.py ProjectionSolver3D, fft_pcg path).
//
// Operator (projection_3d.py:66-175 _fill_var_density_data with alpha_g = 1):
//   A p = div((1/rho_face) grad p) + 1e-6 p, rho floored at 0.01,
//   x: Neumann inlet / Dirichlet p=0 outlet face; y periodic;
//   z: Neumann wall / Dirichlet p=0 top face; non-uniform dz.
// Row k of A carries 1/dz_k, so S = -diag(dz) A is symmetric positive
// definite; S is face conductances g (one per interior face) plus a per-cell
// term e (Dirichlet faces and the -dz_k 1e-6 shift):
//   (S x)_c = e_c x_c + sum_faces g_f (x_c - x_nb),
// stored on the coarse levels and on the finest in FP32, formed from 1/rho on the
// finest in FP64.
// The reference solves A p = rhs with BiCGSTAB + an FFT preconditioner
// (projection_3d.py:756-791); here S p = -dz rhs is solved with CG
// preconditioned by one geometric-multigrid V-cycle:
//   * coarse cells aggregate 2x2x2 fine cells (odd tails keep 1);
//   * coarse operator = 1/2 (P^T S P) with piecewise-constant P, which keeps
//     the face-conductance form (coarse face = sum of fine faces across it);
//   * nu pre- and nu post-sweeps of damped Jacobi (default nu = 4, omega = 0.9:
//     fewer CG iterations than 0.8 at the same cost per iteration, measured);
//   * the coarsest level (<= 64 cells) is solved with a dense inverse built
//     at each rebuild.
// The stopping test mirrors scipy's: ||b - A x||_2 < rtol ||b||_2 on the
// unsymmetrised system, warm-started from the previous solution.
#include <vector>
#include <chrono>
#include <cstdlib>
#include <cmath>
#include "common.cuh"
#include "kernels.h"

#define PROJ_EPS 1.0e-6
#define MG_OMEGA 0.8          // damping of the coarsest level's smoothing-only solve
#define MG_OMEGA_DEFAULT 0.9  // damping of the V-cycle's smoothing sweeps
#define MG_NU_DEFAULT 4
#define MG_COARSE_MAX 48
// blocks of the pointwise reducing kernels (8 per SM of the 148: enough loads in
// flight to stream HBM)
#define RED_BLOCKS 1184
#define RED_THREADS 256
// Device scalar slots: 0 rz, 1 pq, 2 rz_new, 4 ||b_A||^2, 5 ||r_A||^2,
// 6 (rtol ||b_A||)^2, 7 converged flag, 8 iterations done.
#define SC_DONE 7
#define SC_IT 8
// Kernels of a PCG iteration return at once when the solve has converged,
// so iterations queued past convergence change nothing.
#define PCG_SKIP(done) \
  FOLLOW();            \
  if ((done) && *(done) != 0.0) return;

// a level's extents with the divisions that recover (i, j, k) from a flat index
struct Dims {
  int nx, ny, nz;
  FastDiv fnx, fny;
};
inline Dims dims_make(int nx, int ny, int nz) {
  Dims D;
  D.nx = nx; D.ny = ny; D.nz = nz;
  D.fnx = fastdiv_make((uint32_t)nx);
  D.fny = fastdiv_make((uint32_t)ny);
  return D;
}

// The operator of a level >= 1: face conductances and the per-cell term.
template <typename T>
struct OpA {
  const T *gx, *gy, *gz, *e;
};
// Level 0's, from the reciprocal density alone: a face conductance is a factor
// of its direction and level times the sum of the two cells' 1/rho, so a sweep
// reads one field where the stored form read four.  tab: OP_TAB factors a level
// (x face, y face, z face above and below, the shift, the outlet and top faces).
#define OP_TAB 8
template <typename T>
struct OpI {
  const T *ir, *tab;
};

// Level 0's in FP32, stored (the FP64 operator rounded once): what the mixed
// form's steps have always been preconditioned with.  Formed in FP32 from 1/rho it
// gives another iterate within the solve's tolerance, and a step's extinction
// thresholds then fall to the other side in some cells.
template <typename T>
struct OpZ : OpA<T> {};

template <typename T>
struct MGLevelT {
  int nx, ny, nz;
  Dims dims;
  int64_t n;
  // conductances and per-cell term (levels >= 1; level 0 only when it is the
  // coarsest), 1/diag
  T *gx, *gy, *gz, *e, *dinv;
  T *x, *b, *t, *s;            // correction, rhs, temps
};
using MGLevel = MGLevelT<double>;

struct ProjCtx {
  GridDev g;
  int nlev;
  MGLevel lev[16];
  double* Ainv;       // dense inverse at the coarsest level
  double* pc_r;       // PCG residual (level 0)
  double* pc_z;
  double* pc_p;
  double* pc_p2;      // the directions of odd iterations
  double* pc_q;
  double* rhs;        // b_S
  double* partial;    // block partial sums
  double* scal;       // device scalars
  double* h_scal;     // pinned host mirror
  double* p_prev;     // warm start / solution (owned)
  double* ir;         // 1/max(rho, 0.01)
  double* tab;        // level 0's factors (OP_TAB per level)
  int have_prev;
  int last_iters;     // CG iterations of the previous solve (batch size hint)
  cudaStream_t cs;    // private stream for graph capture
  cudaGraphExec_t iter_exec;  // one captured PCG iteration (0 until captured)
  int iter_kernels;   // kernels in that graph
  int graph_failed;
  int nu;             // Jacobi sweeps before and after the coarse correction
  int nu0;            // the same on the finest level (0: nu)
  double omega;       // Jacobi damping
  int tail_on;        // coarse levels in one launch (k_mg_vcycle_tail)
  // mixed-precision form: the V-cycle in FP32 (levels, coarse inverse, the
  // residual it smooths and the correction it returns); CG stays FP64
  int fp32;
  MGLevelT<float> lev32[16];
  float* Ainv32;
  float *r32, *z32;
  // host-side statistics of the last solve (ms): total, fetch waits (sum, max),
  // graph-launch calls (sum, max), fetches, iteration launches, iterations
  double stats[8];
  // learned form: flexible CG preconditioned by a U-Net (unet.cu), falling
  // back to V-cycle PCG from the current iterate when it stalls
  void* net;
  int max_learned;    // learned iterations before the fallback
  double stall;       // fallback when the residual norm shrinks by less than
                      // this factor per iteration (over the last 3)
  double* log_r0;     // optional copies of the starting residual / iterate
  double* log_x0;
  // last solve: learned iterations, V-cycle iterations, fell back (0/1);
  // then the number of fallbacks since creation
  double fcg[4];
};

// ---------------------------------------------------------------------------
// 1/rho (floored) and, by the first block, level 0's factors
__global__ void k_proj_ir(GridDev g, const double* rho, double* ir, double* tab,
                          double dx2, double dy2) {
  FOLLOW();
  const int64_t n = ncells_dev(g);
  const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (blockIdx.x == 0) {
    for (int k = threadIdx.x; k < g.nz; k += blockDim.x) {
      const double dz = g.dz[k];
      const double v[OP_TAB] = {dz * (0.5 / dx2), dz * (0.5 / dy2), 0.5 / g.da[k],
                                k > 0 ? 0.5 / g.da[k - 1] : 0.0, -dz * PROJ_EPS, dz * (2.0 / dx2),
                                2.0 / dz, 0.0};
      for (int q = 0; q < OP_TAB; ++q) tab[k * OP_TAB + q] = v[q];
    }
  }
  if (c >= n) return;
  const double r = rho[c];
  const double m = (r >= 0.01 || r != r) ? r : 0.01;
  ir[c] = 1.0 / m;
}

// the operator's parts: conductance of the face towards +x, +y, +z of cell c
// (0 where there is none) and the per-cell term
template <typename T>
__device__ __forceinline__ T op_fx(const OpA<T>& o, int64_t c, int, int, int) { return o.gx[c]; }
template <typename T>
__device__ __forceinline__ T op_fy(const OpA<T>& o, int64_t c, int64_t, int) { return o.gy[c]; }
template <typename T>
__device__ __forceinline__ T op_fz(const OpA<T>& o, int64_t c, int64_t, int, int) { return o.gz[c]; }
template <typename T>
__device__ __forceinline__ T op_e(const OpA<T>& o, int64_t c, int, int, int, int) { return o.e[c]; }
template <typename T>
__device__ __forceinline__ T op_fx(const OpI<T>& o, int64_t c, int i, int k, int nx) {
  return i < nx - 1 ? o.tab[k * OP_TAB] * (o.ir[c] + o.ir[c + 1]) : T(0);
}
template <typename T>
__device__ __forceinline__ T op_fy(const OpI<T>& o, int64_t c, int64_t cp, int k) {
  return o.tab[k * OP_TAB + 1] * (o.ir[c] + o.ir[cp]);
}
template <typename T>
__device__ __forceinline__ T op_fz(const OpI<T>& o, int64_t c, int64_t sz, int k, int nz) {
  return k < nz - 1 ? o.tab[k * OP_TAB + 2] * (o.ir[c] + o.ir[c + sz]) : T(0);
}
template <typename T>
__device__ __forceinline__ T op_e(const OpI<T>& o, int64_t c, int i, int k, int nx, int nz) {
  T e = o.tab[k * OP_TAB + 4];
  if (i == nx - 1) e += o.tab[k * OP_TAB + 5] * o.ir[c];
  if (k == nz - 1) e += o.tab[k * OP_TAB + 6] * o.ir[c];
  return e;
}

// diagonal of the operator -> 1/diag
template <typename T, typename Op>
__global__ void k_mg_diag(Dims D, Op o, T* dinv) {
  FOLLOW();
  const int nx = D.nx, ny = D.ny, nz = D.nz;
  int64_t n = (int64_t)nx * ny * nz;
  int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (c >= n) return;
  int i, j, k;
  split_cell((uint32_t)c, D.fnx, D.fny, i, j, k);
  int64_t sy = nx, sz = (int64_t)nx * ny;
  const int64_t r = c - (int64_t)j * sy;
  const int jp = j + 1 < ny ? j + 1 : 0, jm = j > 0 ? j - 1 : ny - 1;
  T d = op_e(o, c, i, k, nx, nz) + op_fx(o, c, i, k, nx);
  if (ny > 1) d += op_fy(o, c, r + (int64_t)jp * sy, k);
  d += op_fz(o, c, sz, k, nz);
  if (i > 0) d += op_fx(o, c - 1, i - 1, k, nx);
  if (ny > 1) d += op_fy(o, r + (int64_t)jm * sy, c, k);
  if (k > 0) d += op_fz(o, c - sz, sz, k - 1, nz);
  dinv[c] = T(1) / d;
}

// level 0's operator as arrays (in FP32; in FP64 only where level 0 is the
// coarsest level)
template <typename T>
__global__ void k_op_arrays(Dims D, OpI<double> o, T* gx, T* gy, T* gz, T* e) {
  FOLLOW();
  const int64_t n = (int64_t)D.nx * D.ny * D.nz, sz = (int64_t)D.nx * D.ny;
  const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (c >= n) return;
  int i, j, k;
  split_cell((uint32_t)c, D.fnx, D.fny, i, j, k);
  const int jp = j + 1 < D.ny ? j + 1 : 0;
  gx[c] = (T)op_fx(o, c, i, k, D.nx);
  gy[c] = D.ny > 1 ? (T)op_fy(o, c, c + (int64_t)(jp - j) * D.nx, k) : T(0);
  gz[c] = (T)op_fz(o, c, sz, k, D.nz);
  e[c] = (T)op_e(o, c, i, k, D.nx, D.nz);
}

__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }

// A vector the operator is applied to, cell by cell: stored; the first sweep's
// iterate from x = 0, w b / d; an iterate plus the prolonged coarse correction
// (piecewise constant).  The latter two are formed where they are read, so
// neither the first sweep nor the prolongation is a pass of its own.
template <typename T>
struct VecX {
  const T* x;
  __device__ __forceinline__ T at(int c, int, int, int) const { return x[c]; }
};
template <typename T>
struct VecFirst {
  const T *b, *dinv;
  T w;
  // (rounded as the stored value would be: no product left to contract)
  __device__ __forceinline__ T at(int c, int, int, int) const {
    return mul_rn(w * b[c], dinv[c]);
  }
};
template <typename T>
struct VecProl {
  const T *x, *xc;
  int cx, cy;
  __device__ __forceinline__ T at(int c, int i, int j, int k) const {
    return x[c] + xc[((k >> 1) * cy + (j >> 1)) * cx + (i >> 1)];
  }
};

// (S x)_c; xc = x_c
template <typename T, typename V>
__device__ __forceinline__ T mg_apply(int nx, int ny, int nz, const OpA<T>& o, const V& x, T xc,
                                      int c, int i, int j, int k) {
  const int sy = nx, sz = nx * ny;
  T y = o.e[c] * xc;
  if (i < nx - 1) y += o.gx[c] * (xc - x.at(c + 1, i + 1, j, k));
  if (i > 0) y += o.gx[c - 1] * (xc - x.at(c - 1, i - 1, j, k));
  if (ny > 1) {
    int jp = j + 1 < ny ? j + 1 : 0;
    int jm = j > 0 ? j - 1 : ny - 1;
    int cp = c + (jp - j) * sy;
    int cm = c + (jm - j) * sy;
    y += o.gy[c] * (xc - x.at(cp, i, jp, k));
    y += o.gy[cm] * (xc - x.at(cm, i, jm, k));
  }
  if (k < nz - 1) y += o.gz[c] * (xc - x.at(c + sz, i, j, k + 1));
  if (k > 0) y += o.gz[c - sz] * (xc - x.at(c - sz, i, j, k - 1));
  return y;
}
template <typename T, typename V>
__device__ __forceinline__ T mg_apply(int nx, int ny, int nz, const OpI<T>& o, const V& x, T xc,
                                      int c, int i, int j, int k) {
  const int sy = nx, sz = nx * ny;
  const T* ir = o.ir;
  const T* tb = o.tab + k * OP_TAB;
  const T r = ir[c], hx = tb[0], hy = tb[1];
  T e = tb[4];
  if (i == nx - 1) e += tb[5] * r;
  if (k == nz - 1) e += tb[6] * r;
  T y = e * xc;
  if (i < nx - 1) y += hx * (r + ir[c + 1]) * (xc - x.at(c + 1, i + 1, j, k));
  if (i > 0) y += hx * (r + ir[c - 1]) * (xc - x.at(c - 1, i - 1, j, k));
  if (ny > 1) {
    int jp = j + 1 < ny ? j + 1 : 0;
    int jm = j > 0 ? j - 1 : ny - 1;
    int cp = c + (jp - j) * sy;
    int cm = c + (jm - j) * sy;
    y += hy * (r + ir[cp]) * (xc - x.at(cp, i, jp, k));
    y += hy * (r + ir[cm]) * (xc - x.at(cm, i, jm, k));
  }
  if (k < nz - 1) y += tb[2] * (r + ir[c + sz]) * (xc - x.at(c + sz, i, j, k + 1));
  if (k > 0) y += tb[3] * (r + ir[c - sz]) * (xc - x.at(c - sz, i, j, k - 1));
  return y;
}

// Galerkin aggregation of level f into level c (coarse = scale * P^T S_f P)
template <typename T, typename Op>
__global__ void k_mg_coarsen(int fx, int fy, int fz, Op o, Dims DC, T* gxc, T* gyc, T* gzc, T* ec,
                             double scale_) {
  FOLLOW();
  const int cx = DC.nx, cy = DC.ny, cz = DC.nz;
  int64_t n = (int64_t)cx * cy * cz;
  int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (q >= n) return;
  int I, J, K;
  split_cell((uint32_t)q, DC.fnx, DC.fny, I, J, K);
  const int64_t fsy = fx, fsz = (int64_t)fx * fy;
  const int i0 = 2 * I, i1 = min(2 * I + 1, fx - 1);
  const int j0 = 2 * J, j1 = min(2 * J + 1, fy - 1);
  const int k0 = 2 * K, k1 = min(2 * K + 1, fz - 1);
  const int jp = j1 + 1 < fy ? j1 + 1 : 0;
  T se = 0.0, sx = 0.0, sy = 0.0, sz = 0.0;
  // (every load at a clamped index and none behind a branch: all are in flight at
  // once, where loops up to the extents took 9 to 12 us on the smallest levels)
#pragma unroll
  for (int d = 0; d < 8; ++d) {
    const int k = min(k0 + (d >> 2), k1), j = min(j0 + ((d >> 1) & 1), j1), i = min(i0 + (d & 1), i1);
    const T v = op_e(o, (int64_t)k * fsz + (int64_t)j * fsy + i, i, k, fx, fz);
    if (k == k0 + (d >> 2) && j == j0 + ((d >> 1) & 1) && i == i0 + (d & 1)) se += v;
  }
#pragma unroll
  for (int d = 0; d < 4; ++d) {
    const int a = d >> 1, b = d & 1;
    const int ka = min(k0 + a, k1), ja = min(j0 + a, j1), jb = min(j0 + b, j1), ib = min(i0 + b, i1);
    const int64_t ck = (int64_t)ka * fsz;
    const T vx = op_fx(o, ck + (int64_t)jb * fsy + i1, i1, ka, fx);
    const T vy = op_fy(o, ck + (int64_t)j1 * fsy + ib, ck + (int64_t)jp * fsy + ib, ka);
    const T vz = op_fz(o, (int64_t)k1 * fsz + (int64_t)ja * fsy + ib, fsz, k1, fz);
    const bool ka_in = ka == k0 + a, ja_in = ja == j0 + a, jb_in = jb == j0 + b, ib_in = ib == i0 + b;
    if (I < cx - 1 && ka_in && jb_in) sx += vx;
    if (cy > 1 && ka_in && ib_in) sy += vy;
    if (K < cz - 1 && ja_in && ib_in) sz += vz;
  }
  const T scale = (T)scale_;
  gxc[q] = scale * sx;
  gyc[q] = scale * sy;
  gzc[q] = scale * sz;
  ec[q] = scale * se;
}

// Dense inverse of the coarsest operator (Gauss-Jordan in shared memory, n <= 64).
template <typename T>
__global__ void k_mg_coarse_inverse(int nx, int ny, int nz, const T* gx,
                                    const T* gy, const T* gz,
                                    const T* e, T* Ainv) {
  FOLLOW();
  __shared__ T M[MG_COARSE_MAX][2 * MG_COARSE_MAX + 1];
  const int n = nx * ny * nz;
  const int t = threadIdx.x;
  for (int e_ = t; e_ < n * 2 * n; e_ += blockDim.x) M[e_ / (2 * n)][e_ % (2 * n)] = 0.0;
  __syncthreads();
  if (t == 0) {
    const int sy = nx, sz = nx * ny;
    for (int c = 0; c < n; ++c) {
      int i = c % nx, j = (c / nx) % ny, k = c / (nx * ny);
      M[c][c] += e[c];
      if (i < nx - 1) { M[c][c] += gx[c]; M[c][c + 1] -= gx[c]; }
      if (i > 0) { M[c][c] += gx[c - 1]; M[c][c - 1] -= gx[c - 1]; }
      if (ny > 1) {
        int jp = j + 1 < ny ? j + 1 : 0, jm = j > 0 ? j - 1 : ny - 1;
        int cp = c - j * sy + jp * sy, cm = c - j * sy + jm * sy;
        M[c][c] += gy[c]; M[c][cp] -= gy[c];
        M[c][c] += gy[cm]; M[c][cm] -= gy[cm];
      }
      if (k < nz - 1) { M[c][c] += gz[c]; M[c][c + sz] -= gz[c]; }
      if (k > 0) { M[c][c] += gz[c - sz]; M[c][c - sz] -= gz[c - sz]; }
      M[c][n + c] = 1.0;
    }
  }
  __syncthreads();
  // a warp takes whole rows (the columns are its lanes), so a pivot step is a few
  // shared-memory operations deep; with a thread per row it was 2 n deep (149 us
  // for 48 cells, 16 now)
  const int lane = t & 31, wid = t >> 5, nwarps = blockDim.x >> 5;
  for (int piv = 0; piv < n; ++piv) {
    const T d = M[piv][piv];
    __syncthreads();
    for (int q = t; q < 2 * n; q += blockDim.x) M[piv][q] /= d;
    __syncthreads();
    for (int r = wid; r < n; r += nwarps) {
      if (r == piv) continue;
      const T f = M[r][piv];
      __syncwarp();
      if (f != 0.0)
        for (int q = lane; q < 2 * n; q += 32) M[r][q] -= f * M[piv][q];
    }
    __syncthreads();
  }
  for (int e_ = t; e_ < n * n; e_ += blockDim.x) Ainv[e_] = M[e_ / n][n + e_ % n];
}

template <typename T>
__global__ void k_mg_coarse_solve(int n, const T* Ainv,
                                  const T* b, T* x, const double* done) {
  PCG_SKIP(done);
  int r = threadIdx.x;
  if (r >= n) return;
  T s = 0.0;
  for (int q = 0; q < n; ++q) s += Ainv[r * n + q] * b[q];
  x[r] = s;
}

// damped Jacobi sweep: xo = x + w (b - S x) / d
template <typename T, typename Op, typename V>
__global__ void k_mg_jacobi(Dims D, Op o, const T* dinv, const T* b, V x,
                            T* xo, double w_, const double* done) {
  PCG_SKIP(done);
  const int nx = D.nx, ny = D.ny, nz = D.nz;
  const T w = (T)w_;
  int64_t n = (int64_t)nx * ny * nz;
  int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (c >= n) return;
  int i, j, k;
  split_cell((uint32_t)c, D.fnx, D.fny, i, j, k);
  const T xc = x.at(c, i, j, k);
  T r = b[c] - mg_apply(nx, ny, nz, o, x, xc, c, i, j, k);
  xo[c] = xc + w * r * dinv[c];
}
// the first sweep from x = 0 alone (where it is the only one)
template <typename T>
__global__ void k_mg_first(int64_t n, const T* dinv, const T* b, T* xo,
                           double w_, const double* done) {
  PCG_SKIP(done);
  int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (c < n) xo[c] = (T)w_ * b[c] * dinv[c];
}

// the sum over the eight lanes of a coarse cell, in order (as one thread adds
// the children up)
template <typename T>
__device__ __forceinline__ T octet_sum(T v) {
  const int base = threadIdx.x & 24;
  T s = T(0);
#pragma unroll
  for (int q = 0; q < 8; ++q) s += __shfl_sync(0xffffffffu, v, base + q);
  return s;
}

// coarse rhs = sum over children of the fine residual (b - S x): a lane a child
// (with a thread a coarse cell the eight children's loads came one after the
// other: 11 to 14 us on levels of a few thousand cells)
template <typename T, typename Op>
__global__ void k_mg_restrict_residual(Dims DF, Op o, const T* b, const T* x, Dims DC, T* bc,
                                       const double* done) {
  PCG_SKIP(done);
  const int fx = DF.nx, fy = DF.ny, fz = DF.nz;
  const int64_t n = (int64_t)DC.nx * DC.ny * DC.nz;
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, qu = t >> 3;
  const int64_t q = qu < n ? qu : n - 1;
  int I, J, K;
  split_cell((uint32_t)q, DC.fnx, DC.fny, I, J, K);
  const int i = 2 * I + (t & 1), j = 2 * J + ((t >> 1) & 1), k = 2 * K + ((t >> 2) & 1);
  T v = T(0);
  if (k < fz && j < fy && i < fx) {
    const int c = (k * fy + j) * fx + i;
    v = b[c] - mg_apply(fx, fy, fz, o, VecX<T>{x}, x[c], c, i, j, k);
  }
  const T s = octet_sum(v);
  if (qu < n && (t & 7) == 0) bc[q] = s;
}

// ---------------------------------------------------------------------------
// deterministic FP64 dot products: fixed block count, fixed reduction tree
// ---------------------------------------------------------------------------
__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// A kernel's sum: every block leaves its partial, and one small block adds them
// (a thread every FIN_THREADS-th, then a tree: the same order each time) and does
// the scalar work that follows (post).  (Adding them in the kernel's own last
// block, found by a ticket, took 25 us more at the 5850 blocks of level 0's tiles:
// the tickets queue at one address.)
#define POST_NONE 0
#define POST_DIR 1    // rz of this iteration becomes the old one (slot 0 = slot 2)
#define POST_CHECK 2  // end of a PCG iteration: count it, ||r_A|| < rtol ||b_A||
#define FIN_THREADS 1024
__device__ __forceinline__ double block_sum(double v, double* sh) {
  const int tid = (threadIdx.z * blockDim.y + threadIdx.y) * blockDim.x + threadIdx.x;
  const int lane = tid & 31, wid = tid >> 5;
  v = warp_sum(v);
  if (lane == 0) sh[wid] = v;
  __syncthreads();
  double s = 0.0;
  const int nw = (int)(blockDim.x * blockDim.y * blockDim.z) >> 5;
  if (wid == 0) s = warp_sum(lane < nw ? sh[lane] : 0.0);
  return s;  // in thread 0
}
__device__ __forceinline__ void store_partial(double v, double* partial) {
  __shared__ double sh[32];
  const double s = block_sum(v, sh);
  if ((threadIdx.x | threadIdx.y | threadIdx.z) == 0)
    partial[blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z)] = s;
}
__global__ void __launch_bounds__(FIN_THREADS)
    k_finish_sum(const double* partial, int nb, double* scal, int slot, int post,
                 const double* done) {
  PCG_SKIP(done);
  __shared__ double sh[32];
  double t = 0.0;
  for (int q = threadIdx.x; q < nb; q += FIN_THREADS) t += partial[q];
  t = block_sum(t, sh);
  if (threadIdx.x == 0) {
    scal[slot] = t;
    if (post == POST_DIR) scal[0] = scal[2];
    if (post == POST_CHECK) {
      scal[SC_IT] += 1.0;
      if (t < scal[6]) scal[SC_DONE] = 1.0;
    }
  }
}

// rhs: b_S = -dz_k (div - target)/dt, plus ||(div - target)/dt||^2
__global__ void k_proj_rhs(GridDev g, const double* u, const double* v,
                           const double* w, const double* u_in,
                           const double* target, double inv_dx, double inv_dy,
                           double inv_dt, double* bS, double* partial) {
  FOLLOW();
  const int64_t n = ncells_dev(g);
  const int nx = g.nx, ny = g.ny;
  const int64_t sy = nx, sz = (int64_t)nx * ny;
  double acc = 0.0;
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < n;
       c += (int64_t)gridDim.x * blockDim.x) {
    int i, j, k;
    split_cell((uint32_t)c, g.fnx, g.fny, i, j, k);
    const double dz = g.dz[k];
    const double ul = i > 0 ? u[c - 1] : u_in[(int64_t)k * ny + j];
    double div = (u[c] - ul) * inv_dx;
    if (ny > 1) {
      int jm = j > 0 ? j - 1 : ny - 1;
      div += (v[c] - v[c - (int64_t)j * sy + (int64_t)jm * sy]) * inv_dy;
    }
    div += (w[c] - (k > 0 ? w[c - sz] : 0.0)) / dz;
    if (target) div = div - target[c];
    const double rA = div * inv_dt;
    bS[c] = -dz * rA;
    acc += rA * rA;
  }
  store_partial(acc, partial);
}

// ---------------------------------------------------------------------------
// Level 0's kernels: blocks of consecutive cells, W = 2 neighbours in x a thread
// where nx is even (every row then starts on a pair), one where it is odd.  The
// load/store unit bounds them: a sweep of single cells takes 57 wavefronts for
// 32 cells and 31.7 us at 400 x 120 x 60; pairs loaded as one vector, with the
// x-neighbours taken from the lanes beside, take as many for 64.
// ---------------------------------------------------------------------------
#define Z_THREADS 256
template <typename T>
struct alignas(2 * sizeof(T)) Two {
  T a, b;
};
template <typename T>
__device__ __forceinline__ Two<T> ld2(const T* p) {
  return *(const Two<T>*)p;
}
template <typename T>
__device__ __forceinline__ Two<T> at2(const VecX<T>& x, int c, int, int, int) {
  return ld2(x.x + c);
}
template <typename T>
__device__ __forceinline__ Two<T> at2(const VecFirst<T>& x, int c, int, int, int) {
  const Two<T> b = ld2(x.b + c), d = ld2(x.dinv + c);
  return {mul_rn(x.w * b.a, d.a), mul_rn(x.w * b.b, d.b)};
}
template <typename T>
__device__ __forceinline__ Two<T> at2(const VecProl<T>& x, int c, int i, int j, int k) {
  const Two<T> v = ld2(x.x + c);
  const T e = x.xc[((k >> 1) * x.cy + (j >> 1)) * x.cx + (i >> 1)];
  return {v.a + e, v.b + e};
}
// The search direction where it is read: z + beta p (p the last direction;
// first iteration z).  Z: the type the preconditioner leaves z in.
template <typename Z>
struct VecDir {
  const Z* z;
  const double* p;
  double beta;
  __device__ __forceinline__ double at(int c, int, int, int) const {
    return beta == 0.0 ? (double)z[c] : (double)z[c] + beta * p[c];
  }
};
template <typename Z>
__device__ __forceinline__ Two<double> at2(const VecDir<Z>& x, int c, int, int, int) {
  const Two<Z> z = ld2(x.z + c);
  if (x.beta == 0.0) return {(double)z.a, (double)z.b};
  const Two<double> p = ld2(x.p + c);
  return {(double)z.a + x.beta * p.a, (double)z.b + x.beta * p.b};
}

// a thread's W cells: the first of them (all threads get one, for the shuffles;
// in: it is theirs)
struct ZCell {
  int c, i, j, k;
  bool in;
};
template <int W>
__device__ __forceinline__ ZCell z_cell(const Dims& D) {
  const int n = D.nx * D.ny * D.nz;
  ZCell z;
  z.c = (int)(blockIdx.x * Z_THREADS + threadIdx.x) * W;
  z.in = z.c < n;
  if (!z.in) z.c = n - W;
  split_cell((uint32_t)z.c, D.fnx, D.fny, z.i, z.j, z.k);
  return z;
}
inline int z_width(const Dims& D) { return D.nx % 2 == 0 ? 2 : 1; }
inline int z_blocks(const Dims& D) {
  const int w = z_width(D);
  return (int)(((int64_t)D.nx * D.ny * D.nz / w + Z_THREADS - 1) / Z_THREADS);
}

// x and S x at W cells
template <int W, typename T, typename V>
__device__ __forceinline__ void z_apply(const Dims& D, const OpI<T>& o, const V& x, int c, int i,
                                        int j, int k, T (&xc)[W], T (&y)[W]) {
  const int nx = D.nx, ny = D.ny, nz = D.nz;
  if constexpr (W == 1) {
    xc[0] = x.at(c, i, j, k);
    y[0] = mg_apply(nx, ny, nz, o, x, xc[0], c, i, j, k);
  } else {
    const int sy = nx, sz = nx * ny, lane = threadIdx.x & 31;
    const T* ir = o.ir;
    const T* tb = o.tab + k * OP_TAB;
    const int jp = j + 1 < ny ? j + 1 : 0, jm = j > 0 ? j - 1 : ny - 1;
    const int cp = c + (jp - j) * sy, cm = c + (jm - j) * sy;
    const int kp = min(k + 1, nz - 1), km = max(k - 1, 0);
    const int ch = c + (kp - k) * sz, cl = c - (k - km) * sz;
    const Two<T> X = at2(x, c, i, j, k), R = ld2(ir + c);
    const Two<T> xp = at2(x, cp, i, jp, k), rp = ld2(ir + cp);
    const Two<T> xm = at2(x, cm, i, jm, k), rm = ld2(ir + cm);
    const Two<T> xh = at2(x, ch, i, j, kp), rh = ld2(ir + ch);
    const Two<T> xl = at2(x, cl, i, j, km), rl = ld2(ir + cl);
    T xe = __shfl_down_sync(0xffffffffu, X.a, 1), re = __shfl_down_sync(0xffffffffu, R.a, 1);
    T xw = __shfl_up_sync(0xffffffffu, X.b, 1), rw = __shfl_up_sync(0xffffffffu, R.b, 1);
    if (lane == 31 && i + 2 < nx) { xe = x.at(c + 2, i + 2, j, k); re = ir[c + 2]; }
    if (lane == 0 && i > 0) { xw = x.at(c - 1, i - 1, j, k); rw = ir[c - 1]; }
    const T hx = tb[0], hy = tb[1], hh = tb[2], hl = tb[3];
    T ea = tb[4], eb = ea;
    if (i + 2 == nx) eb += tb[5] * R.b;
    if (k == nz - 1) { ea += tb[6] * R.a; eb += tb[6] * R.b; }
    T ya = ea * X.a, yb = eb * X.b;
    ya += hx * (R.a + R.b) * (X.a - X.b);
    if (i + 2 < nx) yb += hx * (R.b + re) * (X.b - xe);
    if (i > 0) ya += hx * (R.a + rw) * (X.a - xw);
    yb += hx * (R.b + R.a) * (X.b - X.a);
    if (ny > 1) {
      ya += hy * (R.a + rp.a) * (X.a - xp.a);
      yb += hy * (R.b + rp.b) * (X.b - xp.b);
      ya += hy * (R.a + rm.a) * (X.a - xm.a);
      yb += hy * (R.b + rm.b) * (X.b - xm.b);
    }
    if (k < nz - 1) {
      ya += hh * (R.a + rh.a) * (X.a - xh.a);
      yb += hh * (R.b + rh.b) * (X.b - xh.b);
    }
    if (k > 0) {
      ya += hl * (R.a + rl.a) * (X.a - xl.a);
      yb += hl * (R.b + rl.b) * (X.b - xl.b);
    }
    xc[0] = X.a; xc[1] = X.b;
    y[0] = ya; y[1] = yb;
  }
}
template <int W, typename T, typename V>
__device__ __forceinline__ void z_apply(const Dims& D, const OpA<T>& o, const V& x, int c, int i,
                                        int j, int k, T (&xc)[W], T (&y)[W]) {
  const int nx = D.nx, ny = D.ny, nz = D.nz;
  if constexpr (W == 1) {
    xc[0] = x.at(c, i, j, k);
    y[0] = mg_apply(nx, ny, nz, o, x, xc[0], c, i, j, k);
  } else {
    const int sy = nx, sz = nx * ny, lane = threadIdx.x & 31;
    const int jp = j + 1 < ny ? j + 1 : 0, jm = j > 0 ? j - 1 : ny - 1;
    const int cp = c + (jp - j) * sy, cm = c + (jm - j) * sy;
    const int kp = min(k + 1, nz - 1), km = max(k - 1, 0);
    const int ch = c + (kp - k) * sz, cl = c - (k - km) * sz;
    const Two<T> X = at2(x, c, i, j, k), gx = ld2(o.gx + c), e = ld2(o.e + c);
    const Two<T> xp = at2(x, cp, i, jp, k), xm = at2(x, cm, i, jm, k);
    const Two<T> xh = at2(x, ch, i, j, kp), xl = at2(x, cl, i, j, km);
    const Two<T> gp = ld2(o.gy + c), gm = ld2(o.gy + cm), gh = ld2(o.gz + c), gl = ld2(o.gz + cl);
    T xe = __shfl_down_sync(0xffffffffu, X.a, 1), xw = __shfl_up_sync(0xffffffffu, X.b, 1);
    T gw = __shfl_up_sync(0xffffffffu, gx.b, 1);
    if (lane == 31 && i + 2 < nx) xe = x.at(c + 2, i + 2, j, k);
    if (lane == 0 && i > 0) { xw = x.at(c - 1, i - 1, j, k); gw = o.gx[c - 1]; }
    T ya = e.a * X.a, yb = e.b * X.b;
    ya += gx.a * (X.a - X.b);
    if (i + 2 < nx) yb += gx.b * (X.b - xe);
    if (i > 0) ya += gw * (X.a - xw);
    yb += gx.a * (X.b - X.a);
    if (ny > 1) {
      ya += gp.a * (X.a - xp.a);
      yb += gp.b * (X.b - xp.b);
      ya += gm.a * (X.a - xm.a);
      yb += gm.b * (X.b - xm.b);
    }
    if (k < nz - 1) {
      ya += gh.a * (X.a - xh.a);
      yb += gh.b * (X.b - xh.b);
    }
    if (k > 0) {
      ya += gl.a * (X.a - xl.a);
      yb += gl.b * (X.b - xl.b);
    }
    xc[0] = X.a; xc[1] = X.b;
    y[0] = ya; y[1] = yb;
  }
}
template <int W, typename T>
__device__ __forceinline__ void z_load(const T* p, int c, T (&v)[W]) {
  if constexpr (W == 2) {
    const Two<T> t = ld2(p + c);
    v[0] = t.a; v[1] = t.b;
  } else {
    v[0] = p[c];
  }
}
template <int W, typename T>
__device__ __forceinline__ void z_store(T* p, int c, const T (&v)[W]) {
  if constexpr (W == 2) *(Two<T>*)(p + c) = Two<T>{v[0], v[1]};
  else p[c] = v[0];
}

// damped Jacobi sweep; with DOT the sum of rd * (the new iterate) as well (the
// V-cycle's last sweep: r.z)
template <int W, bool DOT, typename T, typename Op, typename V>
__global__ void __launch_bounds__(Z_THREADS, 4)
    k_z_jacobi(Dims D, Op o, const T* dinv, const T* b, V x, T* xo,
               double w_, const double* rd, double* partial, const double* done) {
  PCG_SKIP(done);
  const ZCell z = z_cell<W>(D);
  T bc[W], dc[W], xc[W], y[W], v[W];
  z_load<W>(b, z.c, bc);
  z_load<W>(dinv, z.c, dc);
  z_apply<W>(D, o, x, z.c, z.i, z.j, z.k, xc, y);
#pragma unroll
  for (int q = 0; q < W; ++q) v[q] = xc[q] + (T)w_ * (bc[q] - y[q]) * dc[q];
  if (z.in) z_store<W>(xo, z.c, v);
  if (DOT) {
    double acc = 0.0, rr[W];
    z_load<W>(rd, z.c, rr);
    if (z.in)
#pragma unroll
      for (int q = 0; q < W; ++q) acc += rr[q] * (double)v[q];
    store_partial(acc, partial);
  }
}

// coarse rhs = sum over children of the fine residual, a coarse cell a thread
template <typename T, typename Op>
__global__ void __launch_bounds__(Z_THREADS, 4)
    k_z_restrict(Dims D, Op o, const T* b, const T* x, Dims DC, T* bc,
                 const double* done) {
  PCG_SKIP(done);
  const ZCell z = z_cell<1>(DC);
  T s = T(0);
#pragma unroll
  for (int dk = 0; dk < 2; ++dk)
#pragma unroll
    for (int dj = 0; dj < 2; ++dj) {
      const int k = min(2 * z.k + dk, D.nz - 1), j = min(2 * z.j + dj, D.ny - 1), i = 2 * z.i;
      const int c = (k * D.ny + j) * D.nx + i;
      T xc[2], y[2], r[2];
      z_load<2>(b, c, r);
      z_apply<2>(D, o, VecX<T>{x}, c, i, j, k, xc, y);
      if (2 * z.k + dk < D.nz && 2 * z.j + dj < D.ny) {
        s += r[0] - y[0];
        s += r[1] - y[1];
      }
    }
  if (z.in) bc[z.c] = s;
}

// q = S p and p.q, with p = z + beta p of the last iteration formed on the way
// into the other of the two direction buffers
template <int W, typename Z>
__global__ void __launch_bounds__(Z_THREADS, 4)
    k_z_matvec_dir(Dims D, OpI<double> o, const Z* zv, double* p0, double* p1,
                   double* q, const double* scal, double* partial) {
  PCG_SKIP(scal + SC_DONE);
  const int it = (int)scal[SC_IT];
  const VecDir<Z> x{zv, it & 1 ? p0 : p1, it == 0 ? 0.0 : scal[2] / scal[0]};
  double* pn = it & 1 ? p1 : p0;
  const ZCell z = z_cell<W>(D);
  double pc[W], y[W], acc = 0.0;
  z_apply<W>(D, o, x, z.c, z.i, z.j, z.k, pc, y);
  if (z.in) {
    z_store<W>(pn, z.c, pc);
    z_store<W>(q, z.c, y);
#pragma unroll
    for (int e = 0; e < W; ++e) acc += pc[e] * y[e];
  }
  store_partial(acc, partial);
}
// q = S p and p.q of a stored vector (W = 1 for a caller's: any alignment)
template <int W>
__global__ void __launch_bounds__(Z_THREADS, 4)
    k_z_matvec(Dims D, OpI<double> o, const double* p, double* q, double* partial,
               const double* done) {
  PCG_SKIP(done);
  const ZCell z = z_cell<W>(D);
  double pc[W], y[W], acc = 0.0;
  z_apply<W>(D, o, VecX<double>{p}, z.c, z.i, z.j, z.k, pc, y);
  if (z.in) {
    z_store<W>(q, z.c, y);
#pragma unroll
    for (int e = 0; e < W; ++e) acc += pc[e] * y[e];
  }
  if (partial) store_partial(acc, partial);
}

// r = b - S x (also in FP32 where the preconditioner is), ||r_A||^2 with
// r_A = -r / dz_k
template <int W>
__global__ void __launch_bounds__(Z_THREADS, 4)
    k_z_residual(GridDev g, Dims D, OpI<double> o, const double* b,
                 const double* x, double* r, float* r32, double* partial) {
  FOLLOW();
  const ZCell z = z_cell<W>(D);
  double xc[W], y[W], v[W], acc = 0.0;
  z_load<W>(b, z.c, v);
  z_apply<W>(D, o, VecX<double>{x}, z.c, z.i, z.j, z.k, xc, y);
  if (z.in) {
    const double dz = g.dz[z.k];
#pragma unroll
    for (int e = 0; e < W; ++e) {
      v[e] -= y[e];
      if (r32) r32[z.c + e] = (float)v[e];
      const double ra = v[e] / dz;
      acc += ra * ra;
    }
    z_store<W>(r, z.c, v);
  }
  store_partial(acc, partial);
}

// x += alpha p ; r -= alpha q ; ||r_A||^2   (alpha = rz / pq from device scalars;
// p: the buffer of this iteration's parity, or p0 with p1 null)
__global__ void k_pcg_update(GridDev g, double* x, double* r, float* r32,
                             const double* p0, const double* p1,
                             const double* q, const double* scal,
                             double* partial) {
  PCG_SKIP(scal + SC_DONE);
  const int64_t n = ncells_dev(g);
  const double alpha = scal[0] / scal[1];
  const double* p = p1 && ((int)scal[SC_IT] & 1) ? p1 : p0;
  double acc = 0.0;
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < n;
       c += (int64_t)gridDim.x * blockDim.x) {
    x[c] += alpha * p[c];
    double rr = r[c] - alpha * q[c];
    r[c] = rr;
    if (r32) r32[c] = (float)rr;
    double ra = rr / g.dz[(int)fdiv(fdiv((uint32_t)c, g.fnx), g.fny)];
    acc += ra * ra;
  }
  store_partial(acc, partial);
}

// a.b
__global__ void k_dot(int64_t n, const double* a, const double* b,
                      double* partial, const double* done) {
  PCG_SKIP(done);
  double acc = 0.0;
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < n;
       c += (int64_t)gridDim.x * blockDim.x)
    acc += a[c] * b[c];
  store_partial(acc, partial);
}

__global__ void k_set_scal(double* scal, int dst, int src) {
  PCG_SKIP(scal + SC_DONE);
  scal[dst] = scal[src];
}

// start of a solve: tolerance, initial test, iteration count; b == 0 -> x = 0
__global__ void k_pcg_init(double* scal, double rtol2) {
  FOLLOW();
  scal[6] = rtol2 * scal[4];
  scal[SC_IT] = 0.0;
  scal[SC_DONE] = (scal[5] < scal[6] || scal[4] == 0.0) ? 1.0 : 0.0;
}

__global__ void k_zero_if_zero_rhs(int64_t n, const double* scal, double* x) {
  FOLLOW();
  if (scal[4] != 0.0) return;
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < n;
       c += (int64_t)gridDim.x * blockDim.x)
    x[c] = 0.0;
}

// Flexible CG (truncated to one previous direction): p = z - (z.q_prev / p.q_prev) p,
// first iteration p = z.  Slots: 10 z.q_prev, 11 p.q of the previous iteration.
__global__ void k_fcg_dir(int64_t n, const double* scal, const double* z,
                          double* p) {
  PCG_SKIP(scal + SC_DONE);
  int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (c >= n) return;
  if (scal[SC_IT] == 0.0) { p[c] = z[c]; return; }
  const double beta = -scal[10] / scal[11];
  p[c] = z[c] + beta * p[c];
}

// alpha = p.r / p.q into slot 0 (read by k_pcg_update); a zero direction
// (p.q = 0, e.g. a network output of 0) gives alpha = 0, so the residual
// stalls and the solve falls back instead of dividing by zero
__global__ void k_fcg_alpha(double* scal) {
  FOLLOW();
  if (scal[SC_DONE] != 0.0) return;
  const bool ok = scal[1] > 0.0;
  scal[0] = ok ? scal[12] : 0.0;
  if (!ok) scal[1] = 1.0;
}

// out = b - S x (level operator, any precision)
template <typename T>
__global__ void k_lp_residual(Dims D, OpZ<T> o, const T* b, const T* x,
                              T* out) {
  FOLLOW();
  const int nx = D.nx, ny = D.ny, nz = D.nz;
  int64_t n = (int64_t)nx * ny * nz;
  int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (c >= n) return;
  int i, j, k;
  split_cell((uint32_t)c, D.fnx, D.fny, i, j, k);
  out[c] = b[c] - mg_apply(nx, ny, nz, o, VecX<T>{x}, x[c], c, i, j, k);
}

// e1 = float(e0) - t
__global__ void k_lp_err(int64_t n, const double* e0, const float* t,
                         float* e1) {
  FOLLOW();
  int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (c < n) e1[c] = (float)e0[c] - t[c];
}

// restart as V-cycle PCG from the current iterate (the residual was just
// recomputed into slot 5)
__global__ void k_fcg_restart(double* scal) {
  FOLLOW();
  scal[SC_IT] = 0.0;
  scal[SC_DONE] = (scal[5] < scal[6]) ? 1.0 : 0.0;
}

// ---------------------------------------------------------------------------
// velocity correction (projection_3d.py:818-842)
// ---------------------------------------------------------------------------
__global__ void k_proj_correct(GridDev g, double* u, double* v, double* w,
                               const double* p, const double* ir,
                               double dt, double dt_dx, double dt_dy) {
  FOLLOW();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  int j = blockIdx.y * blockDim.y + threadIdx.y;
  int k = blockIdx.z;
  if (i >= g.nx || j >= g.ny) return;
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const int64_t sy = nx, sz = (int64_t)nx * ny;
  int64_t c = cidx(g, k, j, i);
  const double pc = p[c], irc = ir[c];
  if (nx > 2) {
    if (i < nx - 1) u[c] -= dt_dx * (p[c + 1] - pc) * (0.5 * (irc + ir[c + 1]));
    else u[c] += 2.0 * dt_dx * pc * irc;
  }
  if (ny > 1) {
    int jp = j + 1 < ny ? j + 1 : 0;
    int64_t cp = c - (int64_t)j * sy + (int64_t)jp * sy;
    v[c] -= dt_dy * (p[cp] - pc) * (0.5 * (irc + ir[cp]));
  }
  if (nz > 2) {
    if (k < nz - 1) w[c] -= dt * (p[c + sz] - pc) / g.da[k] * (0.5 * (irc + ir[c + sz]));
    else w[c] += 2.0 * dt * pc / g.dz[nz - 1] * irc;
  }
}

// max |div(u) - target| (projection_3d.py:847-892 plain branch)
// (OUT: the divergence is wanted too; without its stores the loads of four cells
// a thread are in flight together)
template <bool OUT>
__global__ void k_div_resid_max(GridDev g, const double* u,
                                const double* v, const double* w,
                                const double* u_in, const double* target,
                                double inv_dx, double inv_dy, double* div_out,
                                unsigned long long* out_key) {
  FOLLOW();
  const int64_t n = ncells_dev(g);
  const int nx = g.nx, ny = g.ny;
  const int64_t sy = nx, sz = (int64_t)nx * ny;
  double best = 0.0;
  bool nan = false;
#pragma unroll 4
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < n;
       c += (int64_t)gridDim.x * blockDim.x) {
    int i, j, k;
    split_cell((uint32_t)c, g.fnx, g.fny, i, j, k);
    double div;
    if (i > 0) div = (u[c] - u[c - 1]) * inv_dx;
    else div = (u[c] - u_in[(int64_t)k * ny + j]) * inv_dx;
    if (ny > 1) {
      int jm = j > 0 ? j - 1 : ny - 1;
      div += (v[c] - v[c - (int64_t)j * sy + (int64_t)jm * sy]) * inv_dy;
    }
    if (k > 0) div += (w[c] - w[c - sz]) / g.dz[k];
    else div += (w[c] - 0.0) / g.dz[0];
    if (OUT) div_out[c] = div;
    if (target) div = div - target[c];
    double a = fabs(div);
    if (a != a) nan = true;
    else if (a > best) best = a;
  }
  unsigned long long key = nan ? 0x7ff8000000000000ull : (unsigned long long)__double_as_longlong(best);
  block_max_to(key, out_key);
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
static double* dalloc(int64_t n) {
  double* p = nullptr;
  if (cudaMalloc(&p, sizeof(double) * (size_t)(n > 0 ? n : 1)) != cudaSuccess) return nullptr;
  return p;
}

void* proj_create(const GridDev& g) {
  ProjCtx* P = new ProjCtx();
  P->g = g;
  int nx = g.nx, ny = g.ny, nz = g.nz;
  int L = 0;
  while (true) {
    MGLevel& lv = P->lev[L];
    lv.nx = nx; lv.ny = ny; lv.nz = nz; lv.n = (int64_t)nx * ny * nz;
    lv.dims = dims_make(nx, ny, nz);
    // level 0's operator is formed from 1/rho, its vectors are the solver's
    const bool arr = L > 0 || lv.n <= MG_COARSE_MAX;
    lv.gx = lv.gy = lv.gz = lv.e = lv.x = lv.b = nullptr;
    if (arr) {
      lv.gx = dalloc(lv.n); lv.gy = dalloc(lv.n); lv.gz = dalloc(lv.n); lv.e = dalloc(lv.n);
      lv.x = dalloc(lv.n); lv.b = dalloc(lv.n);
    }
    lv.dinv = dalloc(lv.n); lv.t = dalloc(lv.n); lv.s = dalloc(lv.n);
    ++L;
    if (lv.n <= MG_COARSE_MAX || L >= 16) break;
    int cx = (nx + 1) / 2, cy = (ny + 1) / 2, cz = (nz + 1) / 2;
    if (cx == nx && cy == ny && cz == nz) break;
    nx = cx; ny = cy; nz = cz;
  }
  P->nlev = L;
  int64_t n0 = P->lev[0].n;
  int64_t nc = P->lev[L - 1].n;
  P->Ainv = dalloc(nc <= MG_COARSE_MAX ? nc * nc : 1);
  P->pc_r = dalloc(n0); P->pc_z = dalloc(n0); P->pc_p = dalloc(n0); P->pc_q = dalloc(n0);
  P->rhs = dalloc(n0);
  const int zb = z_blocks(P->lev[0].dims);
  P->partial = dalloc(zb > RED_BLOCKS ? zb : RED_BLOCKS);
  P->pc_p2 = dalloc(n0);
  P->scal = dalloc(16);
  cudaMallocHost(&P->h_scal, sizeof(double) * 16);
  P->p_prev = dalloc(n0);
  P->ir = dalloc(n0);
  P->tab = dalloc((int64_t)OP_TAB * g.nz);
  {
    // cleared before any solve is queued, on a private stream
    SetupStream ss;
    cudaMemsetAsync(P->p_prev, 0, sizeof(double) * n0, ss.s);
    cudaMemsetAsync(P->scal, 0, sizeof(double) * 16, ss.s);
    ss.sync();
  }
  P->have_prev = 0;
  P->last_iters = 0;
  P->iter_exec = nullptr;
  P->iter_kernels = 0;
  P->graph_failed = 0;
  P->nu = MG_NU_DEFAULT;
  P->nu0 = 0;
  P->tail_on = 1;
  P->fp32 = 0;
  P->Ainv32 = nullptr; P->r32 = nullptr; P->z32 = nullptr;
  for (int l = 0; l < 16; ++l) P->lev32[l] = MGLevelT<float>{};
  for (int q = 0; q < 8; ++q) P->stats[q] = 0.0;
  P->omega = MG_OMEGA_DEFAULT;
  P->net = nullptr;
  P->max_learned = 30;
  P->stall = 0.9;
  P->log_r0 = nullptr;
  P->log_x0 = nullptr;
  for (int q = 0; q < 4; ++q) P->fcg[q] = 0.0;
  cudaStreamCreateWithFlags(&P->cs, cudaStreamNonBlocking);
  if (cudaGetLastError() != cudaSuccess || !P->p_prev) {
    proj_destroy(P);
    return nullptr;
  }
  return P;
}

void proj_destroy(void* h) {
  ProjCtx* P = (ProjCtx*)h;
  if (!P) return;
  for (int l = 0; l < P->nlev; ++l) {
    MGLevel& lv = P->lev[l];
    cudaFree(lv.gx); cudaFree(lv.gy); cudaFree(lv.gz); cudaFree(lv.e); cudaFree(lv.dinv);
    cudaFree(lv.x); cudaFree(lv.b); cudaFree(lv.t); cudaFree(lv.s);
  }
  for (int l = 0; l < P->nlev; ++l) {
    MGLevelT<float>& lv = P->lev32[l];
    cudaFree(lv.gx); cudaFree(lv.gy); cudaFree(lv.gz); cudaFree(lv.e); cudaFree(lv.dinv);
    cudaFree(lv.x); cudaFree(lv.b); cudaFree(lv.t); cudaFree(lv.s);
  }
  cudaFree(P->Ainv32); cudaFree(P->r32); cudaFree(P->z32);
  if (P->iter_exec) cudaGraphExecDestroy(P->iter_exec);
  if (P->cs) cudaStreamDestroy(P->cs);
  cudaFree(P->Ainv); cudaFree(P->pc_r); cudaFree(P->pc_z); cudaFree(P->pc_p); cudaFree(P->pc_q);
  cudaFree(P->pc_p2);
  cudaFree(P->rhs); cudaFree(P->partial); cudaFree(P->scal); cudaFreeHost(P->h_scal);
  cudaFree(P->p_prev); cudaFree(P->ir); cudaFree(P->tab);
  delete P;
}

double* proj_pressure(void* h) { return ((ProjCtx*)h)->p_prev; }
const double* proj_inv_rho(void* h) { return ((ProjCtx*)h)->ir; }
int proj_nlevels(void* h) { return ((ProjCtx*)h)->nlev; }

__global__ void k_cvt_d2f(int64_t n, const double* a, float* b, const double* done) {
  PCG_SKIP(done);
  int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (c < n) b[c] = (float)a[c];
}
__global__ void k_cvt_f2d(int64_t n, const float* a, double* b, const double* done) {
  PCG_SKIP(done);
  int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (c < n) b[c] = (double)a[c];
}

template <typename T>
static OpA<T> op_a(const MGLevelT<T>& f) {
  return OpA<T>{f.gx, f.gy, f.gz, f.e};
}
static OpI<double> op_0(const ProjCtx* P, double) { return OpI<double>{P->ir, P->tab}; }
static OpZ<float> op_0(const ProjCtx* P, float) {
  return OpZ<float>{op_a(P->lev32[0])};
}

template <typename T>
static void rebuild_levels(ProjCtx* P, MGLevelT<T>* lev, T* Ainv, cudaStream_t st) {
  if (sizeof(T) == 4 || P->nlev == 1) {
    MGLevelT<T>& f = lev[0];
    following(k_op_arrays<T>, blocks_for(f.n, 256), 256, 0, st)(f.dims, op_0(P, 0.0), f.gx, f.gy, f.gz, f.e);
    fs_count_launch();
  }
  const auto o0 = op_0(P, T(0));
  typedef std::remove_const_t<decltype(o0)> Op0;
  for (int l = 0; l < P->nlev; ++l) {
    MGLevelT<T>& f = lev[l];
    if (l > 0) {
      MGLevelT<T>& pf = lev[l - 1];
      if (l == 1)
        following(k_mg_coarsen<T, Op0>, blocks_for(f.n, 128), 128, 0, st)(pf.nx, pf.ny, pf.nz, o0, f.dims, f.gx,
                                                             f.gy, f.gz, f.e, 0.5);
      else
        following(k_mg_coarsen<T, OpA<T>>, blocks_for(f.n, 128), 128, 0, st)(pf.nx, pf.ny, pf.nz, op_a(pf), f.dims,
                                                             f.gx, f.gy, f.gz, f.e, 0.5);
      fs_count_launch();
      following(k_mg_diag<T, OpA<T>>, blocks_for(f.n, 256), 256, 0, st)(f.dims, op_a(f), f.dinv);
    } else {
      following(k_mg_diag<T, Op0>, blocks_for(f.n, 256), 256, 0, st)(f.dims, o0, f.dinv);
    }
    fs_count_launch();
  }
  MGLevelT<T>& c = lev[P->nlev - 1];
  if (c.n <= MG_COARSE_MAX) {
    following(k_mg_coarse_inverse<T>, 1, 1024, 0, st)(c.nx, c.ny, c.nz, c.gx, c.gy, c.gz, c.e, Ainv);
    fs_count_launch();
  }
}

int proj_rebuild(void* h, const double* rho, cudaStream_t st) {
  ProjCtx* P = (ProjCtx*)h;
  const GridDev& g = P->g;
  const unsigned nb = blocks_for(P->lev[0].n, 256);
  // the FP64 level-0 operator stays the CG's; the FP32 preconditioner has its own
  following(k_proj_ir, nb, 256, 0, st)(g, rho, P->ir, P->tab, g.dx * g.dx, g.dy * g.dy);
  fs_count_launch();
  if (P->fp32) rebuild_levels<float>(P, P->lev32, P->Ainv32, st);
  else rebuild_levels<double>(P, P->lev, P->Ainv, st);
  return cuda_status();
}

int proj_set_precision(void* h, int fp32) {
  ProjCtx* P = (ProjCtx*)h;
  fp32 = fp32 ? 1 : 0;
  if (fp32 == P->fp32) return FS_OK;
  // (what is there stays: after a call that ran out of memory the next one asks
  // for the rest)
  if (fp32) {
    bool got = true;
    auto have = [&](float*& a, int64_t n) {
      if (!a && cudaMalloc(&a, sizeof(float) * (size_t)(n > 0 ? n : 1)) != cudaSuccess) {
        a = nullptr;
        got = false;
      }
    };
    for (int l = 0; l < P->nlev && got; ++l) {
      MGLevelT<float>& lv = P->lev32[l];
      const MGLevel& ld = P->lev[l];
      lv.nx = ld.nx; lv.ny = ld.ny; lv.nz = ld.nz; lv.n = ld.n; lv.dims = ld.dims;
      float** arrs[9] = {&lv.gx, &lv.gy, &lv.gz, &lv.e, &lv.dinv, &lv.x, &lv.b, &lv.t, &lv.s};
      for (float** a : arrs) have(*a, lv.n);
    }
    const int64_t nc = P->lev[P->nlev - 1].n;
    have(P->Ainv32, nc <= MG_COARSE_MAX ? nc * nc : 1);
    have(P->r32, P->lev[0].n);
    have(P->z32, P->lev[0].n);
    if (!got) return FS_ECUDA;
  }
  P->fp32 = fp32;
  if (P->iter_exec) cudaGraphExecDestroy(P->iter_exec);  // the iteration graph changes
  P->iter_exec = nullptr;
  P->graph_failed = 0;
  return FS_OK;
}

// z = V-cycle(r) on level l (b = rhs, x = result); returns kernels launched
// ---------------------------------------------------------------------------
// The coarse end of the V-cycle in one launch: every level from the first one
// whose tail fits in shared memory (operator, right-hand sides and vectors of
// all coarser levels, plus the coarsest level's dense inverse) down to the
// coarsest and back, in one CTA, with a __syncthreads between the sweeps,
// instead of one launch per sweep (a few microseconds of launch and drain
// each for a few hundred cells).  The first tail level's right-hand side
// comes from global memory and its correction goes back there.  The order of
// operations and every per-cell expression are those of vcycle() with
// k_mg_jacobi, k_mg_restrict_residual and k_mg_coarse_solve, so
// the correction is bit-identical.
#define MG_TAIL_SMEM (200 * 1024)
#define MG_TAIL_MAX 10
#define MG_TAIL_THREADS 512
template <typename T>
struct MGTail {
  MGLevelT<T> lev[MG_TAIL_MAX];  // the tail's levels (global arrays), finest first
  int nl, nu;
  double omega;
  const T* Ainv;
};

// elements of shared memory the tail of levels lev[0..nl-1] needs
template <typename T>
__host__ __device__ inline int64_t tail_smem_elems(const MGLevelT<T>* lev, int nl) {
  int64_t e = 0;
  for (int q = 0; q < nl; ++q) e += 9 * lev[q].n;
  const int64_t nc = lev[nl - 1].n;
  return e + (nc <= MG_COARSE_MAX ? nc * nc : 0);
}

// A level in shared memory: its extents and where its nine arrays begin.  All
// accesses are the one shared array plus an index, so they are shared-memory
// instructions with 32-bit addresses.
struct TailLevel {
  int nx, ny, nz, n, o;
  Dims dims;
  __device__ __forceinline__ int gx() const { return o; }
  __device__ __forceinline__ int gy() const { return o + n; }
  __device__ __forceinline__ int gz() const { return o + 2 * n; }
  __device__ __forceinline__ int e() const { return o + 3 * n; }
  __device__ __forceinline__ int dinv() const { return o + 4 * n; }
  __device__ __forceinline__ int b() const { return o + 5 * n; }
  __device__ __forceinline__ int x() const { return o + 6 * n; }
  __device__ __forceinline__ int t() const { return o + 7 * n; }
  __device__ __forceinline__ int s() const { return o + 8 * n; }
};

template <typename T>
__device__ __forceinline__ T tail_apply(const T* S, const TailLevel& f, int x, int c, int i, int j,
                                        int k) {
  const int nx = f.nx, ny = f.ny, nz = f.nz, sz = nx * ny;
  const T* X = S + x;
  const T *gx = S + f.gx(), *gy = S + f.gy(), *gz = S + f.gz();
  const T xc = X[c];
  T y = S[f.e() + c] * xc;
  if (i < nx - 1) y += gx[c] * (xc - X[c + 1]);
  if (i > 0) y += gx[c - 1] * (xc - X[c - 1]);
  if (ny > 1) {
    const int cp = j + 1 < ny ? c + nx : c - j * nx;
    const int cm = j > 0 ? c - nx : c + (ny - 1) * nx;
    y += gy[c] * (xc - X[cp]);
    y += gy[cm] * (xc - X[cm]);
  }
  if (k < nz - 1) y += gz[c] * (xc - X[c + sz]);
  if (k > 0) y += gz[c - sz] * (xc - X[c - sz]);
  return y;
}

// x < 0: from zero
template <typename T>
__device__ __forceinline__ void tail_jacobi(T* S, const TailLevel& f, int x, int xo, T w) {
  for (int c = threadIdx.x; c < f.n; c += MG_TAIL_THREADS) {
    const T b = S[f.b() + c], d = S[f.dinv() + c];
    if (x < 0) {
      S[xo + c] = w * b * d;
      continue;
    }
    int i, j, k;
    split_cell((uint32_t)c, f.dims.fnx, f.dims.fny, i, j, k);
    const T r = b - tail_apply(S, f, x, c, i, j, k);
    S[xo + c] = S[x + c] + w * r * d;
  }
}

template <typename T>
__global__ void __launch_bounds__(MG_TAIL_THREADS, 1)
    k_mg_vcycle_tail(MGTail<T> a, const double* done) {
  PCG_SKIP(done);
  extern __shared__ __align__(16) unsigned char tsh[];
  __shared__ TailLevel L[MG_TAIL_MAX];
  T* const S = (T*)tsh;
  if (threadIdx.x == 0) {
    int o = 0;
    for (int q = 0; q < a.nl; ++q) {
      const MGLevelT<T>& g = a.lev[q];
      L[q] = TailLevel{g.nx, g.ny, g.nz, (int)g.n, o, g.dims};
      o += 9 * (int)g.n;
    }
  }
  __syncthreads();
  // the operators copied in; the vectors are private
  for (int q = 0; q < a.nl; ++q) {
    const MGLevelT<T>& g = a.lev[q];
    const TailLevel f = L[q];
    for (int c = threadIdx.x; c < f.n; c += MG_TAIL_THREADS) {
      S[f.gx() + c] = g.gx[c]; S[f.gy() + c] = g.gy[c]; S[f.gz() + c] = g.gz[c];
      S[f.e() + c] = g.e[c]; S[f.dinv() + c] = g.dinv[c];
      if (q == 0) S[f.b() + c] = g.b[c];
    }
  }
  const int ncs = L[a.nl - 1].n, Ainv = L[a.nl - 1].o + 9 * ncs;
  if (ncs <= MG_COARSE_MAX)
    for (int c = threadIdx.x; c < ncs * ncs; c += MG_TAIL_THREADS) S[Ainv + c] = a.Ainv[c];
  __syncthreads();
  const T w = (T)a.omega;
  const int nu = a.nu;
  // down: pre-smoothing from x = 0 ending in t, residual restricted to the next level's b
  for (int l = 0; l + 1 < a.nl; ++l) {
    const TailLevel f = L[l], cl = L[l + 1];
    int src = -1;
    for (int s = 0; s < nu; ++s) {
      const int dst = ((nu - 1 - s) % 2 == 0) ? f.t() : f.s();
      tail_jacobi(S, f, src, dst, w);
      __syncthreads();
      src = dst;
    }
    for (int t = threadIdx.x; (t & ~31) < 8 * cl.n; t += MG_TAIL_THREADS) {
      const int qu = t >> 3, q = min(qu, cl.n - 1);
      int I, J, K;
      split_cell((uint32_t)q, cl.dims.fnx, cl.dims.fny, I, J, K);
      const int i = 2 * I + (t & 1), j = 2 * J + ((t >> 1) & 1), k = 2 * K + ((t >> 2) & 1);
      T v = T(0);
      if (k < f.nz && j < f.ny && i < f.nx) {
        const int c = (k * f.ny + j) * f.nx + i;
        v = S[f.b() + c] - tail_apply(S, f, f.t(), c, i, j, k);
      }
      const T sum = octet_sum(v);
      if (qu < cl.n && (t & 7) == 0) S[cl.b() + q] = sum;
    }
    __syncthreads();
  }
  // coarsest level: dense solve, or smoothing only when it is too large for it
  {
    const TailLevel f = L[a.nl - 1];
    if (f.n <= MG_COARSE_MAX) {
      for (int r = threadIdx.x; r < f.n; r += MG_TAIL_THREADS) {
        T sum = 0.0;
        for (int q = 0; q < f.n; ++q) sum += S[Ainv + r * f.n + q] * S[f.b() + q];
        S[f.x() + r] = sum;
      }
      __syncthreads();
    } else {
      const T wc = (T)MG_OMEGA;
      tail_jacobi(S, f, -1, f.x(), wc);
      __syncthreads();
      for (int s = 0; s < 8; ++s) {
        tail_jacobi(S, f, (s & 1) ? f.t() : f.x(), (s & 1) ? f.x() : f.t(), wc);
        __syncthreads();
      }
    }
  }
  // up: prolongation into t, post-smoothing from t ending in the level's x
  for (int l = a.nl - 2; l >= 0; --l) {
    const TailLevel f = L[l], cl = L[l + 1];
    for (int c = threadIdx.x; c < f.n; c += MG_TAIL_THREADS) {
      int i, j, k;
      split_cell((uint32_t)c, f.dims.fnx, f.dims.fny, i, j, k);
      S[f.t() + c] += S[cl.x() + ((k >> 1) * cl.ny + (j >> 1)) * cl.nx + (i >> 1)];
    }
    __syncthreads();
    int src = f.t();
    for (int s = 0; s < nu; ++s) {
      const int dst = (s == nu - 1) ? f.x() : ((s % 2 == 0) ? f.s() : f.t());
      tail_jacobi(S, f, src, dst, w);
      __syncthreads();
      src = dst;
    }
  }
  // the first tail level's correction back to global memory
  for (int c = threadIdx.x; c < L[0].n; c += MG_TAIL_THREADS) a.lev[0].x[c] = S[L[0].x() + c];
}

// the sum of the partials that the kernel before left
static void launch_finish(ProjCtx* P, int nb, int slot, int post, const double* done,
                          cudaStream_t st) {
  following(k_finish_sum, 1, FIN_THREADS, 0, st)(P->partial, nb, P->scal, slot, post, done);
}
// a sweep and a restriction on level 0 and on the others (returns the launches)
template <int W, typename T, typename Op, typename V>
static int launch_z_jacobi(ProjCtx* P, const Dims& D, const Op& o, const T* dinv, const T* b, V x,
                           T* xo, double w, bool dot, const double* done, cudaStream_t st) {
  const int nb = z_blocks(D);
  if (!dot) {
    following(k_z_jacobi<W, false, T, Op, V>, nb, Z_THREADS, 0, st)(D, o, dinv, b, x, xo, w, nullptr, nullptr, done);
    return 1;
  }
  following(k_z_jacobi<W, true, T, Op, V>, nb, Z_THREADS, 0, st)(D, o, dinv, b, x, xo, w, P->pc_r, P->partial, done);
  launch_finish(P, nb, 2, POST_NONE, done, st);  // rz_new
  return 2;
}
template <typename T, typename V, typename Op>
static int launch_jacobi(ProjCtx* P, const Dims& D, const Op& o, const T* dinv, const T* b, V x,
                         T* xo, double w, bool dot, const double* done, cudaStream_t st) {
  return z_width(D) == 2 ? launch_z_jacobi<2>(P, D, o, dinv, b, x, xo, w, dot, done, st)
                         : launch_z_jacobi<1>(P, D, o, dinv, b, x, xo, w, dot, done, st);
}
template <typename T, typename V>
static int launch_jacobi(ProjCtx*, const Dims& D, const OpA<T>& o, const T* dinv, const T* b, V x,
                          T* xo, double w, bool, const double* done, cudaStream_t st) {
  following(k_mg_jacobi<T, OpA<T>, V>, blocks_for((int64_t)D.nx * D.ny * D.nz, 256), 256, 0, st)(D, o, dinv, b, x, xo,
                                                                              w, done);
  return 1;
}
template <typename T>
static void launch_restrict(const Dims& D, const OpA<T>& o, const T* b, const T* x, const Dims& DC,
                            T* bc, const double* done, cudaStream_t st) {
  following(k_mg_restrict_residual<T, OpA<T>>, blocks_for(8 * (int64_t)DC.nx * DC.ny * DC.nz, 256), 256,
            0, st)(
      D, o, b, x, DC, bc, done);
}
template <typename T, typename Op>
static void launch_restrict(const Dims& D, const Op& o, const T* b, const T* x, const Dims& DC,
                            T* bc, const double* done, cudaStream_t st) {
  const unsigned nc = blocks_for((int64_t)DC.nx * DC.ny * DC.nz, Z_THREADS);
  if (z_width(D) == 2)
    following(k_z_restrict<T, Op>, nc, Z_THREADS, 0, st)(D, o, b, x, DC, bc, done);
  else
    following(k_mg_restrict_residual<T, Op>, blocks_for(8 * (int64_t)DC.nx * DC.ny * DC.nz, Z_THREADS),
              Z_THREADS, 0, st)(D, o, b, x, DC, bc, done);
}
template <typename Z>
static void launch_matvec_dir(ProjCtx* P, const Z* z, cudaStream_t st) {
  const Dims& D = P->lev[0].dims;
  const int nb = z_blocks(D);
  const OpI<double> o = op_0(P, 0.0);
  if (z_width(D) == 2)
    following(k_z_matvec_dir<2, Z>, nb, Z_THREADS, 0, st)(D, o, z, P->pc_p, P->pc_p2, P->pc_q, P->scal,
                                                   P->partial);
  else
    following(k_z_matvec_dir<1, Z>, nb, Z_THREADS, 0, st)(D, o, z, P->pc_p, P->pc_p2, P->pc_q, P->scal,
                                                   P->partial);
  launch_finish(P, nb, 1, POST_DIR, P->scal + SC_DONE, st);  // p.q
}
// pc_r = rhs - S x and its norm
static void launch_residual(ProjCtx* P, const double* x, float* r32, cudaStream_t st) {
  const Dims& D = P->lev[0].dims;
  const int nb = z_blocks(D);
  const OpI<double> o = op_0(P, 0.0);
  if (z_width(D) == 2)
    following(k_z_residual<2>, nb, Z_THREADS, 0, st)(P->g, D, o, P->rhs, x, P->pc_r, r32, P->partial);
  else
    following(k_z_residual<1>, nb, Z_THREADS, 0, st)(P->g, D, o, P->rhs, x, P->pc_r, r32, P->partial);
  launch_finish(P, nb, 5, POST_NONE, nullptr, st);
}

template <typename T>
static int vcycle(ProjCtx* P, MGLevelT<T>* lev, const T* Ainv, int l, const T* b, T* x,
                  const double* done, cudaStream_t st);

// one level of the V-cycle in launches: the sweeps before (from x = 0, the first
// two in one pass), the coarse correction, and the sweeps after (the
// prolongation part of the first)
template <typename T, typename Op>
static int vcycle_level(ProjCtx* P, MGLevelT<T>* lev, const T* Ainv, int l, Op o, const T* b, T* x,
                        const double* done, cudaStream_t st) {
  MGLevelT<T>& f = lev[l];
  MGLevelT<T>& cl = lev[l + 1];
  const unsigned nb = blocks_for(f.n, 256);
  const int nu = (l == 0 && P->nu0 > 0) ? P->nu0 : P->nu;
  const double om = P->omega;
  int nk = 0;
  // pre-smoothing, ending in t: sweep i writes t when (nu-1-i) is even, else s
  const T* src = nullptr;
  if (nu == 1) {
    following(k_mg_first<T>, nb, 256, 0, st)(f.n, f.dinv, b, f.t, om, done);
    ++nk;
  }
  for (int i = 1; i < nu; ++i) {
    T* dst = ((nu - 1 - i) % 2 == 0) ? f.t : f.s;
    if (i == 1)
      nk += launch_jacobi(P, f.dims, o, f.dinv, b, VecFirst<T>{b, f.dinv, (T)om}, dst, om, false,
                          done, st);
    else
      nk += launch_jacobi(P, f.dims, o, f.dinv, b, VecX<T>{src}, dst, om, false, done, st);
    src = dst;
  }
  launch_restrict(f.dims, o, b, f.t, cl.dims, cl.b, done, st);
  ++nk;
  nk += vcycle<T>(P, lev, Ainv, l + 1, cl.b, cl.x, done, st);
  // post-smoothing from t + P xc, ending in x:  s, t, s, ... then x
  src = f.t;
  for (int i = 0; i < nu; ++i) {
    T* dst = (i == nu - 1) ? x : ((i % 2 == 0) ? f.s : f.t);
    const bool dot = l == 0 && i == nu - 1;  // r.z with the last one
    if (i == 0)
      nk += launch_jacobi(P, f.dims, o, f.dinv, b, VecProl<T>{src, cl.x, cl.nx, cl.ny}, dst, om, dot,
                          done, st);
    else
      nk += launch_jacobi(P, f.dims, o, f.dinv, b, VecX<T>{src}, dst, om, dot, done, st);
    src = dst;
  }
  return nk;
}

template <typename T>
static int vcycle(ProjCtx* P, MGLevelT<T>* lev, const T* Ainv, int l, const T* b, T* x,
                  const double* done, cudaStream_t st) {
  MGLevelT<T>& f = lev[l];
  int nk = 0;
  // the coarse end in one launch (its first level's b and x are the level's own)
  if (l > 0 && P->tail_on && P->nlev - l <= MG_TAIL_MAX && b == f.b && x == f.x &&
      tail_smem_elems(lev + l, P->nlev - l) * (int64_t)sizeof(T) <= MG_TAIL_SMEM) {
    MGTail<T> ta{};
    ta.nl = P->nlev - l;
    for (int q = 0; q < ta.nl; ++q) ta.lev[q] = lev[l + q];
    ta.nu = P->nu;
    ta.omega = P->omega;
    ta.Ainv = Ainv;
    const size_t smem = (size_t)tail_smem_elems(lev + l, ta.nl) * sizeof(T);
    cudaFuncSetAttribute(k_mg_vcycle_tail<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         MG_TAIL_SMEM);
    following(k_mg_vcycle_tail<T>, 1, MG_TAIL_THREADS, smem, st)(ta, done);
    return 1;
  }
  if (l == P->nlev - 1) {
    if (f.n <= MG_COARSE_MAX) {
      following(k_mg_coarse_solve<T>, 1, 64, 0, st)((int)f.n, Ainv, b, x, done);
      ++nk;
    } else {
      // not coarsenable and too large for the dense solve: smoothing only
      const unsigned nb = blocks_for(f.n, 256);
      following(k_mg_first<T>, nb, 256, 0, st)(f.n, f.dinv, b, x, MG_OMEGA, done);
      ++nk;
      for (int s = 0; s < 8; ++s) {
        const T* src = (s & 1) ? f.t : x;
        T* dst = (s & 1) ? x : f.t;
        following(k_mg_jacobi<T, OpA<T>, VecX<T>>, nb, 256, 0, st)(f.dims, op_a(f), f.dinv, b, VecX<T>{src}, dst, MG_OMEGA,
                                           done);
        ++nk;
      }
    }
    return nk;
  }
  return nk + (l == 0 ? vcycle_level<T>(P, lev, Ainv, l, op_0(P, T(0)), b, x, done, st)
                      : vcycle_level<T>(P, lev, Ainv, l, op_a(f), b, x, done, st));
}

void proj_stats(void* h, double* out8) {
  ProjCtx* P = (ProjCtx*)h;
  for (int q = 0; q < 8; ++q) out8[q] = P->stats[q];
}

int proj_configure(void* h, int nu, double omega) {
  ProjCtx* P = (ProjCtx*)h;
  if (nu < 1 || nu > 16 || !(omega > 0.0 && omega < 2.0)) return FS_EARG;
  if (nu != P->nu || omega != P->omega) {
    P->nu = nu;
    P->omega = omega;
    if (P->iter_exec) cudaGraphExecDestroy(P->iter_exec);
    P->iter_exec = nullptr;
    P->graph_failed = 0;
  }
  return FS_OK;
}

int proj_set_fine_sweeps(void* h, int nu0) {
  ProjCtx* P = (ProjCtx*)h;
  if (nu0 < 0 || nu0 > 16) return FS_EARG;
  if (nu0 != P->nu0) {
    P->nu0 = nu0;
    if (P->iter_exec) cudaGraphExecDestroy(P->iter_exec);
    P->iter_exec = nullptr;
    P->graph_failed = 0;
  }
  return FS_OK;
}

int proj_set_coarse_tail(void* h, int on) {
  ProjCtx* P = (ProjCtx*)h;
  if ((on != 0) != (P->tail_on != 0)) {
    P->tail_on = on ? 1 : 0;
    if (P->iter_exec) cudaGraphExecDestroy(P->iter_exec);
    P->iter_exec = nullptr;
    P->graph_failed = 0;
  }
  return FS_OK;
}

// One preconditioned-CG iteration, every kernel a no-op once converged.
static int pcg_iteration(ProjCtx* P, double* x, cudaStream_t st) {
  MGLevel& l0 = P->lev[0];
  const int64_t n = l0.n;
  const double* done = P->scal + SC_DONE;
  int nk;
  if (P->fp32)
    nk = vcycle<float>(P, P->lev32, P->Ainv32, 0, P->r32, P->z32, done, st);
  else
    nk = vcycle<double>(P, P->lev, P->Ainv, 0, P->pc_r, P->pc_z, done, st);
  if (P->nlev == 1) {  // no sweeps: r.z is a pass of its own
    if (P->fp32) {
      following(k_cvt_f2d, blocks_for(n, 256), 256, 0, st)(n, P->z32, P->pc_z, done);
      ++nk;
    }
    following(k_dot, RED_BLOCKS, RED_THREADS, 0, st)(n, P->pc_r, P->pc_z, P->partial, done);
    launch_finish(P, RED_BLOCKS, 2, POST_NONE, done, st);
    nk += 2;
  }
  if (P->fp32)
    launch_matvec_dir(P, P->z32, st);
  else
    launch_matvec_dir(P, P->pc_z, st);
  following(k_pcg_update, RED_BLOCKS, RED_THREADS, 0, st)(P->g, x, P->pc_r, P->fp32 ? P->r32 : nullptr,
                                                   P->pc_p, P->pc_p2, P->pc_q, P->scal, P->partial);
  launch_finish(P, RED_BLOCKS, 5, POST_CHECK, done, st);  // ||r_A||^2
  return nk + 4;
}

// Capture one iteration as a CUDA graph (on the context's private stream).
static void capture_iteration(ProjCtx* P) {
  cudaGraph_t graph = nullptr;
  if (cudaStreamBeginCapture(P->cs, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
    cudaGetLastError();
    P->graph_failed = 1;
    return;
  }
  int nk = pcg_iteration(P, P->p_prev, P->cs);
  if (cudaStreamEndCapture(P->cs, &graph) != cudaSuccess || !graph) {
    cudaGetLastError();
    P->graph_failed = 1;
    return;
  }
  if (cudaGraphInstantiate(&P->iter_exec, graph, 0) != cudaSuccess) {
    cudaGetLastError();
    P->iter_exec = nullptr;
    P->graph_failed = 1;
  }
  cudaGraphDestroy(graph);
  P->iter_kernels = nk;
}

static int launch_iterations(ProjCtx* P, int count, cudaStream_t st) {
  for (int q = 0; q < count; ++q) {
    if (P->iter_exec) {
      if (cudaGraphLaunch(P->iter_exec, st) != cudaSuccess) return FS_ECUDA;
      for (int k = 0; k < P->iter_kernels; ++k) fs_count_launch();
    } else {
      int nk = pcg_iteration(P, P->p_prev, st);
      for (int k = 0; k < nk; ++k) fs_count_launch();
    }
  }
  return FS_OK;
}

using Clock = std::chrono::steady_clock;
static double ms_since(Clock::time_point t0) {
  return std::chrono::duration<double, std::milli>(Clock::now() - t0).count();
}

static int fetch(ProjCtx* P, int n, cudaStream_t st) {
  const auto t0 = Clock::now();
  cudaMemcpyAsync(P->h_scal, P->scal, sizeof(double) * n, cudaMemcpyDeviceToHost, st);
  const int rc = fs_stream_wait(st) != FS_OK ? FS_ECUDA : FS_OK;
  const double w = ms_since(t0);
  P->stats[1] += w;
  if (w > P->stats[2]) P->stats[2] = w;
  P->stats[5] += 1.0;
  return rc;
}

// Pre-smoothing of the learned preconditioner: nu damped-Jacobi sweeps on
// the FP32 level-0 operator from x = 0 for S t = r32, ending in f.t (the
// V-cycle's first half at level 0); then f.b = r32 - S t.
static void lp_presmooth(ProjCtx* P, cudaStream_t st) {
  MGLevelT<float>& f = P->lev32[0];
  const unsigned nb = blocks_for(f.n, 256);
  const float* src = nullptr;
  for (int i = 0; i < P->nu; ++i) {
    float* dst = ((P->nu - 1 - i) % 2 == 0) ? f.t : f.s;
    if (!src)
      following(k_mg_first<float>, nb, 256, 0, st)(f.n, f.dinv, P->r32, dst, P->omega, nullptr);
    else
      following(k_mg_jacobi<float, OpZ<float>, VecX<float>>, nb, 256, 0, st)(f.dims, op_0(P, 0.0f), f.dinv, P->r32,
                                             VecX<float>{src}, dst, P->omega, nullptr);
    src = dst;
    fs_count_launch();
  }
  following(k_lp_residual<float>, nb, 256, 0, st)(f.dims, op_0(P, 0.0f), P->r32, f.t, f.b);
  fs_count_launch();
}

// The learned preconditioner z = M(r), a two-level cycle whose coarse
// correction is the network: pre-smoothing (lp_presmooth), s = t + N(r1)
// (the network's estimate of S^-1 r1, scaled back), then nu post-smoothing
// sweeps from s.  The sweeps remove the high-frequency part of the network's
// error, which the residual norm would otherwise be dominated by.
static int learned_precond(ProjCtx* P, cudaStream_t st) {
  MGLevelT<float>& f = P->lev32[0];
  const int64_t n = f.n;
  const unsigned nb = blocks_for(n, 256);
  following(k_cvt_d2f, nb, 256, 0, st)(n, P->pc_r, P->r32, nullptr);
  fs_count_launch();
  lp_presmooth(P, st);
  int rc = unet_correct(P->net, f.b, f.t, f.s, st);
  if (rc) return rc;
  const float* src = f.s;
  for (int i = 0; i < P->nu; ++i) {
    float* dst = (i == P->nu - 1) ? P->z32 : ((i % 2 == 0) ? f.t : f.x);
    following(k_mg_jacobi<float, OpZ<float>, VecX<float>>, nb, 256, 0, st)(f.dims, op_0(P, 0.0f), f.dinv, P->r32, VecX<float>{src},
                                           dst, P->omega, nullptr);
    src = dst;
    fs_count_launch();
  }
  following(k_cvt_f2d, nb, 256, 0, st)(n, P->z32, P->pc_z, nullptr);
  fs_count_launch();
  return cuda_status();
}

// Training pair for the network from a logged solve (r0, e0 with S e0 = r0):
// the residual after pre-smoothing and the error left, r1 = r0 - S t and
// e1 = e0 - t, in FP32 (the operator of the last rebuild).
int proj_smooth_pair(void* h, const double* r0, const double* e0, float* r1, float* e1,
                     cudaStream_t st) {
  ProjCtx* P = (ProjCtx*)h;
  if (!P->fp32) return FS_EARG;
  MGLevelT<float>& f = P->lev32[0];
  const int64_t n = f.n;
  const unsigned nb = blocks_for(n, 256);
  following(k_cvt_d2f, nb, 256, 0, st)(n, r0, P->r32, nullptr);
  fs_count_launch();
  lp_presmooth(P, st);
  cudaMemcpyAsync(r1, f.b, sizeof(float) * n, cudaMemcpyDeviceToDevice, st);
  following(k_lp_err, nb, 256, 0, st)(n, e0, f.t, e1);
  fs_count_launch();
  return cuda_status();
}

// One flexible-CG iteration with the learned preconditioner (kernels as in
// pcg_iteration; the host reads the scalars after every iteration).
static int fcg_iteration(ProjCtx* P, double* x, int it, cudaStream_t st) {
  MGLevel& l0 = P->lev[0];
  const int64_t n = l0.n;
  const double* done = P->scal + SC_DONE;
  int rc = learned_precond(P, st);
  if (rc) return rc;
  if (it > 0) {
    following(k_dot, RED_BLOCKS, RED_THREADS, 0, st)(n, P->pc_z, P->pc_q, P->partial, done);
    launch_finish(P, RED_BLOCKS, 10, POST_NONE, done, st);  // z.q_prev
    fs_count_launch(); fs_count_launch();
  }
  following(k_fcg_dir, blocks_for(n, 256), 256, 0, st)(n, P->scal, P->pc_z, P->pc_p);
  const int nb = z_blocks(l0.dims);
  if (z_width(l0.dims) == 2)
    following(k_z_matvec<2>, nb, Z_THREADS, 0, st)(l0.dims, op_0(P, 0.0), P->pc_p, P->pc_q, P->partial, done);
  else
    following(k_z_matvec<1>, nb, Z_THREADS, 0, st)(l0.dims, op_0(P, 0.0), P->pc_p, P->pc_q, P->partial, done);
  launch_finish(P, nb, 1, POST_NONE, done, st);  // p.q
  following(k_dot, RED_BLOCKS, RED_THREADS, 0, st)(n, P->pc_p, P->pc_r, P->partial, done);
  launch_finish(P, RED_BLOCKS, 12, POST_NONE, done, st);  // p.r
  following(k_fcg_alpha, 1, 1, 0, st)(P->scal);  // alpha = p.r / p.q
  following(k_set_scal, 1, 1, 0, st)(P->scal, 11, 1);
  following(k_pcg_update, RED_BLOCKS, RED_THREADS, 0, st)(P->g, x, P->pc_r, nullptr, P->pc_p, nullptr,
                                                   P->pc_q, P->scal, P->partial);
  launch_finish(P, RED_BLOCKS, 5, POST_CHECK, done, st);
  for (int k = 0; k < 9; ++k) fs_count_launch();
  return cuda_status();
}

// Learned iterations until convergence, a stall or max_learned; on a stall
// the residual is recomputed and the scalars reset so that the V-cycle PCG
// loop continues from the current iterate.
static int fcg_solve(ProjCtx* P, double* x, int maxiter, int* learned, cudaStream_t st) {
  const GridDev& g = P->g;
  MGLevel& l0 = P->lev[0];
  std::vector<double> rn;
  int it = 0;
  while (true) {
    int stt = fetch(P, 9, st);
    if (stt) return stt;
    const double bn2 = P->h_scal[4], rn2 = P->h_scal[5];
    if (!(bn2 == bn2) || !(rn2 == rn2)) return FS_ENONFINITE;
    if (P->h_scal[SC_DONE] != 0.0) break;
    rn.push_back(rn2);
    bool fall = it >= P->max_learned || it >= maxiter;
    if (!fall && it >= 3) {
      const double f = std::pow(rn2 / rn[it - 3], 1.0 / 6.0);  // per-iteration norm factor
      fall = !(f < P->stall);
    }
    if (fall) {
      launch_residual(P, x, P->r32, st);
      following(k_fcg_restart, 1, 1, 0, st)(P->scal);
      fs_count_launch(); fs_count_launch(); fs_count_launch();
      P->fcg[2] = 1.0;
      P->fcg[3] += 1.0;
      break;
    }
    stt = fcg_iteration(P, x, it, st);
    if (stt) return stt;
    ++it;
  }
  *learned = it;
  P->fcg[0] = it;
  return cuda_status();
}

int proj_set_learned(void* h, void* net, int max_learned, double stall) {
  ProjCtx* P = (ProjCtx*)h;
  if (max_learned < 0 || !(stall > 0.0 && stall <= 1.0)) return FS_EARG;
  // the learned cycle runs on the FP32 level-0 operator of the mixed form
  if (net && (!P->fp32 || unet_cells(net) != P->lev[0].n)) return FS_EARG;
  P->net = net;
  P->max_learned = max_learned;
  P->stall = stall;
  return FS_OK;
}

int proj_set_log(void* h, double* r0, double* x0) {
  ProjCtx* P = (ProjCtx*)h;
  if ((r0 == nullptr) != (x0 == nullptr)) return FS_EARG;
  P->log_r0 = r0;
  P->log_x0 = x0;
  return FS_OK;
}

void proj_fcg_stats(void* h, double* out4) {
  ProjCtx* P = (ProjCtx*)h;
  for (int q = 0; q < 4; ++q) out4[q] = P->fcg[q];
}

// Solve for the pressure and correct u, v, w in place.  The iterations run
// as graph launches in batches (sized from the previous solve's count); the
// host reads the converged flag once per batch.
int proj_project(void* h, double* u, double* v, double* w, const double* u_in,
                 const double* target, double dt, double rtol, int maxiter, int* iters,
                 cudaStream_t st) {
  ProjCtx* P = (ProjCtx*)h;
  const GridDev& g = P->g;
  MGLevel& l0 = P->lev[0];
  const int64_t n = l0.n;
  const auto t_start = Clock::now();
  for (int q = 0; q < 8; ++q) P->stats[q] = 0.0;
  *iters = 0;
  following(k_proj_rhs, RED_BLOCKS, RED_THREADS, 0, st)(g, u, v, w, u_in, target, 1.0 / g.dx, 1.0 / g.dy,
                                                 1.0 / dt, P->rhs, P->partial);
  launch_finish(P, RED_BLOCKS, 4, POST_NONE, nullptr, st);
  fs_count_launch(); fs_count_launch();
  double* x = P->p_prev;
  launch_residual(P, x, P->fp32 ? P->r32 : nullptr, st);
  fs_count_launch(); fs_count_launch();
  following(k_pcg_init, 1, 1, 0, st)(P->scal, rtol * rtol); fs_count_launch();
  following(k_zero_if_zero_rhs, 296, 256, 0, st)(n, P->scal, x); fs_count_launch();
  if (P->log_r0) {
    cudaMemcpyAsync(P->log_r0, P->pc_r, sizeof(double) * n, cudaMemcpyDeviceToDevice, st);
    cudaMemcpyAsync(P->log_x0, x, sizeof(double) * n, cudaMemcpyDeviceToDevice, st);
  }
  int learned = 0;
  P->fcg[0] = P->fcg[1] = P->fcg[2] = 0.0;
  if (P->net) {
    int stt = fcg_solve(P, x, maxiter, &learned, st);
    if (stt) return stt;
  }
  if (!P->iter_exec && !P->graph_failed) capture_iteration(P);
  int launched = learned;
  int batch = P->last_iters > 2 ? P->last_iters - 2 : 1;
  while (true) {
    int stt = fetch(P, 9, st);
    if (stt) return stt;
    const double bn2 = P->h_scal[4], rn2 = P->h_scal[5];
    if (!(bn2 == bn2) || !(rn2 == rn2)) return FS_ENONFINITE;
    if (P->h_scal[SC_DONE] != 0.0) break;
    if (launched >= maxiter) return FS_ENOCONV;
    if (batch > maxiter - launched) batch = maxiter - launched;
    const auto tl = Clock::now();
    stt = launch_iterations(P, batch, st);
    const double lw = ms_since(tl);
    P->stats[3] += lw;
    if (lw > P->stats[4]) P->stats[4] = lw;
    if (stt) return stt;
    launched += batch;
    P->stats[6] += batch;
    batch = 2;
  }
  if (P->net && P->fcg[2] != 0.0) P->fcg[1] = P->h_scal[SC_IT];
  *iters = P->fcg[2] != 0.0 ? learned + (int)P->h_scal[SC_IT] : (int)P->h_scal[SC_IT];
  P->last_iters = *iters;
  P->stats[7] = *iters;
  P->stats[0] = ms_since(t_start);
  P->have_prev = 1;
  Launch3 L = launch_cells(g);
  following(k_proj_correct, L.grid, L.block, 0, st)(g, u, v, w, x, P->ir, dt, dt / g.dx, dt / g.dy);
  fs_count_launch();
  return cuda_status();
}

int launch_div_resid_max(const GridDev& g, const double* u, const double* v, const double* w,
                         const double* u_in, const double* target, double* div_out,
                         unsigned long long* out_key, cudaStream_t st) {
  cudaMemsetAsync(out_key, 0, sizeof(unsigned long long), st);
  int64_t n = ncells(g);
  unsigned nb = blocks_for(n, 256);
  if (nb > 1184) nb = 1184;
  following(div_out ? k_div_resid_max<true> : k_div_resid_max<false>, nb, 256, 0, st)(
      g, u, v, w, u_in, target, 1.0 / g.dx, 1.0 / g.dy, div_out, out_key);
  fs_count_launch();
  return cuda_status();
}

// apply the symmetrised operator to x (test hook): y = S x  and A x = -y / dz
int proj_apply(void* h, const double* x, double* y, cudaStream_t st) {
  ProjCtx* P = (ProjCtx*)h;
  MGLevel& l0 = P->lev[0];
  following(k_z_matvec<1>, blocks_for(l0.n, Z_THREADS), Z_THREADS, 0, st)(l0.dims, op_0(P, 0.0), x, y,
                                                                  nullptr, nullptr);
  fs_count_launch();
  return cuda_status();
}
