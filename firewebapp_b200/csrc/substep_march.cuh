// The sub-step's marching stencils in either precision: species transport
// (march.cuh has the scheme) and turbulent diffusion.
#pragma once
#include "march.cuh"

// ---------------------------------------------------------------------------
// Species transport, up to 3 species in one pass
// (species_3d.py:41-175 step_species_transport, called x3 at spread_3d.py:3015-3038)
// ---------------------------------------------------------------------------
template <typename T>
struct SpeciesArgs {
  const T* Y[3];
  T* Yo[3];
  const T* S[3];
  T Y_inlet[3];
  // fused form (fuel, O2, H2O in that order): the sources from S_pyro and
  // S_drying as k_species_sources forms them, and O2 clipped to [0, o2_cap]
  // after the update as k_clip does
  const T *Sp, *Sd;
  const T *rho, *u, *v, *w;
  T dt, D, inv_dx, inv_dy, inv_dx2, inv_dy2, o2_cap;
};

// Bound by instructions issued.  With the limiters face by face the three
// species took 940 a warp and level in FP64: 143 us at 400 x 120 x 60, 108 as
// cell differences; FP32 at 301 x 119 x 47, where every neighbour was loaded from
// L1, 65 us and now 45.  The expressions keep their order and roundings: cells sit on
// the EDC's thresholds.
template <typename T, int NS, bool FUSED, bool DIRECT>
__global__ void __launch_bounds__(MR_THREADS, sizeof(T) == 8 ? 3 : 4)
    k_species(GridDev g, SpeciesArgs<T> a, int kz) {
  FOLLOW();
  typedef PlaneRing<T, NS, 2, 6> Ring;
  extern __shared__ __align__(16) unsigned char mr_raw[];
  T* const ring = (T*)mr_raw;
  T* const rks = (T*)(mr_raw + (DIRECT ? 0 : Ring::BYTES));
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const int64_t sz = (int64_t)nx * ny;
  const int k0 = blockIdx.z * kz, k1 = min(nz, k0 + kz);
  const T* f[NS];
#pragma unroll
  for (int s = 0; s < NS; ++s) f[s] = a.Y[s];
  Ring R;
  if constexpr (!DIRECT) {
    R.init(ring, g);
    for (int q = 0; q < 5; ++q) R.load(g, f, k0 - 2 + q, q);
    copy_commit();
  }
  march_spacings(g, k0, k1, rks);
  const int i = blockIdx.x * MR_TX + threadIdx.x, j = blockIdx.y * MR_TY + threadIdx.y;
  const bool inside = i < nx && j < ny;
  const int64_t col = (int64_t)min(j, ny - 1) * nx + min(i, nx - 1);
  T n_u, n_v, n_w, n_r, n_p = T(0), n_d = T(0);
  auto centre = [&](int64_t c) {
    n_u = a.u[c]; n_v = a.v[c]; n_w = a.w[c]; n_r = a.rho[c];
    if (FUSED) { n_p = a.Sp[c]; n_d = a.Sd[c]; }
  };
  centre(k0 * sz + col);
  const bool mx = i >= 2 && i <= nx - 3;
  Near<DIRECT, Ring::HX> N;
  N.init(g, i, min(j, ny - 1));
  int sl = 2;  // the slot of plane k
  for (int k = k0; k < k1; ++k, sl = Ring::slot(sl, 1)) {
    if constexpr (!DIRECT) copy_wait<0>();
    __syncthreads();
    if constexpr (!DIRECT) {
      if (k + 3 <= k1 + 1) R.load(g, f, k + 3, Ring::slot(sl, 3));
      copy_commit();
    }
    const T ui = n_u, vi = n_v, wi = n_w, rho_c = n_r, sp = n_p, sd = n_d;
    const int64_t c = k * sz + col;
    if (k + 1 < k1) centre(c + sz);
    if (!inside) continue;
    const T* const p0 = Ring::at(ring, sl);
    const T* const pl = Ring::at(ring, Ring::slot(sl, -1));
    const T* const ph = Ring::at(ring, Ring::slot(sl, 1));
    const bool ux = ui >= T(0), uy = vi >= T(0), uz = wi >= T(0);
    const T* const pf = Ring::at(ring, Ring::slot(sl, uz ? -2 : 2));
    const int ox = ux ? -2 : 2, oy = uy ? N.yl2 : N.yr2;
    const T* rk = rks + (k - k0) * MR_RK;
    const T ida = rk[0], idb = rk[1], idz = rk[2], ihz = rk[3];
    const bool mz = k >= 2 && k <= nz - 3;
    const T inv_rho = T(1) / rho_c;
    const T stot = sp + sd;
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      const T* const P = DIRECT ? f[s] + c : p0 + s * Ring::PLANE;
      const T C = P[0];
      const T xL = i == 0 ? a.Y_inlet[s] : P[N.xl], xR = i == nx - 1 ? C : P[N.xr];
      const T yL = P[N.yl], yR = P[N.yr];
      const T zL = k == 0 ? C : *(DIRECT ? P - sz : pl + s * Ring::PLANE);
      const T zR = k == nz - 1 ? C : *(DIRECT ? P + sz : ph + s * Ring::PLANE);
      T fx, fz;
      if (mx) fx = fabs(ui) * muscl_diff(xR - C, C - xL, C, ux ? xL : xR, P[ox], ux) * a.inv_dx;
      else fx = ux ? ui * (C - xL) * a.inv_dx : ui * (xR - C) * a.inv_dx;
      const T fy = fabs(vi) * muscl_diff(yR - C, C - yL, C, uy ? yL : yR, P[oy], uy) * a.inv_dy;
      if (mz)
        fz = fabs(wi) * muscl_diff(zR - C, C - zL, C, uz ? zL : zR,
                                  *(DIRECT ? P + (uz ? -2 * sz : 2 * sz) : pf + s * Ring::PLANE), uz) *
             ihz;
      else
        fz = uz ? wi * (C - zL) * idb : wi * (zR - C) * ida;
      const T adv = -(fx + fy + fz);
      const T d2x = (xR - T(2) * C + xL) * a.inv_dx2;
      const T d2y = (yR - T(2) * C + yL) * a.inv_dy2;
      const T d2z = ((zR - C) * ida - (C - zL) * idb) * idz;
      const T diff = a.D * (d2x + d2y + d2z);
      T S;
      if (FUSED) S = (s == 0) ? sp - C * stot : ((s == 1) ? -(C * stot) : sd - C * stot);
      else S = a.S[s][c];
      const T src = S * inv_rho;
      T nw = C + (adv + diff + src) * a.dt;
      if (nw < T(0)) nw = T(0);
      else if (nw > T(1)) nw = T(1);
      if (FUSED && s == 1) {
        if (nw > a.o2_cap) nw = a.o2_cap;
        if (nw < T(0)) nw = T(0);
      }
      a.Yo[s][c] = nw;
    }
  }
}

template <typename T, int NS, bool FUSED>
static int launch_species_march(const GridDev& g, const SpeciesArgs<T>& a, cudaStream_t st) {
  constexpr int spacings = MR_MAXK * MR_RK * (int)sizeof(T);
  constexpr int smem = PlaneRing<T, NS, 2, 6>::BYTES + spacings;
  if (march_direct<T>(g)) {
    following(k_species<T, NS, FUSED, true>, march_grid(g, 1), dim3(MR_TX, MR_TY), spacings, st)(g, a, 1);
    fs_count_launch();
    return cuda_status();
  }
  const int kz = march_levels(g);
  if (!march_smem((const void*)k_species<T, NS, FUSED, false>, smem)) return cuda_status();
  following(k_species<T, NS, FUSED, false>, march_grid(g, kz), dim3(MR_TX, MR_TY), smem, st)(g, a, kz);
  fs_count_launch();
  return cuda_status();
}

// ---------------------------------------------------------------------------
// Turbulent diffusion sub-iteration for up to 4 fields sharing nu_t and sc_t
// (turbulence_3d.py:862-949 apply_turbulent_diffusion, inner prange pair)
// Optional clip [lo, hi] after the LAST sub-iteration is applied by the caller.
// ---------------------------------------------------------------------------
template <typename T>
struct DiffArgs {
  const T* f[4];
  T* fo[4];
  T lo[4], hi[4];
  const T* nu_t;
  T sc_t, inv_sc, dt, inv_dx2, inv_dy2;
  int clip;
};

// A thread marches up its column with the levels below and above in registers, one
// more level requested, and takes the neighbours in x and y from L1.  A level reads
// one plane's halo only, so the ring of planes that the other stencils use did not
// pay for its copies: three FP64 fields at 400 x 120 x 60 43 us with the ring, 40 so
// (FP32 31 and 24), one field 21 and 17 (17 and 11); at 133 x 45 x 37 10.2 and 5.8
// (9.0 and 4.4), 5.4 and 3.7 (4.8 and 3.6).  (Three FP64 fields spill 72 bytes at
// four blocks an SM; at three they took 44 and 6.2.)
template <typename T, int NF>
__global__ void __launch_bounds__(MR_THREADS, sizeof(T) == 4 || NF < 4 ? 4 : 2)
    k_turb_diff(GridDev g, DiffArgs<T> a, int kz) {
  FOLLOW();
  __shared__ T rks[MR_MAXK * MR_RK];
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const int64_t sz = (int64_t)nx * ny;
  const int k0 = blockIdx.z * kz, k1 = min(nz, k0 + kz);
  march_spacings(g, k0, k1, rks);
  __syncthreads();
  const int i = blockIdx.x * MR_TX + threadIdx.x, j = blockIdx.y * MR_TY + threadIdx.y;
  if (i >= nx || j >= ny) return;
  int64_t c = k0 * sz + (int64_t)j * nx + i;
  // zero gradient at the inlet, the outlet, the ground and the top
  const int oL = i == 0 ? 0 : -1, oR = i == nx - 1 ? 0 : 1;
  const int oB = (j > 0 ? -1 : ny - 1) * nx, oF = (j < ny - 1 ? 1 : 1 - ny) * nx;
  T zL[NF], C[NF], zR[NF];
#pragma unroll
  for (int s = 0; s < NF; ++s) {
    C[s] = a.f[s][c];
    zL[s] = k0 == 0 ? C[s] : a.f[s][c - sz];
    zR[s] = k0 == nz - 1 ? C[s] : a.f[s][c + sz];
  }
  T nu = a.nu_t[c];
  for (int k = k0; k < k1; ++k, c += sz) {
    const bool more = k + 1 < k1;
    const T nu_n = more ? a.nu_t[c + sz] : T(0);
    T far[NF], xL[NF], xR[NF], yL[NF], yR[NF];
#pragma unroll
    for (int s = 0; s < NF; ++s) {
      const T* const f = a.f[s] + c;
      far[s] = more && k + 2 < nz ? f[2 * sz] : zR[s];
      xL[s] = f[oL];
      xR[s] = f[oR];
      yL[s] = f[oB];
      yR[s] = f[oF];
    }
    // (each precision as it has always rounded: a cell on an extinction threshold
    // must not change sides)
    const T D_t = sizeof(T) == 8 ? nu / a.sc_t : nu * a.inv_sc;
    nu = nu_n;
    const T* rk = rks + (k - k0) * MR_RK;
    const T ida = rk[0], idb = rk[1], idz = rk[2];
#pragma unroll
    for (int s = 0; s < NF; ++s) {
      const T c0 = C[s];
      const T d2x = (xR[s] - T(2) * c0 + xL[s]) * a.inv_dx2;
      const T d2y = (yR[s] - T(2) * c0 + yL[s]) * a.inv_dy2;
      const T d2z = ((zR[s] - c0) * ida - (c0 - zL[s]) * idb) * idz;
      T nv = c0 + D_t * (d2x + d2y + d2z) * a.dt;
      if (a.clip) {
        if (nv < a.lo[s]) nv = a.lo[s];
        if (nv > a.hi[s]) nv = a.hi[s];
      }
      a.fo[s][c] = nv;
      zL[s] = c0;
      C[s] = zR[s];
      zR[s] = far[s];
    }
  }
}

template <typename T, int NF>
static int launch_turb_march(const GridDev& g, const DiffArgs<T>& a, cudaStream_t st) {
  const int kz = march_levels(g);
  following(k_turb_diff<T, NF>, march_grid(g, kz), dim3(MR_TX, MR_TY), 0, st)(g, a, kz);
  fs_count_launch();
  return cuda_status();
}
