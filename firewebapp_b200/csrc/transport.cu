// Explicit transport stencils of the Tier-3 step (FP64).
//
// Each kernel restates one reference operator; the comment above it names
// the reference function and lines.  All kernels are out-of-place (read the
// old field, write a new one), which is what the reference's double buffers
// (dY, du/dv/dw, k_turb_new, T_s_new) amount to.
#include "common.cuh"
#include "kernels.h"
#include "substep_march.cuh"

#define MR_RK_BYTES (MR_MAXK * MR_RK * (int)sizeof(double))

// ---------------------------------------------------------------------------
// Species transport (the kernel: substep_march.cuh)
// ---------------------------------------------------------------------------
static SpeciesArgs<double> species_args(const GridDev& g, int nspec, const double* const* Y,
                                        double* const* Yo, const double* Y_inlet,
                                        const double* rho, const double* u, const double* v,
                                        const double* w, double dt, double D) {
  SpeciesArgs<double> a{};
  for (int s = 0; s < nspec; ++s) {
    a.Y[s] = Y[s]; a.Yo[s] = Yo[s]; a.Y_inlet[s] = Y_inlet[s];
  }
  a.rho = rho; a.u = u; a.v = v; a.w = w;
  a.dt = dt; a.D = D;
  a.inv_dx = 1.0 / g.dx; a.inv_dy = 1.0 / g.dy;
  a.inv_dx2 = a.inv_dx * a.inv_dx; a.inv_dy2 = a.inv_dy * a.inv_dy;
  return a;
}

int launch_species(const GridDev& g, int nspec, const double* const* Y, double* const* Yo,
                   const double* const* S, const double* Y_inlet, const double* rho,
                   const double* u, const double* v, const double* w, double dt, double D,
                   cudaStream_t st) {
  if (nspec < 1 || nspec > 3) return FS_EARG;
  SpeciesArgs<double> a = species_args(g, nspec, Y, Yo, Y_inlet, rho, u, v, w, dt, D);
  for (int s = 0; s < nspec; ++s) a.S[s] = S[s];
  switch (nspec) {
    case 1: return launch_species_march<double, 1, false>(g, a, st);
    case 2: return launch_species_march<double, 2, false>(g, a, st);
    default: return launch_species_march<double, 3, false>(g, a, st);
  }
}

// The sub-step's species work in one pass: the sources with dilution
// (k_species_sources), the transport of fuel, O2 and H2O, and the O2 clip
// that follows it (spread_3d.py:2996-3004, 3015-3038, 3059); the results equal
// those three launches'.
int launch_species_step(const GridDev& g, const double* const* Y, double* const* Yo,
                        const double* Sp, const double* Sd, const double* Y_inlet,
                        const double* rho, const double* u, const double* v, const double* w,
                        double dt, double D, double o2_cap, cudaStream_t st) {
  SpeciesArgs<double> a = species_args(g, 3, Y, Yo, Y_inlet, rho, u, v, w, dt, D);
  a.Sp = Sp;
  a.Sd = Sd;
  a.o2_cap = o2_cap;
  return launch_species_march<double, 3, true>(g, a, st);
}

// The stencils wait on their own copies only: nothing to expire.  What callers
// have of it is what a blocking copy from the legacy stream gave: that stream's
// work has run, or an error of it is reported (one that an earlier call of the
// thread left is not).
int stencil_status(int) {
  return cudaStreamSynchronize(cudaStreamLegacy) == cudaSuccess ? 0 : -1;
}
void set_tma(int) {}

// ---------------------------------------------------------------------------
// Species source terms with dilution (spread_3d.py:2996-3004, Lagrangian branch)
//   S_F = Sp - Y_F (Sp + Sd); S_O2 = -Y_O2 (Sp + Sd); S_H2O = Sd - Y_H2O (Sp + Sd)
// ---------------------------------------------------------------------------
__global__ void k_species_sources(int64_t n, const double* __restrict__ Sp,
                                  const double* __restrict__ Sd, const double* __restrict__ YF,
                                  const double* __restrict__ YO, const double* __restrict__ YH,
                                  double* SF, double* SO, double* SH) {
  int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (c >= n) return;
  double sp = Sp[c], sd = Sd[c];
  double st = sp + sd;
  SF[c] = sp - YF[c] * st;
  SO[c] = -(YO[c] * st);
  SH[c] = sd - YH[c] * st;
}

int launch_species_sources(int64_t n, const double* Sp, const double* Sd, const double* YF,
                           const double* YO, const double* YH, double* SF, double* SO,
                           double* SH, cudaStream_t st) {
  k_species_sources<<<blocks_for(n, 256), 256, 0, st>>>(n, Sp, Sd, YF, YO, YH, SF, SO, SH); fs_count_launch();
  return cuda_status();
}

// ---------------------------------------------------------------------------
// Scalar MUSCL advection accumulator (muscl_3d.py:67-171):  rhs -= u . grad(phi)
// ---------------------------------------------------------------------------
__device__ __forceinline__ double advect_flux_sum(const GridDev& g, const double* __restrict__ phi,
                                                  int k, int j, int i, int64_t c, double uc,
                                                  double vc, double wc, double phi_inlet) {
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const int64_t sy = nx, sz = (int64_t)nx * ny;
  const double pc = phi[c];
  const double xL = (i == 0) ? phi_inlet : phi[c - 1];
  const double xR = (i == nx - 1) ? pc : phi[c + 1];
  const double zL = (k == 0) ? pc : phi[c - sz];
  const double zR = (k == nz - 1) ? pc : phi[c + sz];
  double fx, fz;
  if (i >= 2 && i <= nx - 3) {
    double fp = muscl_face(phi[c - 1], pc, phi[c + 1], phi[c + 2], uc);
    double fm = muscl_face(phi[c - 2], phi[c - 1], pc, phi[c + 1], uc);
    fx = uc * (fp - fm) / g.dx;
  } else {
    fx = (uc >= 0.0) ? uc * (pc - xL) / g.dx : uc * (xR - pc) / g.dx;
  }
  const int64_t crow = c - (int64_t)j * sy;
  const int jm2 = wrapj(j - 2, ny), jm1 = wrapj(j - 1, ny);
  const int jp1 = wrapj(j + 1, ny), jp2 = wrapj(j + 2, ny);
  double fyp = muscl_face(phi[crow + jm1 * sy], pc, phi[crow + jp1 * sy], phi[crow + jp2 * sy], vc);
  double fym = muscl_face(phi[crow + jm2 * sy], phi[crow + jm1 * sy], pc, phi[crow + jp1 * sy], vc);
  double fy = vc * (fyp - fym) / g.dy;
  if (k >= 2 && k <= nz - 3) {
    double fp = muscl_face(phi[c - sz], pc, phi[c + sz], phi[c + 2 * sz], wc);
    double fm = muscl_face(phi[c - 2 * sz], phi[c - sz], pc, phi[c + sz], wc);
    fz = wc * (fp - fm) / (0.5 * (g.da[k] + g.db[k]));
  } else {
    double inv_db = 1.0 / g.db[k], inv_da = 1.0 / g.da[k];
    fz = (wc >= 0.0) ? wc * (pc - zL) * inv_db : wc * (zR - pc) * inv_da;
  }
  return fx + fy + fz;
}

__global__ void k_advect_scalar(GridDev g, const double* __restrict__ phi,
                                const double* __restrict__ u, const double* __restrict__ v,
                                const double* __restrict__ w, double* rhs, double phi_inlet) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  int j = blockIdx.y * blockDim.y + threadIdx.y;
  int k = blockIdx.z;
  if (i >= g.nx || j >= g.ny) return;
  int64_t c = cidx(g, k, j, i);
  rhs[c] -= advect_flux_sum(g, phi, k, j, i, c, u[c], v[c], w[c], phi_inlet);
}

int launch_advect_scalar(const GridDev& g, const double* phi, const double* u, const double* v,
                         const double* w, double* rhs, double phi_inlet, cudaStream_t st) {
  Launch3 L = launch_cells(g);
  k_advect_scalar<<<L.grid, L.block, 0, st>>>(g, phi, u, v, w, rhs, phi_inlet); fs_count_launch();
  return cuda_status();
}

// ---------------------------------------------------------------------------
// Gas-temperature advection + molecular diffusion (spread_3d.py:3827-3897 _adv_gas_energy)
// ---------------------------------------------------------------------------
// (a ring of T's planes; a thread a cell took 104 us at 400 x 120 x 60, 800
// instructions a warp, a third of them divisions by spacings; 38 now)
typedef PlaneRing<double, 1, 2, 6> GasRing;
__global__ void __launch_bounds__(MR_THREADS, 4)
    k_gas_energy_adv(GridDev g, const double* T, const double* u,
                     const double* v, const double* w,
                     double* To, double dt, double alpha, double T_amb, double inv_dx,
                     double inv_dy, int kz) {
  FOLLOW();
  extern __shared__ __align__(16) unsigned char mr_raw[];
  double* const ring = (double*)mr_raw;
  double* const rks = (double*)(mr_raw + GasRing::BYTES);
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const int64_t sz = (int64_t)nx * ny;
  const int k0 = blockIdx.z * kz, k1 = min(nz, k0 + kz);
  const double* const f[1] = {T};
  GasRing R;
  R.init(ring, g);
  for (int q = 0; q < 5; ++q) R.load(g, f, k0 - 2 + q, q);
  copy_commit();
  march_spacings(g, k0, k1, rks);
  const int i = blockIdx.x * MR_TX + threadIdx.x, j = blockIdx.y * MR_TY + threadIdx.y;
  const bool inside = i < nx && j < ny;
  const int64_t col = (int64_t)min(j, ny - 1) * nx + min(i, nx - 1);
  double n_u = u[k0 * sz + col], n_v = v[k0 * sz + col], n_w = w[k0 * sz + col];
  const bool mx = i >= 2 && i <= nx - 3;
  const double ax = alpha * (inv_dx * inv_dx), ay = alpha * (inv_dy * inv_dy);
  int s = 2;
  for (int k = k0; k < k1; ++k, s = GasRing::slot(s, 1)) {
    copy_wait<0>();
    __syncthreads();
    if (k + 3 <= k1 + 1) R.load(g, f, k + 3, GasRing::slot(s, 3));
    copy_commit();
    const double uc = n_u, vc = n_v, wc = n_w;
    const int64_t c = k * sz + col;
    if (k + 1 < k1) { n_u = u[c + sz]; n_v = v[c + sz]; n_w = w[c + sz]; }
    if (!inside) continue;
    const bool ux = uc >= 0.0, uy = vc >= 0.0, uz = wc >= 0.0;
    const double* const P = GasRing::at(ring, s);
    const double* rk = rks + (k - k0) * MR_RK;
    const double ida = rk[0], idb = rk[1];
    const double C = P[0];
    // inlet ghost T_amb, zero gradient at the outlet, the ground and the top
    double L = i == 0 ? T_amb : P[-1], H = i == nx - 1 ? C : P[1];
    double dp = H - C, dm = C - L, n = ux ? L : H;
    double adv = fabs(uc) * (mx ? muscl_diff(dp, dm, C, n, P[ux ? -2 : 2], ux) : C - n) * inv_dx;
    double dif = ax * (dp - dm);
    L = P[-GasRing::HX];
    H = P[GasRing::HX];
    dp = H - C;
    dm = C - L;
    adv += fabs(vc) * muscl_diff(dp, dm, C, uy ? L : H, P[uy ? -2 * GasRing::HX : 2 * GasRing::HX], uy) *
           inv_dy;
    dif += ay * (dp - dm);
    L = k == 0 ? C : GasRing::at(ring, GasRing::slot(s, -1))[0];
    H = k == nz - 1 ? C : GasRing::at(ring, GasRing::slot(s, 1))[0];
    dp = H - C;
    dm = C - L;
    n = uz ? L : H;
    adv += fabs(wc) *
           (k >= 2 && k <= nz - 3
                ? muscl_diff(dp, dm, C, n, GasRing::at(ring, GasRing::slot(s, uz ? -2 : 2))[0], uz) *
                      rk[3]
                : (C - n) * (uz ? idb : ida));
    dif += alpha * ((dp * ida - dm * idb) * rk[2]);
    double Tn = C + (dif - adv) * dt;
    if (Tn < T_amb) Tn = T_amb;
    if (Tn > 10000.0) Tn = 10000.0;
    To[c] = Tn;
  }
}

int launch_gas_energy_adv(const GridDev& g, const double* T, const double* u, const double* v,
                          const double* w, double* To, double dt, double alpha, double T_amb,
                          cudaStream_t st) {
  if (g.nx < 3 || g.nz < 3) return FS_EARG;
  const int kz = march_levels(g);
  if (!march_smem((const void*)k_gas_energy_adv, GasRing::BYTES + MR_RK_BYTES)) return cuda_status();
  following(k_gas_energy_adv, march_grid(g, kz), dim3(MR_TX, MR_TY), GasRing::BYTES + MR_RK_BYTES,
            st)(
      g, T, u, v, w, To, dt, alpha, T_amb, 1.0 / g.dx, 1.0 / g.dy, kz);
  fs_count_launch();
  return cuda_status();
}

// ---------------------------------------------------------------------------
// Turbulent diffusion (the kernel: substep_march.cuh)
// ---------------------------------------------------------------------------
int launch_turb_diff(const GridDev& g, int nfield, const double* const* f, double* const* fo,
                     const double* nu_t, double sc_t, double dt_sub, int clip, const double* lo,
                     const double* hi, cudaStream_t st) {
  if (nfield < 1 || nfield > 4) return FS_EARG;
  DiffArgs<double> a{};
  a.nu_t = nu_t;
  a.sc_t = sc_t;
  a.dt = dt_sub;
  a.inv_dx2 = 1.0 / (g.dx * g.dx); a.inv_dy2 = 1.0 / (g.dy * g.dy);
  a.clip = clip;
  for (int s = 0; s < nfield; ++s) {
    a.f[s] = f[s]; a.fo[s] = fo[s];
    a.lo[s] = clip ? lo[s] : 0.0;
    a.hi[s] = clip ? hi[s] : 0.0;
  }
  switch (nfield) {
    case 1: return launch_turb_march<double, 1>(g, a, st);
    case 2: return launch_turb_march<double, 2>(g, a, st);
    case 3: return launch_turb_march<double, 3>(g, a, st);
    default: return launch_turb_march<double, 4>(g, a, st);
  }
}

// ---------------------------------------------------------------------------
// Porous drag (drag_3d.py:100-144 step_drag_force)
// ---------------------------------------------------------------------------
__device__ __forceinline__ double drag_coeff(double ui, double vi, double wi, double rho,
                                             double a, double sigma, double sigma2, double C_D) {
  double speed = sqrt(ui * ui + vi * vi + wi * wi);
  double om = 1.0 - a;
  double K_visc = 50.0 * 3.0e-5 * sigma2 * a * a / (om * om * om);
  double K_quad = C_D * sigma * a * 0.5 * rho * speed;
  return -(K_visc + K_quad);
}

__global__ void k_drag(int64_t n, const double* __restrict__ u, const double* __restrict__ v,
                       const double* __restrict__ w, const double* __restrict__ rho,
                       const double* __restrict__ as, double sigma, double sigma2, double C_D,
                       double* Fx, double* Fy, double* Fz) {
  int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (c >= n) return;
  double a = as[c];
  if (a <= 0.0) {
    Fx[c] = 0.0; Fy[c] = 0.0; Fz[c] = 0.0;
    return;
  }
  double ui = u[c], vi = v[c], wi = w[c];
  double co = drag_coeff(ui, vi, wi, rho[c], a, sigma, sigma2, C_D);
  Fx[c] = co * ui; Fy[c] = co * vi; Fz[c] = co * wi;
}

int launch_drag(int64_t n, const double* u, const double* v, const double* w, const double* rho,
                const double* as, double sigma, double C_D, double* Fx, double* Fy, double* Fz,
                cudaStream_t st) {
  k_drag<<<blocks_for(n, 256), 256, 0, st>>>(n, u, v, w, rho, as, sigma, sigma * sigma, C_D, Fx,
                                             Fy, Fz); fs_count_launch();
  return cuda_status();
}

// ---------------------------------------------------------------------------
// Tentative velocity (momentum_3d.py:42-276), optionally with the porous drag
// force evaluated in-kernel (drag_3d.py:128-144) instead of read from Fx/Fy/Fz.
// ---------------------------------------------------------------------------
struct MomArgs {
  const double *u, *v, *w, *rho, *T;
  const double *Fx, *Fy, *Fz;           // null when drag is fused
  const double *alpha_s;                // used when drag is fused
  const double *u_in, *v_in, *w_in;     // (Nz, Ny) inlet ghosts; v_in/w_in may be null
  double *uo, *vo, *wo;
  double sigma, sigma2, C_D;
  double dt, T_amb;
  double inv_dx, inv_dy, inv_dx2, inv_dy2;
};

// The planes of u, v and w in a ring, the cell's other inputs one level ahead in
// registers.  With a thread a cell and every neighbour loaded it was latency
// bound: 1200 instructions a warp, 98 registers, 12 warps an SM, 268 us at
// 400 x 120 x 60; 104 now.
typedef PlaneRing<double, 3, 2, 6> MomRing;
template <bool DIRECT>
__global__ void __launch_bounds__(MR_THREADS, 3) k_momentum(GridDev g, MomArgs a, int kz) {
  FOLLOW();
  extern __shared__ __align__(16) unsigned char mr_raw[];
  double* const ring = (double*)mr_raw;
  double* const rks = (double*)(mr_raw + (DIRECT ? 0 : MomRing::BYTES));
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const int64_t sz = (int64_t)nx * ny;
  const int k0 = blockIdx.z * kz, k1 = min(nz, k0 + kz);
  const double* const f[3] = {a.u, a.v, a.w};
  MomRing R;
  if constexpr (!DIRECT) {
    R.init(ring, g);
    for (int q = 0; q < 5; ++q) R.load(g, f, k0 - 2 + q, q);
    copy_commit();
  }
  march_spacings(g, k0, k1, rks);
  const int i = blockIdx.x * MR_TX + threadIdx.x, j = blockIdx.y * MR_TY + threadIdx.y;
  const bool inside = i < nx && j < ny;
  const int64_t col = (int64_t)min(j, ny - 1) * nx + min(i, nx - 1);
  double n_rho = a.rho[k0 * sz + col], n_T = a.T[k0 * sz + col];
  double n_as = a.Fx ? 0.0 : a.alpha_s[k0 * sz + col];
  const bool mx = i >= 2 && i <= nx - 3;
  const double g_T = 9.81 / a.T_amb;
  Near<DIRECT, MomRing::HX> N;
  N.init(g, i, min(j, ny - 1));
  int s = 2;  // the slot of plane k
  for (int k = k0; k < k1; ++k, s = MomRing::slot(s, 1)) {
    if constexpr (!DIRECT) copy_wait<0>();
    __syncthreads();
    if constexpr (!DIRECT) {
      if (k + 3 <= k1 + 1) R.load(g, f, k + 3, MomRing::slot(s, 3));
      copy_commit();
    }
    const double rho_i = n_rho, T = n_T, as = n_as;
    const int64_t c = k * sz + col;
    if (k + 1 < k1) {
      n_rho = a.rho[c + sz];
      n_T = a.T[c + sz];
      if (!a.Fx) n_as = a.alpha_s[c + sz];
    }
    if (!inside) continue;
    const double* const p0 = MomRing::at(ring, s);
    const double* const pl = MomRing::at(ring, MomRing::slot(s, -1));
    const double* const ph = MomRing::at(ring, MomRing::slot(s, 1));
    double vel[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) vel[q] = *(DIRECT ? f[q] + c : p0 + q * MomRing::PLANE);
    const bool ux = vel[0] >= 0.0, uy = vel[1] >= 0.0, uz = vel[2] >= 0.0;
    const double* const pf = MomRing::at(ring, MomRing::slot(s, uz ? -2 : 2));
    const int fx = ux ? -2 : 2, fy = uy ? N.yl2 : N.yr2;
    const double* rk = rks + (k - k0) * MR_RK;
    const double ida = rk[0], idb = rk[1], idz = rk[2], ihz = rk[3];
    const bool mz = k >= 2 && k <= nz - 3;
    const double inv_rho = 1.0 / rho_i;
    const double nu = 1.8e-5 * inv_rho;
    double F[3] = {0.0, 0.0, 0.0};
    if (a.Fx) {
      F[0] = a.Fx[c]; F[1] = a.Fy[c]; F[2] = a.Fz[c];
    } else if (!(as <= 0.0)) {
      const double co = drag_coeff(vel[0], vel[1], vel[2], rho_i, as, a.sigma, a.sigma2, a.C_D);
#pragma unroll
      for (int q = 0; q < 3; ++q) F[q] = co * vel[q];
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const double* const P = DIRECT ? f[q] + c : p0 + q * MomRing::PLANE;
      const double C = vel[q];
      double L = P[N.xl], H = P[N.xr];
      if (i == 0) {
        const double* in = q == 0 ? a.u_in : (q == 1 ? a.v_in : a.w_in);
        L = in ? in[(int64_t)k * ny + j] : 0.0;
      }
      if (i == nx - 1) H = C;
      double dp = H - C, dm = C - L;
      double n = ux ? L : H;
      const double dx = mx ? muscl_diff(dp, dm, C, n, P[fx], ux) : C - n;
      double d2 = (dp - dm) * a.inv_dx2;
      L = P[N.yl];
      H = P[N.yr];
      dp = H - C;
      dm = C - L;
      const double dy = muscl_diff(dp, dm, C, uy ? L : H, P[fy], uy);
      d2 += (dp - dm) * a.inv_dy2;
      L = k == 0 ? 0.0 : *(DIRECT ? P - sz : pl + q * MomRing::PLANE);
      H = k == nz - 1 ? C : *(DIRECT ? P + sz : ph + q * MomRing::PLANE);
      dp = H - C;
      dm = C - L;
      n = uz ? L : H;
      const double dz =
          mz ? muscl_diff(dp, dm, C, n,
                          *(DIRECT ? P + (uz ? -2 * sz : 2 * sz) : pf + q * MomRing::PLANE), uz) *
                   ihz
             : (C - n) * (uz ? idb : ida);
      d2 += (dp * ida - dm * idb) * idz;
      const double adv =
          -(fabs(vel[0]) * (dx * a.inv_dx) + fabs(vel[1]) * (dy * a.inv_dy) + fabs(vel[2]) * dz);
      double r = adv + nu * d2;
      if (q == 2) r += (T - a.T_amb) * g_T;
      r += F[q] * inv_rho;
      (q == 0 ? a.uo : (q == 1 ? a.vo : a.wo))[c] = C + r * a.dt;
    }
  }
}

int launch_momentum(const GridDev& g, const double* u, const double* v, const double* w,
                    const double* rho, const double* T, const double* Fx, const double* Fy,
                    const double* Fz, const double* alpha_s, double sigma, double C_D,
                    const double* u_in, const double* v_in, const double* w_in, double* uo,
                    double* vo, double* wo, double dt, double T_amb, cudaStream_t st) {
  MomArgs a{};
  a.u = u; a.v = v; a.w = w; a.rho = rho; a.T = T;
  a.Fx = Fx; a.Fy = Fy; a.Fz = Fz; a.alpha_s = alpha_s;
  if (!Fx && !alpha_s) return FS_EARG;
  a.u_in = u_in; a.v_in = v_in; a.w_in = w_in;
  a.uo = uo; a.vo = vo; a.wo = wo;
  a.sigma = sigma; a.sigma2 = sigma * sigma; a.C_D = C_D;
  a.dt = dt; a.T_amb = T_amb;
  a.inv_dx = 1.0 / g.dx; a.inv_dy = 1.0 / g.dy;
  a.inv_dx2 = a.inv_dx * a.inv_dx; a.inv_dy2 = a.inv_dy * a.inv_dy;
  if (march_direct<double>(g)) {
    following(k_momentum<true>, march_grid(g, 1), dim3(MR_TX, MR_TY), MR_RK_BYTES, st)(g, a, 1);
    fs_count_launch();
    return cuda_status();
  }
  const int kz = march_levels(g);
  if (!march_smem((const void*)k_momentum<false>, MomRing::BYTES + MR_RK_BYTES)) return cuda_status();
  following(k_momentum<false>, march_grid(g, kz), dim3(MR_TX, MR_TY), MomRing::BYTES + MR_RK_BYTES, st)(
      g, a, kz);
  fs_count_launch();
  return cuda_status();
}

// ---------------------------------------------------------------------------
// Outflow sponge (momentum_3d.py:293-317), in place
// ---------------------------------------------------------------------------
__global__ void k_sponge(GridDev g, double* u, const double* u_t,
                         const double* sig_x, const double* YF,
                         double skip, double dt) {
  FOLLOW();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  int j = blockIdx.y * blockDim.y + threadIdx.y;
  int k = blockIdx.z;
  if (i >= g.nx || j >= g.ny) return;
  double s = sig_x[i];
  int64_t c = cidx(g, k, j, i);
  if (s > 0.0 && YF[c] < skip) {
    double ut = u_t[(int64_t)k * g.ny + j];
    u[c] += s * dt * (ut - u[c]);
  }
}

int launch_sponge(const GridDev& g, double* u, const double* u_t, const double* sig_x,
                  const double* YF, double skip, double dt, cudaStream_t st) {
  Launch3 L = launch_cells(g);
  following(k_sponge, L.grid, L.block, 0, st)(g, u, u_t, sig_x, YF, skip, dt); fs_count_launch();
  return cuda_status();
}

// ---------------------------------------------------------------------------
// Realizable k-epsilon with in-kernel strain/vorticity invariants
// (turbulence_3d.py:392-478 _strain_and_vorticity_squared and :482-858
//  step_k_epsilon; buoyancy gradient with the one-sided boundary form of the
//  upstream fix, docs/js/physics/kepsilon.js:182-185,233-236)
// ---------------------------------------------------------------------------
struct KepsArgs {
  const double *k, *e, *u, *v, *w, *T, *alpha_s, *u_in, *kwall, *ewall;
  double *ko, *eo, *nuo;
  double *S2o, *O2o;  // optional outputs of the invariants (may be null)
  double sigma, dt, T_amb, beta_p, beta_d;
  double inv_dx, inv_dy, inv_dx2, inv_dy2;
};

#define K_MIN 1.0e-8
#define EPS_MIN 1.0e-8

// one transported scalar's advection and second differences
struct KepsTransport {
  double adv, d2;
};

// k and epsilon in a ring with two-cell halos, the velocity in one with single
// cells, T's column in registers.  The divisions are by common reciprocals
// (eight a cell, and two where the air is unstable), and tanh runs only there.  A
// thread a cell took 359 us at 400 x 120 x 60: 1490 instructions a warp and 12
// warps an SM waiting for loads; 140 now.
typedef PlaneRing<double, 2, 2, 6> KeRing;
typedef PlaneRing<double, 3, 1, 4> VelRing;
#define KEPS_SMEM (KeRing::BYTES + VelRing::BYTES)
template <bool DIRECT>
__global__ void __launch_bounds__(MR_THREADS, 2) k_keps(GridDev g, KepsArgs a, int kz) {
  FOLLOW();
  extern __shared__ __align__(16) unsigned char mr_raw[];
  double* const ring = (double*)mr_raw;
  double* const vring = (double*)(mr_raw + KeRing::BYTES);
  double* const rks = (double*)(mr_raw + (DIRECT ? 0 : KEPS_SMEM));
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const int64_t sz = (int64_t)nx * ny;
  const int k0 = blockIdx.z * kz, k1 = min(nz, k0 + kz);
  const double* const f[2] = {a.k, a.e};
  const double* const fv[3] = {a.u, a.v, a.w};
  KeRing R;
  VelRing V;
  if constexpr (!DIRECT) {
    R.init(ring, g);
    V.init(vring, g);
    for (int q = 0; q < 5; ++q) R.load(g, f, k0 - 2 + q, q);
    for (int q = 0; q < 3; ++q) V.load(g, fv, k0 - 1 + q, q);
    copy_commit();
  }
  march_spacings(g, k0, k1, rks);
  const int i = blockIdx.x * MR_TX + threadIdx.x, j = blockIdx.y * MR_TY + threadIdx.y;
  const bool inside = i < nx && j < ny;
  const int64_t col = (int64_t)min(j, ny - 1) * nx + min(i, nx - 1);
  double Tl = a.T[max(k0 - 1, 0) * sz + col], T0 = a.T[k0 * sz + col];
  double Th = a.T[min(k0 + 1, nz - 1) * sz + col];
  double n_as = a.alpha_s[k0 * sz + col];
  const bool mx = i >= 2 && i <= nx - 3;
  constexpr int VP = VelRing::PLANE;
  Near<DIRECT, KeRing::HX> N;
  Near<DIRECT, VelRing::HX> NV;
  N.init(g, i, min(j, ny - 1));
  NV.init(g, i, min(j, ny - 1));
  int s = 2, sv = 1;
  for (int k = k0; k < k1; ++k, s = KeRing::slot(s, 1), sv = VelRing::slot(sv, 1)) {
    if constexpr (!DIRECT) copy_wait<0>();
    __syncthreads();
    if constexpr (!DIRECT) {
      if (k + 3 <= k1 + 1) R.load(g, f, k + 3, KeRing::slot(s, 3));
      if (k + 2 <= k1) V.load(g, fv, k + 2, VelRing::slot(sv, 2));
      copy_commit();
    }
    const int64_t c = k * sz + col;
    const double as = n_as;
    const double Tn = a.T[min(k + 2, nz - 1) * sz + col];
    if (k + 1 < k1) n_as = a.alpha_s[c + sz];
    const double* rk = rks + (k - k0) * MR_RK;
    if (inside) {
      const double ida = rk[0], idb = rk[1], idz = rk[2], ihz = rk[3], idzc = rk[4];
      const double* const v0 = VelRing::at(vring, sv);
      const double* const vl = VelRing::at(vring, VelRing::slot(sv, -1));
      const double* const vh = VelRing::at(vring, VelRing::slot(sv, 1));
      double vel[3];
#pragma unroll
      for (int q = 0; q < 3; ++q) vel[q] = *(DIRECT ? fv[q] + c : v0 + q * VP);
      // the velocity gradient D[q][x, y, z]
      double D[3][3];
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const double* const P = DIRECT ? fv[q] + c : v0 + q * VP;
        const double xL = i == 0 ? (q == 0 ? a.u_in[(int64_t)k * ny + j] : 0.0) : P[NV.xl];
        const double xH = i == nx - 1 ? vel[q] : P[NV.xr];
        const double zL = k == 0 ? 0.0 : *(DIRECT ? P - sz : vl + q * VP);
        const double zH = k == nz - 1 ? vel[q] : *(DIRECT ? P + sz : vh + q * VP);
        D[q][0] = (xH - xL) * 0.5 * a.inv_dx;
        D[q][1] = (P[NV.yr] - P[NV.yl]) * 0.5 * a.inv_dy;
        D[q][2] = (zH - zL) * idzc;
      }
      const double S12 = 0.5 * (D[0][1] + D[1][0]), S13 = 0.5 * (D[0][2] + D[2][0]),
                   S23 = 0.5 * (D[1][2] + D[2][1]);
      const double S2 = 2.0 * (D[0][0] * D[0][0] + D[1][1] * D[1][1] + D[2][2] * D[2][2]) +
                        4.0 * (S12 * S12 + S13 * S13 + S23 * S23);
      const double O12 = 0.5 * (D[0][1] - D[1][0]), O13 = 0.5 * (D[0][2] - D[2][0]),
                   O23 = 0.5 * (D[1][2] - D[2][1]);
      const double O2 = 4.0 * (O12 * O12 + O13 * O13 + O23 * O23);
      if (a.S2o) { a.S2o[c] = S2; a.O2o[c] = O2; }

      const double* const p0 = KeRing::at(ring, s);
      const double* const pl = KeRing::at(ring, KeRing::slot(s, -1));
      const double* const ph = KeRing::at(ring, KeRing::slot(s, 1));
      const bool ux = vel[0] >= 0.0, uy = vel[1] >= 0.0, uz = vel[2] >= 0.0;
      const double* const pf = KeRing::at(ring, KeRing::slot(s, uz ? -2 : 2));
      const bool mz = k >= 2 && k <= nz - 3;
      double loc[2] = {*(DIRECT ? f[0] + c : p0), *(DIRECT ? f[1] + c : p0 + KeRing::PLANE)};
      if (loc[0] < K_MIN) loc[0] = K_MIN;
      if (loc[1] < EPS_MIN) loc[1] = EPS_MIN;
      KepsTransport tr[2];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const double* const P = DIRECT ? f[q] + c : p0 + q * KeRing::PLANE;
        const double C = loc[q];
        double L = i == 0 ? (q == 0 ? K_MIN : EPS_MIN) : P[N.xl], H = i == nx - 1 ? C : P[N.xr];
        double dp = H - C, dm = C - L, n = ux ? L : H;
        double adv = fabs(vel[0]) *
                     (mx ? muscl_diff(dp, dm, C, n, P[ux ? -2 : 2], ux) : C - n) * a.inv_dx;
        double d2 = (dp - dm) * a.inv_dx2;
        L = P[N.yl];
        H = P[N.yr];
        dp = H - C;
        dm = C - L;
        adv += fabs(vel[1]) *
               muscl_diff(dp, dm, C, uy ? L : H, P[uy ? N.yl2 : N.yr2], uy) * a.inv_dy;
        d2 += (dp - dm) * a.inv_dy2;
        L = k == 0 ? (q == 0 ? a.kwall : a.ewall)[col] : *(DIRECT ? P - sz : pl + q * KeRing::PLANE);
        H = k == nz - 1 ? C : *(DIRECT ? P + sz : ph + q * KeRing::PLANE);
        dp = H - C;
        dm = C - L;
        n = uz ? L : H;
        adv += fabs(vel[2]) *
               (mz ? muscl_diff(dp, dm, C, n,
                                *(DIRECT ? P + (uz ? -2 * sz : 2 * sz) : pf + q * KeRing::PLANE),
                                uz) *
                         ihz
                   : (C - n) * (uz ? idb : ida));
        d2 += (dp * ida - dm * idb) * idz;
        tr[q].adv = adv;
        tr[q].d2 = d2;
      }
      const double k_loc = loc[0], e_loc = loc[1];
      const double inv_e = 1.0 / e_loc, inv_k = 1.0 / k_loc;
      const double ke = k_loc * inv_e, ek = e_loc * inv_k;
      const double U_star = sqrt(0.5 * (S2 + O2));
      double nu_t = k_loc * ke / (4.04 + 4.5 * U_star * ke);
      if (nu_t < 0.0) nu_t = 0.0;
      double P_k_lim = nu_t * S2;
      if (P_k_lim > 10.0 * e_loc) P_k_lim = 10.0 * e_loc;
      const double dTdz = (Th - Tl) * idzc;  // (at the ground and the top Tl, Th repeat T0)
      // buoyant production: none where the gradient is stable or zero (it is formed
      // there too where the temperature that divides it is NaN or infinite)
      double G_k = 0.0, C3 = 0.0;
      if (!(nu_t * dTdz <= 0.0) || !(T0 < INFINITY)) {
        double Tfb = T0;
        if (Tfb < a.T_amb) Tfb = a.T_amb;
        G_k = (nu_t / 0.85) * (9.81 / Tfb) * dTdz;
        double u_h = sqrt(vel[0] * vel[0] + vel[1] * vel[1]);
        if (u_h < 0.01) u_h = 0.01;
        C3 = tanh(fabs(vel[2]) / u_h);
      }
      double G_kk = G_k;
      if (G_kk > P_k_lim) G_kk = P_k_lim;
      double Pc = 0.0, Dc = 0.0;
      if (as > 0.0) {
        const double speed =
            sqrt(vel[0] * vel[0] + vel[1] * vel[1] + vel[2] * vel[2]);
        const double cds = a.sigma * as * speed;
        Pc = a.beta_p * cds * speed * speed;
        Dc = a.beta_d * cds * k_loc;
      }
      // ---- k  (the BVG term is 0 at the production call site)
      const double diff_k = (1.5e-5 + nu_t) * tr[0].d2;
      double k_new = (k_loc + (diff_k - tr[0].adv + (P_k_lim + G_kk + Pc)) * a.dt) /
                     (1.0 + (e_loc + Dc) * a.dt * inv_k);
      if (k_new < K_MIN) k_new = K_MIN;
      // ---- epsilon
      const double diff_e = (1.5e-5 + nu_t * (1.0 / 1.3)) * tr[1].d2;
      const double eta = sqrt(S2) * ke;
      const double eta3 = eta * (eta * eta);
      double rng = 0.09 * eta3 * (1.0 - eta * (1.0 / 4.38)) / (1.0 + 0.012 * eta3);
      if (rng < 0.0) rng = 0.0;
      const double C2 = 1.92 + rng;
      const double S_pos_e = (1.44 * (P_k_lim + C3 * G_k) + 0.9 * Pc) * ek;
      const double S_neg_e = (C2 * e_loc + 0.9 * Dc) * ek;
      double e_new = (e_loc + (diff_e - tr[1].adv + S_pos_e) * a.dt) / (1.0 + S_neg_e * a.dt * inv_e);
      if (e_new < EPS_MIN) e_new = EPS_MIN;
      a.ko[c] = k_new;
      a.eo[c] = e_new;
      const double kn = k_new / e_new;
      double nu_new = k_new * kn / (4.04 + 4.5 * U_star * kn);
      if (nu_new < 0.0) nu_new = 0.0;
      a.nuo[c] = nu_new;
    }
    Tl = T0;
    T0 = Th;
    Th = Tn;
  }
}

int launch_keps(const GridDev& g, const double* k, const double* e, const double* u,
                const double* v, const double* w, const double* T, const double* alpha_s,
                const double* u_in, const double* kwall, const double* ewall, double* ko,
                double* eo, double* nuo, double* S2o, double* O2o, double sigma, double dt,
                double T_amb, double beta_p, double beta_d, cudaStream_t st) {
  KepsArgs a{};
  a.k = k; a.e = e; a.u = u; a.v = v; a.w = w; a.T = T; a.alpha_s = alpha_s; a.u_in = u_in;
  a.kwall = kwall; a.ewall = ewall; a.ko = ko; a.eo = eo; a.nuo = nuo; a.S2o = S2o; a.O2o = O2o;
  a.sigma = sigma; a.dt = dt; a.T_amb = T_amb; a.beta_p = beta_p; a.beta_d = beta_d;
  a.inv_dx = 1.0 / g.dx; a.inv_dy = 1.0 / g.dy;
  a.inv_dx2 = 1.0 / (g.dx * g.dx); a.inv_dy2 = 1.0 / (g.dy * g.dy);
  if (g.nz < 2) return FS_EARG;
  if (march_direct<double>(g)) {
    following(k_keps<true>, march_grid(g, 1), dim3(MR_TX, MR_TY), MR_RK_BYTES, st)(g, a, 1);
    fs_count_launch();
    return cuda_status();
  }
  const int kz = march_levels(g);
  if (!march_smem((const void*)k_keps<false>, KEPS_SMEM + MR_RK_BYTES)) return cuda_status();
  following(k_keps<false>, march_grid(g, kz), dim3(MR_TX, MR_TY), KEPS_SMEM + MR_RK_BYTES, st)(g, a, kz);
  fs_count_launch();
  return cuda_status();
}

// ---------------------------------------------------------------------------
// Vertical solid conduction on the bed T_s grid (solid_conduction_3d.py:56-127)
// ---------------------------------------------------------------------------
// cap = 1: the result is then clipped to [lo, hi] as k_clip does (the T_s
// cap that follows the conduction, spread_3d.py:3193-3196)
__global__ void k_solid_cond(GridDev g, const double* Ts,
                             const double* as, double* To,
                             double k_solid, double inv_rho_cp, double dt, int cap, double lo,
                             double hi) {
  FOLLOW();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  int j = blockIdx.y * blockDim.y + threadIdx.y;
  int k = blockIdx.z;
  if (i >= g.nx || j >= g.ny) return;
  const int64_t c = cidx(g, k, j, i);
  To[c] = solid_cond_cell(g, Ts, as, k, c, Ts[c], k_solid, inv_rho_cp, dt, cap, lo, hi);
}

int launch_solid_cond(const GridDev& g, const double* Ts, const double* as, double* To,
                      double k_solid, double rho_s, double cp_s, double dt, int nz_active,
                      cudaStream_t st, int cap, double lo, double hi) {
  GridDev gg = g;
  Launch3 L = launch_cells(g);
  (void)nz_active;
  following(k_solid_cond, L.grid, L.block, 0, st)(gg, Ts, as, To, k_solid, 1.0 / (rho_s * cp_s), dt,
                                           cap, lo, hi); fs_count_launch();
  return cuda_status();
}

// ---------------------------------------------------------------------------
// Soil columns (soil_3d.py:106-153): sequential in k per column (in-place
// Gauss-Seidel order: cell k sees the already-updated cell k-1).
// ---------------------------------------------------------------------------
__global__ void k_soil(int nsoil, int ny, int nx, double* T, const double* __restrict__ qin,
                       double dt, const double* __restrict__ sdz, const double* __restrict__ sda,
                       const double* __restrict__ sdb, double k_s, double rho_cp_inv,
                       double eps_s, double T_amb) {
  int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  int64_t n2 = (int64_t)ny * nx;
  if (q >= n2) return;
  for (int k = 0; k < nsoil; ++k) {
    double Tk = T[k * n2 + q];
    double qtop, qbot;
    if (k == 0) {
      double T2 = Tk * Tk;
      qtop = qin[q] - eps_s * 5.67e-8 * (T2 * T2);
    } else {
      qtop = k_s * (T[(k - 1) * n2 + q] - Tk) * (1.0 / sda[k]);
    }
    if (k == nsoil - 1) qbot = k_s * (Tk - T_amb) * (1.0 / sdb[k]);
    else qbot = k_s * (Tk - T[(k + 1) * n2 + q]) * (1.0 / sdb[k]);
    T[k * n2 + q] = Tk + dt * (qtop - qbot) * rho_cp_inv / sdz[k];
  }
}

int launch_soil(int nsoil, int ny, int nx, double* T, const double* qin, double dt,
                const double* sdz, const double* sda, const double* sdb, double k_s,
                double rho_s, double cp_s, double eps_s, double T_amb, cudaStream_t st) {
  int64_t n2 = (int64_t)ny * nx;
  k_soil<<<blocks_for(n2, 128), 128, 0, st>>>(nsoil, ny, nx, T, qin, dt, sdz, sda, sdb, k_s,
                                             1.0 / (rho_s * cp_s), eps_s, T_amb); fs_count_launch();
  return cuda_status();
}
