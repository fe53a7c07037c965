// Single-precision forms of the chemistry/transport sub-step kernels, for the
// mixed-precision solver (no counterpart in the reference, which is FP64
// throughout).  The ten sub-steps of an outer step (spread_3d.py:2678-3196)
// run on FP32 copies of the fields they update (T_g, Y_F, Y_O2, Y_H2O) and of
// the fields they only read (rho, u, v, w, k, eps, nu_t, the bed sources);
// the copies are made once before the first sub-step and T_g, the mass
// fractions, omega and Q_comb are widened back to FP64 after the last.  The
// solid conduction and every other operator of the step stay FP64.
//
// Each kernel restates its FP64 counterpart (transport.cu, pointwise.cu)
// expression for expression in float arithmetic: the EDC closure
// (edc.py:134-335, the same flat-order H2O-quench flag scan), the fused
// species step (species_3d.py:41-175 with the dilution sources and the O2
// clip), the turbulent diffusion sub-iteration (turbulence_3d.py:862-949)
// and the Lagrangian-branch gas-energy update (spread_3d.py:3088-3146).
#include "common.cuh"
#include "substep_march.cuh"
#include "kernels.h"

// ---- conversions -------------------------------------------------------------
#define CV_MAX 16
struct CvArgs {
  const void* src[CV_MAX];
  void* dst[CV_MAX];
  int nf;
};

__global__ void k_to_f32(int64_t n, CvArgs a) {
  FOLLOW();
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < n;
       c += (int64_t)gridDim.x * blockDim.x)
    for (int f = 0; f < a.nf; ++f) ((float*)a.dst[f])[c] = (float)((const double*)a.src[f])[c];
}

__global__ void k_to_f64(int64_t n, CvArgs a) {
  FOLLOW();
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < n;
       c += (int64_t)gridDim.x * blockDim.x)
    for (int f = 0; f < a.nf; ++f) ((double*)a.dst[f])[c] = (double)((const float*)a.src[f])[c];
}

int launch_convert(int64_t n, int nf, const void* const* src, void* const* dst, int to_f32,
                   cudaStream_t st) {
  if (nf < 1 || nf > CV_MAX || n < 0) return FS_EARG;
  if (n == 0) return FS_OK;
  CvArgs a{};
  a.nf = nf;
  for (int f = 0; f < nf; ++f) {
    a.src[f] = src[f];
    a.dst[f] = dst[f];
  }
  unsigned nb = blocks_for(n, 256);
  if (nb > 148 * 16) nb = 148 * 16;
  if (to_f32) following(k_to_f32, nb, 256, 0, st)(n, a);
  else following(k_to_f64, nb, 256, 0, st)(n, a);
  fs_count_launch();
  return cuda_status();
}

// ---- EDC -----------------------------------------------------------------------
// The FP64 kernels' tiling: EDC_TPB threads own EDC_TILE consecutive cells,
// EDC_CPT (four) per thread: consecutive in the flags' aggregate (one 16-byte load
// per field), a warp's width apart in the update.
#define E32_BLK EDC_TILE

__device__ __forceinline__ int edc_flag_code32(float Yf, float YO2, float YH, int t) {
  if (Yf <= 1e-9f || YO2 <= 1e-9f) return -1;
  int f = 0;
  if (YH > 0.0f) {
    float fac = 1.0f - YH / 0.18f;
    if (fac < 0.0f) fac = 0.0f;
    if (fac < 0.5f) f = 1;
  }
  return (t << 1) | f;
}

__device__ __forceinline__ void e32_ld4(const float* p, int64_t c0, int64_t n, bool vec, float* v) {
  if (vec) {
    const float4 x = *reinterpret_cast<const float4*>(p + c0);
    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
  } else {
#pragma unroll
    for (int q = 0; q < EDC_CPT; ++q) v[q] = (c0 + q < n) ? p[c0 + q] : 0.0f;
  }
}

__global__ void __launch_bounds__(EDC_TPB)
k_edc_agg32(int64_t n, const float* Yf, const float* YO, const float* YH, int vec_ok,
            signed char* agg) {
  FOLLOW();
  __shared__ int sh[EDC_TPB / 32];
  const int t = threadIdx.x;
  const int64_t c0 = (int64_t)blockIdx.x * E32_BLK + EDC_CPT * t;
  const bool vec = vec_ok && c0 + EDC_CPT <= n;
  // (O2 and H2O matter where there is fuel: a small part of the domain)
  float yf[EDC_CPT], yo[EDC_CPT] = {}, yh[EDC_CPT] = {};
  e32_ld4(Yf, c0, n, vec, yf);
  bool fuel = false;
#pragma unroll
  for (int q = 0; q < EDC_CPT; ++q) fuel |= c0 + q < n && !(yf[q] <= 1e-9f);
  if (fuel) {
    e32_ld4(YO, c0, n, vec, yo);
    e32_ld4(YH, c0, n, vec, yh);
  }
  int v = -1;
#pragma unroll
  for (int q = 0; q < EDC_CPT; ++q)
    if (c0 + q < n) v = max(v, edc_flag_code32(yf[q], yo[q], yh[q], EDC_CPT * t + q));
  const int lane = t & 31, wid = t >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
  if (lane == 0) sh[wid] = v;
  __syncthreads();
  if (t == 0) {
    for (int w = 1; w < EDC_TPB / 32; ++w) v = max(v, sh[w]);
    agg[blockIdx.x] = (signed char)(v < 0 ? -1 : (v & 1));
  }
}

struct Edc32Args {
  const float* rho;
  float *Tg, *Yf, *YO;
  const float *kt, *et, *YH;
  float* omega;
  const signed char* carry;
  float cp_g, dt, s_stoich, HoC_eff, relax, inv_s, inv_dt;
  int extinction, nsub, idle_ok;
};

// A cell without fuel or O2 has no reaction in any substep: the rate is 0 and
// its mass fractions keep their values, whatever k and epsilon are, as long as
// 0 / (rho cp) is a zero and the substep's length, the heat of combustion and the
// stoichiometry are finite (idle_ok: else 0 times them is NaN, in every cell).
__device__ __forceinline__ bool edc_idle32(const Edc32Args& a, float Yf, float YO2, float YH, float rho) {
  const float cp = (1.0f - YH) * a.cp_g + YH * 2000.0f;
  return a.idle_ok && (Yf <= 1e-9f || YO2 <= 1e-9f) && fabsf(rho) > 1e-37f && (cp > 0.0f || cp < 0.0f);
}
// what the update does to such a cell: the relaxation and the bounds
__device__ __forceinline__ void edc_idle_cell32(const Edc32Args& a, bool flag, float& Yf, float& YO2,
                                              float YH, float& Tg) {
  if (Yf < 0.0f) Yf = 0.0f;
  if (YO2 < 0.0f) YO2 = 0.0f;
  for (int sub = 0; sub < a.nsub; ++sub) {
    if (flag && Tg > 373.15f && YH > 0.0f) {
      float wb = YH * (1.0f / 0.10f);
      if (wb > 1.0f) wb = 1.0f;
      Tg = Tg - (Tg - 373.15f) * a.relax * wb;
    }
    if (Tg > 2400.0f) Tg = 2400.0f;
  }
}

// One cell's EDC update in float arithmetic (edc_cell's steps); Yf, YO2, Tg
// in place, the mean reaction rate returned.
__device__ __forceinline__ float edc_cell32(const Edc32Args& a, bool flag, float& Yf, float& YO2,
                                            float YH, float& Tg, float rho_i, float k_t,
                                            float e_t) {
  if (k_t < 1.0e-4f) k_t = 1.0e-4f;
  if (e_t < 1.0e-6f) e_t = 1.0e-6f;
  float ratio = 1.5e-5f * e_t / (k_t * k_t);
  if (ratio < 1e-30f) ratio = 1e-30f;
  const float gx = 2.1377f * sqrtf(sqrtf(ratio));
  float gamma_star = gx * (gx * gx);
  if (gamma_star > 1.0f) gamma_star = 1.0f;
  const float tau_star = 0.4083f * sqrtf(1.5e-5f / e_t);
  const float inv_tau = 1.0f / tau_star;
  const float inv_rho = 1.0f / rho_i;
  const float h = a.dt / (float)a.nsub;
  float acc = 0.0f;
  for (int sub = 0; sub < a.nsub; ++sub) {
    float omega;
    if (Yf <= 1e-9f || YO2 <= 1e-9f) {
      omega = 0.0f;
    } else {
      const float lim = YO2 * a.inv_s;
      const float Y_lim = Yf < lim ? Yf : lim;
      omega = gamma_star * (rho_i * Y_lim * inv_tau);
      if (YH > 0.0f) {
        float fac = 1.0f - YH * (1.0f / 0.18f);
        if (fac < 0.0f) fac = 0.0f;
        omega = omega * fac;
      }
    }
    bool fired = false;
    if (a.extinction && omega > 0.0f) {
      const float Yib = 1.0f - Yf - YO2;
      if (Yib > 0.88f) {
        float rs = (1.0f - Yib) * (1.0f / (1.0f - 0.88f));
        if (rs < 0.0f) rs = 0.0f;
        omega = omega * rs;
        if (rs < 0.5f) fired = true;
      }
      if (omega > 0.0f && Tg < 1200.0f) { omega = 0.0f; fired = true; }
      if (omega > 0.0f && omega * a.HoC_eff < 75000.0f) { omega = 0.0f; fired = true; }
    }
    if ((fired || flag) && Tg > 373.15f && YH > 0.0f) {
      float wb = YH * (1.0f / 0.10f);
      if (wb > 1.0f) wb = 1.0f;
      Tg = Tg - (Tg - 373.15f) * a.relax * wb;
    }
    const float dY = -omega * h * inv_rho;
    Yf = Yf + dY;
    if (Yf < 0.0f) Yf = 0.0f;
    YO2 = YO2 + a.s_stoich * dY;
    if (YO2 < 0.0f) YO2 = 0.0f;
    const float cp_mix = (1.0f - YH) * a.cp_g + YH * 2000.0f;
    Tg = Tg + omega * a.HoC_eff * h * inv_rho / cp_mix;
    if (Tg > 2400.0f) Tg = 2400.0f;
    acc += omega * h;
  }
  return a.dt > 0.0f ? acc * a.inv_dt : 0.0f;
}

// A warp owns EDC_CPT x 32 consecutive cells, 32 of them a pass, so the cells
// that react (a band of some tens in x) fill its lanes and the passes without
// any are short.  With four consecutive cells a thread the band kept a few
// lanes busy four cells deep: 26 us at 301 x 119 x 47, 22 so.
__global__ void __launch_bounds__(EDC_TPB, 4)
k_edc_main32(int64_t n, Edc32Args a) {
  FOLLOW();
  __shared__ int sh[EDC_TPB / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t c0 = (int64_t)blockIdx.x * EDC_TILE + wid * (32 * EDC_CPT) + lane;
  float yf[EDC_CPT], yo[EDC_CPT], yh[EDC_CPT], tg[EDC_CPT], rh[EDC_CPT];
#pragma unroll
  for (int q = 0; q < EDC_CPT; ++q) {
    const int64_t c = c0 + 32 * q;
    const bool in = c < n;
    yf[q] = in ? a.Yf[c] : 0.0f;
    yo[q] = in ? a.YO[c] : 0.0f;
    yh[q] = in ? a.YH[c] : 0.0f;
    tg[q] = in ? a.Tg[c] : 0.0f;
    rh[q] = in ? a.rho[c] : 1.0f;
  }
  bool cur = a.carry[blockIdx.x] > 0;
  // k and epsilon only where a cell may react
  bool idle[EDC_CPT];
  float kt[EDC_CPT] = {}, et[EDC_CPT] = {};
#pragma unroll
  for (int q = 0; q < EDC_CPT; ++q) {
    const int64_t c = c0 + 32 * q;
    idle[q] = c >= n || edc_idle32(a, yf[q], yo[q], yh[q], rh[q]);
    if (!idle[q]) {
      kt[q] = a.kt[c];
      et[q] = a.et[c];
    }
  }
  // the cells that set the quench flag, and those that set it to 1
  unsigned sets[EDC_CPT], ones[EDC_CPT];
  int last = -1;
#pragma unroll
  for (int q = 0; q < EDC_CPT; ++q) {
    const int code = edc_flag_code32(yf[q], yo[q], yh[q], 0);
    sets[q] = __ballot_sync(0xffffffffu, code >= 0);
    ones[q] = __ballot_sync(0xffffffffu, code == 1);
    if (sets[q]) last = (ones[q] >> (31 - __clz(sets[q]))) & 1;
  }
  if (lane == 0) sh[wid] = last;
  __syncthreads();
  for (int w = 0; w < wid; ++w)
    if (sh[w] >= 0) cur = sh[w] != 0;
#pragma unroll
  for (int q = 0; q < EDC_CPT; ++q) {
    const int64_t c = c0 + 32 * q;
    const unsigned upto = sets[q] & (0xffffffffu >> (31 - lane));
    const bool flag = upto ? (ones[q] >> (31 - __clz(upto))) & 1 : cur;
    if (sets[q]) cur = (ones[q] >> (31 - __clz(sets[q]))) & 1;
    if (c >= n) continue;
    float om = 0.0f;
    bool changed = true;
    if (idle[q]) {
      const float f0 = yf[q], o0 = yo[q], t0 = tg[q];
      edc_idle_cell32(a, flag, yf[q], yo[q], yh[q], tg[q]);
      changed = yf[q] != f0 || yo[q] != o0 || tg[q] != t0;
    } else {
      om = edc_cell32(a, flag, yf[q], yo[q], yh[q], tg[q], rh[q], kt[q], et[q]);
    }
    // (updated in place: where nothing changed the arrays hold the result)
    if (changed) {
      a.Yf[c] = yf[q];
      a.YO[c] = yo[q];
      a.Tg[c] = tg[q];
    }
    a.omega[c] = om;
  }
}

int64_t edc32_scratch_bytes(int64_t n) { return 2 * ((n + E32_BLK - 1) / E32_BLK) + 16; }

static bool al16(const void* p) { return ((uintptr_t)p & 15) == 0; }

int launch_edc32(int64_t n, const float* rho, float* Tg, float* Yf, float* YO, const float* kt,
                 const float* et, const float* YH, float* omega, double chi_rad, double cp_g,
                 double dt, int n_substeps, double s_stoich, double hoc_J, int extinction,
                 void* scratch, cudaStream_t st) {
  if (n == 0) return FS_OK;
  const int64_t nb = (n + E32_BLK - 1) / E32_BLK;
  signed char* agg = (signed char*)scratch;
  signed char* carry = agg + nb;
  const int vec_ok = al16(Yf) && al16(YO) && al16(YH);
  following(k_edc_agg32, (unsigned)nb, EDC_TPB, 0, st)(n, Yf, YO, YH, vec_ok, agg);
  fs_count_launch();
  int rc = launch_edc_carry((int)nb, agg, carry, st);
  if (rc != FS_OK) return rc;
  Edc32Args a{};
  a.rho = rho; a.Tg = Tg; a.Yf = Yf; a.YO = YO; a.kt = kt; a.et = et; a.YH = YH;
  a.omega = omega; a.carry = carry;
  a.cp_g = (float)cp_g; a.dt = (float)dt; a.s_stoich = (float)s_stoich;
  a.inv_s = (float)(1.0 / s_stoich);
  a.inv_dt = dt > 0.0 ? (float)(1.0 / dt) : 0.0f;
  a.HoC_eff = (float)(hoc_J * (1.0 - chi_rad));
  a.nsub = n_substeps > 1 ? n_substeps : 1;
  a.relax = (float)(1.0 - exp(-(dt / (double)a.nsub) / 0.5));
  a.extinction = extinction;
  a.idle_ok = isfinite(a.dt) && isfinite(a.HoC_eff) && isfinite(a.s_stoich);
  following(k_edc_main32, (unsigned)nb, EDC_TPB, 0, st)(n, a);
  fs_count_launch();
  return cuda_status();
}

// ---- species step and turbulent diffusion (the kernels: substep_march.cuh) -----
int launch_species_step32(const GridDev& g, const float* const* Y, float* const* Yo,
                          const float* Sp, const float* Sd, const double* Y_inlet,
                          const float* rho, const float* u, const float* v, const float* w,
                          double dt, double D, double o2_cap, cudaStream_t st) {
  SpeciesArgs<float> a{};
  for (int s = 0; s < 3; ++s) {
    a.Y[s] = Y[s];
    a.Yo[s] = Yo[s];
    a.Y_inlet[s] = (float)Y_inlet[s];
  }
  a.Sp = Sp; a.Sd = Sd; a.rho = rho; a.u = u; a.v = v; a.w = w;
  a.dt = (float)dt; a.D = (float)D; a.o2_cap = (float)o2_cap;
  a.inv_dx = (float)(1.0 / g.dx); a.inv_dy = (float)(1.0 / g.dy);
  a.inv_dx2 = (float)(1.0 / (g.dx * g.dx)); a.inv_dy2 = (float)(1.0 / (g.dy * g.dy));
  return launch_species_march<float, 3, true>(g, a, st);
}

int launch_turb_diff32(const GridDev& g, int nfield, const float* const* f, float* const* fo,
                       const float* nu_t, double sc_t, double dt_sub, int clip, const double* lo,
                       const double* hi, cudaStream_t st) {
  if (nfield != 1 && nfield != 3) return FS_EARG;
  DiffArgs<float> a{};
  a.nu_t = nu_t;
  a.inv_sc = (float)(1.0 / sc_t);
  a.dt = (float)dt_sub;
  a.inv_dx2 = (float)(1.0 / (g.dx * g.dx)); a.inv_dy2 = (float)(1.0 / (g.dy * g.dy));
  a.clip = clip;
  for (int s = 0; s < nfield; ++s) {
    a.f[s] = f[s];
    a.fo[s] = fo[s];
    a.lo[s] = clip ? (float)lo[s] : 0.0f;
    a.hi[s] = clip ? (float)hi[s] : 0.0f;
  }
  return nfield == 1 ? launch_turb_march<float, 1>(g, a, st) : launch_turb_march<float, 3>(g, a, st);
}

// ---- gas-energy update -------------------------------------------------------
struct Gas32Args {
  float* Tg;
  const float *rho, *YH, *Sp, *Sd, *Qgc;
  const double *Ts, *qrg;  // T_s (FP64 solid state) and the DOM's gas source
  float* Qcomb_out;
  float dt_sub, T_amb, q_drip_gas;
  int drip_on, n_z_bed, i_src0, i_src1;
};

__global__ void k_gas_update32(GridDev g, Gas32Args a) {
  FOLLOW();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int k = blockIdx.z;
  if (i >= g.nx || j >= g.ny) return;
  const int64_t c = cidx(g, k, j, i);
  float qc = 0.0f;
  if (a.drip_on && k < a.n_z_bed && i >= a.i_src0 && i < a.i_src1) qc = qc + a.q_drip_gas;
  qc = qc + (float)(a.qrg[c] / g.dz[k]);
  const float T = a.Tg[c];
  const float YH = a.YH[c];
  const float cp = (1.0f - YH) * 1100.0f + YH * 2000.0f;
  float d1 = T - (float)a.Ts[c];
  if (!(d1 >= 0.0f)) d1 = (d1 != d1) ? d1 : 0.0f;
  float d2 = T - 373.15f;
  if (!(d2 >= 0.0f)) d2 = (d2 != d2) ? d2 : 0.0f;
  const float debit = (a.Sp[c] * d1 + a.Sd[c] * d2) * 2000.0f;
  const float r = a.rho[c];
  const float rm = (r >= 1.0e-3f || r != r) ? r : 1.0e-3f;
  float Tn = T + (qc - a.Qgc[c] - debit) * (a.dt_sub / (rm * cp));
  if (Tn < a.T_amb) Tn = a.T_amb;
  a.Tg[c] = Tn;
  if (a.Qcomb_out) a.Qcomb_out[c] = qc;
}

int launch_gas_update32(const GridDev& g, float* Tg, const float* rho, const float* YH,
                        const double* Ts, const float* Sp, const float* Sd, const float* Qgc,
                        const double* qrg, float* Qcomb_out, double dt_sub, double T_amb,
                        double h_bed, int drip_on, int n_z_bed, int i_src0, int i_src1,
                        cudaStream_t st) {
  Gas32Args a{};
  a.Tg = Tg; a.rho = rho; a.YH = YH; a.Ts = Ts; a.Sp = Sp; a.Sd = Sd; a.Qgc = Qgc; a.qrg = qrg;
  a.Qcomb_out = Qcomb_out;
  a.dt_sub = (float)dt_sub; a.T_amb = (float)T_amb;
  const double q_drip = 30000.0 / (h_bed > 1e-3 ? h_bed : 1e-3);
  a.q_drip_gas = (float)((1.0 - 0.80) * q_drip);
  a.drip_on = drip_on; a.n_z_bed = n_z_bed; a.i_src0 = i_src0; a.i_src1 = i_src1;
  Launch3 L = launch_cells(g);
  following(k_gas_update32, L.grid, L.block, 0, st)(g, a);
  fs_count_launch();
  return cuda_status();
}

// ---- clip ------------------------------------------------------------------------
__global__ void k_clip32(int64_t n, float* f, float lo, float hi) {
  FOLLOW();
  const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (c >= n) return;
  float x = f[c];
  if (x > hi) x = hi;
  if (x < lo) x = lo;
  f[c] = x;
}

int launch_clip32(int64_t n, float* f, double lo, double hi, cudaStream_t st) {
  if (n == 0) return FS_OK;
  following(k_clip32, blocks_for(n, 256), 256, 0, st)(n, f, (float)lo, (float)hi);
  fs_count_launch();
  return cuda_status();
}
