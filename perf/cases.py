"""Workloads of the Tier-3 fire step, as a user's program calls them.

Kinds of case:

``step``       one outer step of a case through :class:`firewebapp_b200.ctx.StepContext`
``radiation``  one discrete-ordinates solve (``fs_dom_solve``)
``pressure``   tentative velocity, divergence target, operator rebuild and
               projection with its divergence test, marching in time
``explicit``   the explicit flow operators: tentative velocity, k-epsilon and
               gas-temperature advection
``substep``    one chemistry/transport sub-step: EDC, species, turbulent
               diffusion, gas energy and solid conduction, marching in time

``nx``, ``ny``, ``nz`` are the grid's cells, ``order`` the quadrature (S4, S6,
S8) and ``form`` the solver's form: ``plain`` is FP64 throughout, ``mixed``
runs the sweep, the preconditioner and the sub-steps in FP32.  The grid is the
400 x 120 x 60 workload's (dx = dy = 0.1 m, dz = 0.0625 m, four bed layers) or
a part of it; fields hold a wind profile and a flame line over a grass bed.
"""
import ctypes as C
import math

import numpy as np
import torch

from firewebapp_b200 import _lib
from firewebapp_b200._lib import FsGrid, check, dbl_array, ptr, ptr_array
from firewebapp_b200.cases import CFG1, CFG2, scaled
from firewebapp_b200.ctx import FIELD_IDS, StepContext
from firewebapp_b200.quadrature import level_symmetric

DX, DZ, NBED = 0.1, 0.0625, 4
T_AMB, P0, R_AIR, SIGMA = 300.0, 101325.0, 287.0, 5.67e-8
SAV, C_D, K_GAS, EPS_W, RELAX, TOL = 12240.0, 0.30, 0.5, 0.85, 0.7, 1.0e-3
DT, RTOL = 4.0e-3, 1.0e-6
DT_SUB = DT / 10
SC_T, PR_T, T_CAP = 0.7, 0.85, 1.0e4
CHI, CP_G, S_ST, HOC = 0.34, 1100.0, 1.3, 1.7e7
K_S, RHO_S, CP_S, H_BED = 0.20, 500.0, 1300.0, 0.25
# state that the sub-steps leave in FP32 in the mixed form, and the fields of
# a step that a run's snapshots and front tracking read
STEP_OUT = ("rho", "u", "v", "w", "T_g", "Y_fuel", "Y_O2", "Y_H2O", "T_s", "k_turb", "eps_turb",
            "nu_t", "omega", "q_rad", "q_rad_gas", "T_soil", "p_prev", "p_m_solid", "p_T_s")


def listed():
    return [
        # the CPU-runnable 64 x 24 x 20 case: launches and host waits count
        dict(name="step_64x24x20", kind="step", nx=64, ny=24, nz=20, order=4, form="plain"),
        # a ragged, odd grid at the middle of the range
        dict(name="step_133x45x37_mixed", kind="step", nx=133, ny=45, nz=37, order=6, form="mixed"),
        # the workload itself, in both forms
        dict(name="step_400x120x60", kind="step", nx=400, ny=120, nz=60, order=8, form="plain"),
        dict(name="step_400x120x60_mixed", kind="step", nx=400, ny=120, nz=60, order=8,
             form="mixed"),
        # radiation alone: a small odd grid, the workload's, and the longest
        # domain of the batched sweep (Nx 200 to 600)
        dict(name="radiation_97x41x23", kind="radiation", nx=97, ny=41, nz=23, order=4,
             form="plain"),
        dict(name="radiation_400x120x60", kind="radiation", nx=400, ny=120, nz=60, order=8,
             form="plain"),
        dict(name="radiation_600x120x60_mixed", kind="radiation", nx=600, ny=120, nz=60, order=8,
             form="mixed"),
        # the pressure step: small and odd (latency of the coarse levels), and
        # the workload's
        dict(name="pressure_115x37x29", kind="pressure", nx=115, ny=37, nz=29, order=4,
             form="plain"),
        dict(name="pressure_400x120x60", kind="pressure", nx=400, ny=120, nz=60, order=8,
             form="plain"),
        # the explicit stencils of the flow
        dict(name="explicit_400x120x60", kind="explicit", nx=400, ny=120, nz=60, order=8,
             form="plain"),
        # a chemistry/transport sub-step (ten per outer step) in each precision
        dict(name="substep_400x120x60", kind="substep", nx=400, ny=120, nz=60, order=8,
             form="plain"),
        dict(name="substep_301x119x47_mixed", kind="substep", nx=301, ny=119, nz=47, order=8,
             form="mixed"),
    ]


def draw(rng):
    kind = rng.choice(("step", "radiation", "radiation", "pressure", "explicit", "substep",
                       "substep"))
    order = rng.choice((4, 6, 8, 8))
    form = rng.choice(("plain", "mixed")) if kind in ("step", "radiation", "substep") else "plain"
    top = 4_320_000 if (kind, form) == ("radiation", "mixed") else 2_880_000
    while True:
        nx = round(math.exp(rng.uniform(math.log(48), math.log(600))))
        ny = round(math.exp(rng.uniform(math.log(9), math.log(120))))
        nz = round(math.exp(rng.uniform(math.log(12), math.log(60))))
        if nx * ny * nz <= top:
            return dict(kind=kind, nx=nx, ny=ny, nz=nz, order=order, form=form)


# ---- inputs --------------------------------------------------------------------
def _noise(gen, shape, dev):
    """Smooth noise of unit amplitude: coarse normal values, interpolated."""
    low = [max(2, s // 8) for s in shape]
    a = torch.randn([1, 1] + low, generator=gen, device=dev, dtype=torch.float64)
    a = torch.nn.functional.interpolate(a, size=tuple(shape), mode="trilinear",
                                        align_corners=True)
    return a[0, 0].clamp(-3.0, 3.0)


def _fields(case, seed, dev="cuda"):
    """A wind profile over a grass bed with a wavy flame line across it."""
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed))
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    shp = (nz, ny, nx)
    f64 = dict(dtype=torch.float64, device=dev)
    u01 = torch.rand(4, generator=gen, **f64).tolist()
    x = (torch.arange(nx, **f64) + 0.5) * DX
    y = (torch.arange(ny, **f64) + 0.5) * DX
    z = (torch.arange(nz, **f64) + 0.5) * DZ
    n = [_noise(gen, shp, dev) for _ in range(6)]
    front = (0.25 + 0.3 * u01[0]) * nx * DX + 0.4 * torch.sin(y * (1.0 + u01[1]))
    d = x[None, None, :] - front[None, :, None] - 0.3 * z[:, None, None]
    hot = torch.exp(-(d / 0.6) ** 2 - z[:, None, None] / 1.2) * (0.8 + 0.1 * n[0])
    hot = hot.clamp(0.0, 1.0)
    bed = ((z < NBED * DZ)[:, None, None] & (x > 0.5)[None, None, :]).expand(shp)
    f = {}
    f["T_g"] = T_AMB + 1500.0 * hot
    f["rho"] = P0 / (R_AIR * f["T_g"])
    f["rho_prev"] = f["rho"] * (1.0 + 1.0e-4 * hot * n[1])
    f["Y_fuel"] = (0.12 * hot * (1.0 + 0.2 * n[1])).clamp(0.0, 1.0)
    f["Y_O2"] = (0.232 * (1.0 - 0.7 * hot)).clamp(0.0, 0.232)
    f["Y_H2O"] = (0.008 + 0.06 * hot * (1.0 + 0.3 * n[2])).clamp(0.0, 1.0)
    f["omega"] = torch.where(hot > 0.35, 0.4 * hot, torch.zeros_like(hot))
    f["alpha_s"] = torch.where(bed, 9.0e-4, 0.0).to(torch.float64).contiguous()
    f["T_s"] = torch.where(bed, T_AMB + 700.0 * hot, torch.full_like(hot, T_AMB))
    ahead = (d > 0.0) & bed
    f["M_local"] = torch.where(ahead, 0.04 + 0.04 * u01[2], 0.0).to(torch.float64).contiguous()
    f["S_pyro"] = torch.where(bed, 0.3 * hot, torch.zeros_like(hot))
    f["S_drying"] = torch.where(ahead, 0.1 * hot, torch.zeros_like(hot))
    f["Q_g_conv"] = torch.where(bed, 4.0e4 * hot * (1.0 + 0.2 * n[3]), torch.zeros_like(hot))
    f["q_rad_gas"] = -3.0e3 * hot * (1.0 + 0.2 * n[4])
    U = (4.0 + 3.0 * u01[3]) * torch.log((z + 0.01) / 0.01) / math.log(10.01 / 0.01)
    f["u_inlet"] = U[:, None].expand(nz, ny).contiguous()
    f["u"] = U[:, None, None] + 0.3 * n[2] - 0.4 * hot
    f["v"] = 0.25 * n[3]
    f["w"] = 0.15 * n[4] + 1.5 * hot
    f["k_turb"] = 0.05 + 0.5 * hot + 0.02 * n[5].abs()
    f["eps_turb"] = 0.09 * f["k_turb"] ** 1.5 / 0.15
    f["nu_t"] = 0.09 * f["k_turb"] ** 2 / f["eps_turb"]
    f["T_soil"] = T_AMB + 40.0 * hot[0].contiguous()
    return {k: v.contiguous() for k, v in f.items()}


class _Handle:
    """A library object that is destroyed with the state that holds it."""

    def __init__(self, create, destroy, *args):
        self.h, self.destroy = C.c_void_p(), destroy
        check(create(*args, C.byref(self.h)))

    def __del__(self):
        if self.h:
            self.destroy(self.h)


class _Buffer:
    """A buffer of the library as a tensor; `keep` lives as long as the tensor."""

    def __init__(self, addr, shape, keep, typestr="<f8"):
        self.keep = keep
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": typestr, "version": 3,
                                         "data": (int(addr), False), "strides": None}

    def tensor(self):
        return torch.as_tensor(self, device="cuda")


def _step_case(case, seed):
    rng = np.random.default_rng(seed)
    base = CFG1 if case["order"] == 4 else CFG2
    c = scaled(base, nx=case["nx"], ny=case["ny"], nz=case["nz"])
    c.update(n_quadrature=case["order"], wind_speed_m_s=float(rng.uniform(3.0, 7.0)),
             initial_moisture_frac=float(rng.uniform(0.03, 0.10)), jitter_seed=int(seed))
    return c


def prepare(case, seed):
    L = _lib.lib()
    kind, form = case["kind"], case["form"]
    st = {"kind": kind, "form": form, "lib": L}
    f = _fields(case, seed)
    if kind == "step":
        ctx = StepContext(_step_case(case, seed), form=form)
        for k in ("T_g", "Y_fuel", "Y_O2", "Y_H2O", "u", "v", "w"):
            ctx.write(k, f[k].cpu().numpy())
        st.update(ctx=ctx)
        return st
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    shp = (nz, ny, nx)
    f64 = dict(dtype=torch.float64, device="cuda")
    dz = torch.full((nz,), DZ, **f64)
    da, db = dz.clone(), dz.clone()
    da[-1] = 0.5 * DZ
    db[0] = 0.5 * DZ
    grid = FsGrid(nx, ny, nz, DX, DX, ptr(dz), ptr(da), ptr(db))
    st.update(f=f, geo=(dz, da, db), grid=grid, g=C.byref(grid), n=nx * ny * nz)

    def empty(count, dtype=torch.float64):
        return [torch.zeros(shp, dtype=dtype, device="cuda") for _ in range(count)]

    if kind == "radiation":
        om, wq = level_symmetric(case["order"])
        st["dom"] = _Handle(L.fs_dom_create, L.fs_dom_destroy, st["g"], om.shape[0],
                            dbl_array(om[:, 0]), dbl_array(om[:, 1]), dbl_array(om[:, 2]),
                            dbl_array(wq), K_GAS)
        if form == "mixed":
            check(L.fs_dom_set_precision(st["dom"].h, 1))
        st["out"] = empty(2) + [torch.zeros((ny, nx), **f64)]
    elif kind == "pressure":
        st["proj"] = _Handle(L.fs_proj_create, L.fs_proj_destroy, st["g"])
        st["zero2"] = torch.zeros((nz, ny), **f64)
        st["new"] = empty(3)
        st["target"] = empty(1)[0]
        st["p"] = _Buffer(L.fs_proj_pressure(st["proj"].h), shp, st["proj"]).tensor()
    elif kind == "explicit":
        st["zero2"] = torch.zeros((nz, ny), **f64)
        st["wall"] = [torch.full((ny, nx), 1.0e-8, **f64) for _ in range(2)]
        st["out"] = empty(7)
    else:
        if form == "mixed":
            for k in ("T_g", "Y_fuel", "Y_O2", "Y_H2O", "rho", "u", "v", "w", "k_turb", "eps_turb",
                      "nu_t", "S_pyro", "S_drying", "Q_g_conv", "omega"):
                f[k] = f[k].float()
            dt = torch.float32
            size = L.fs_edc_f32_scratch_bytes(st["n"])
        else:
            dt = torch.float64
            size = L.fs_edc_scratch_bytes(st["n"])
        st["tmp"] = empty(4, dt)
        st["ts_new"] = empty(1)[0]
        st["Q_comb"] = empty(1, dt)[0]
        st["scratch"] = torch.zeros(int(size) + 64, dtype=torch.uint8, device="cuda")
    return st


# ---- one pass --------------------------------------------------------------------
def _tentative(st, out):
    f = st["f"]
    check(st["lib"].fs_tentative_velocity(
        st["g"], ptr(f["u"]), ptr(f["v"]), ptr(f["w"]), ptr(f["rho"]), ptr(f["T_g"]), None, None,
        None, ptr(f["alpha_s"]), SAV, C_D, ptr(f["u_inlet"]), ptr(st["zero2"]), ptr(st["zero2"]),
        ptr(out[0]), ptr(out[1]), ptr(out[2]), DT, T_AMB, _lib.stream_ptr()))


def _run_step(st):
    ctx = st["ctx"]
    ctx.step(1)
    out = {}
    for name in STEP_OUT:
        fid = FIELD_IDS[name]
        size = int(ctx.lib.fs_ctx_field_size(ctx.h, fid))
        out[name] = _Buffer(ctx.lib.fs_ctx_field(ctx.h, fid), (size,), ctx).tensor()
    if st["form"] == "mixed":
        # results of FP32 arithmetic, in the type that snapshots hold them in
        out = {k: v.float() for k, v in out.items()}
    return out


def _run_radiation(st):
    f, (qs, qg, qsoil) = st["f"], st["out"]
    check(st["lib"].fs_dom_solve(
        st["dom"].h, ptr(f["T_s"]), ptr(f["T_g"]), ptr(f["alpha_s"]), ptr(f["omega"]), SAV, T_AMB,
        ptr(f["T_soil"]), ptr(f["Y_H2O"]), ptr(f["rho"]), ptr(f["M_local"]), ptr(qs), ptr(qg),
        ptr(qsoil), _lib.stream_ptr()))
    out = {"q_rad": qs, "q_rad_gas": qg, "q_in_soil": qsoil}
    if st["form"] == "mixed":
        out = {k: v.float() for k, v in out.items()}
    return out


def _run_pressure(st):
    L, f, s = st["lib"], st["f"], _lib.stream_ptr()
    new = st["new"]
    _tentative(st, new)
    check(L.fs_div_target(st["n"], ptr(f["rho"]), ptr(f["rho_prev"]), ptr(f["S_pyro"]),
                          ptr(f["S_drying"]), DT, ptr(st["target"]), s))
    check(L.fs_proj_rebuild(st["proj"].h, ptr(f["rho"]), s))
    its, res = C.c_int(), C.c_double()
    check(L.fs_proj_project(st["proj"].h, ptr(new[0]), ptr(new[1]), ptr(new[2]), ptr(f["u_inlet"]),
                            ptr(st["target"]), DT, RTOL, 200, C.byref(its), s))
    check(L.fs_divergence_max(st["g"], ptr(new[0]), ptr(new[1]), ptr(new[2]), ptr(f["u_inlet"]),
                              ptr(st["target"]), None, C.byref(res), s))
    for q, k in enumerate(("u", "v", "w")):
        f[k], new[q] = new[q], f[k]
    return {"u": f["u"], "v": f["v"], "w": f["w"], "p": st["p"], "target": st["target"]}


def _run_explicit(st):
    L, f, o = st["lib"], st["f"], st["out"]
    s = _lib.stream_ptr()
    _tentative(st, o)
    check(L.fs_k_epsilon(st["g"], ptr(f["k_turb"]), ptr(f["eps_turb"]), ptr(f["u"]), ptr(f["v"]),
                         ptr(f["w"]), ptr(f["T_g"]), ptr(f["alpha_s"]), ptr(f["u_inlet"]),
                         ptr(st["wall"][0]), ptr(st["wall"][1]), ptr(o[3]), ptr(o[4]), ptr(o[5]),
                         None, None, SAV, DT, T_AMB, 1.0, 4.0, s))
    check(L.fs_gas_energy_adv(st["g"], ptr(f["T_g"]), ptr(f["u"]), ptr(f["v"]), ptr(f["w"]),
                              ptr(o[6]), DT, 2.0e-5, T_AMB, s))
    return dict(zip(("u", "v", "w", "k", "eps", "nu_t", "T_g"), o))


def _run_substep(st):
    L, f, t, g, n = st["lib"], st["f"], st["tmp"], st["g"], st["n"]
    s = _lib.stream_ptr()
    mixed = st["form"] == "mixed"
    edc = L.fs_edc_f32 if mixed else L.fs_edc
    check(edc(n, ptr(f["rho"]), ptr(f["T_g"]), ptr(f["Y_fuel"]), ptr(f["Y_O2"]), ptr(f["k_turb"]),
              ptr(f["eps_turb"]), ptr(f["Y_H2O"]), ptr(f["omega"]), CHI, CP_G, DT_SUB, 1, S_ST,
              HOC, 0, ptr(st["scratch"]), s))
    names = ("Y_fuel", "Y_O2", "Y_H2O")

    def swap():
        for q, k in enumerate(names):
            f[k], t[q] = t[q], f[k]

    species = L.fs_species_step_f32 if mixed else L.fs_species_step
    check(species(g, ptr_array([f[k] for k in names]), ptr_array(t[:3]), ptr(f["S_pyro"]),
                  ptr(f["S_drying"]), dbl_array([0.0, 0.232, 0.0]), ptr(f["rho"]), ptr(f["u"]),
                  ptr(f["v"]), ptr(f["w"]), DT_SUB, 1.0e-5, 0.232, s))
    swap()
    diff = L.fs_turb_diffusion_substep_f32 if mixed else L.fs_turb_diffusion_substep
    check(diff(g, 3, ptr_array([f[k] for k in names]), ptr_array(t[:3]), ptr(f["nu_t"]), SC_T,
               DT_SUB, 1, dbl_array([0.0, 0.0, 0.0]), dbl_array([1.0, 0.232, 1.0]), s))
    swap()
    gas = (g, ptr(f["T_g"]), ptr(f["rho"]), ptr(f["Y_H2O"]), ptr(f["T_s"]), ptr(f["S_pyro"]),
           ptr(f["S_drying"]), ptr(f["Q_g_conv"]), ptr(f["q_rad_gas"]), ptr(st["Q_comb"]), DT_SUB,
           T_AMB, H_BED, 1, NBED, 5, 7)
    if mixed:
        check(L.fs_gas_energy_update_f32(*gas, s))
        check(L.fs_solid_conduction_capped(g, ptr(f["T_s"]), ptr(f["alpha_s"]),
                                           ptr(st["ts_new"]), K_S, RHO_S, CP_S, DT_SUB, T_AMB,
                                           T_CAP, s))
    else:
        check(L.fs_gas_energy_solid_update(*gas, ptr(f["alpha_s"]), ptr(st["ts_new"]), K_S, RHO_S,
                                           CP_S, T_AMB, T_CAP, s))
    f["T_s"], st["ts_new"] = st["ts_new"], f["T_s"]
    check(diff(g, 1, ptr_array([f["T_g"]]), ptr_array([t[3]]), ptr(f["nu_t"]), PR_T, DT_SUB, 1,
               dbl_array([T_AMB]), dbl_array([T_CAP]), s))
    f["T_g"], t[3] = t[3], f["T_g"]
    return {"T_g": f["T_g"], "Y_fuel": f["Y_fuel"], "Y_O2": f["Y_O2"], "Y_H2O": f["Y_H2O"],
            "omega": f["omega"], "T_s": f["T_s"], "Q_comb": st["Q_comb"]}


def run(state):
    return {"step": _run_step, "radiation": _run_radiation, "pressure": _run_pressure,
            "explicit": _run_explicit, "substep": _run_substep}[state["kind"]](state)


# ---- the work of one pass -----------------------------------------------------------
def work(case):
    n = case["nx"] * case["ny"] * case["nz"]
    n2 = case["nx"] * case["ny"]
    M = {4: 24, 6: 48, 8: 80}[case["order"]]
    # a radiation solve runs at least two source iterations of M ordinates:
    # about ten operations to a cell and ordinate
    dom = 2 * M * n * 10
    mixed = case["form"] == "mixed"
    size = 4 if mixed else 8
    kind = case["kind"]
    if kind == "step":
        # 14 state fields in and out, three radiative/reaction fields out, the
        # particles' eleven arrays in and six out, six soil layers
        parts = 16 * NBED * n2 if case["order"] != 4 else 4 * 2 * n2
        return {"bytes": 8 * (31 * n + 12 * n2 + 17 * parts), "flops": dom + 12_000 * n}
    if kind == "radiation":
        return {"bytes": 8 * (7 * n + n2) + size * (2 * n + n2), "flops": dom}
    if kind == "pressure":
        return {"bytes": 8 * (9 * n + 5 * n), "flops": 600 * n}
    if kind == "explicit":
        return {"bytes": 8 * (8 * n + 7 * n), "flops": 800 * n}
    # 14 sub-step fields in, six out; T_s, alpha_s and the radiative source in
    # FP64, T_s out
    return {"bytes": size * (14 * n + 6 * n) + 8 * 4 * n, "flops": 450 * n}


# ---- the same passes in 64-bit torch -----------------------------------------------
def _zvec(v):
    return v[:, None, None]


class _Geo:
    def __init__(self, case, dev):
        nz = case["nz"]
        self.dz = torch.full((nz,), DZ, dtype=torch.float64, device=dev)
        self.da, self.db = self.dz.clone(), self.dz.clone()
        self.da[-1] = 0.5 * DZ
        self.db[0] = 0.5 * DZ


def _minmod(a, b):
    m = torch.copysign(torch.minimum(a.abs(), b.abs()), a)
    return torch.where(a * b <= 0.0, torch.zeros_like(m), m)


def _face(m1, c, p1, p2, vel):
    up = vel >= 0.0
    s = _minmod(p1 - c, torch.where(up, c - m1, p2 - p1))
    return torch.where(up, c + 0.5 * s, p1 - 0.5 * s)


def _sh(f, dim, o):
    """f at the neighbour `o` away (periodic; the ends are replaced by the caller)."""
    return torch.roll(f, -o, dim)


def _edge(f, dim, where, value):
    f = f.clone()
    f.select(dim, where).copy_(value)
    return f


def _inner(shape, dim, dev):
    i = torch.arange(shape[dim], device=dev)
    ok = (i >= 2) & (i <= shape[dim] - 3)
    return ok[:, None, None] if dim == 0 else ok[None, None, :]


def _neighbours(f, inlet, below=None):
    """x and z neighbours with the boundary values of the transport stencils."""
    xL = _edge(_sh(f, 2, -1), 2, 0, inlet)
    xR = _edge(_sh(f, 2, 1), 2, -1, f[:, :, -1])
    zL = _edge(_sh(f, 0, -1), 0, 0, f[0] if below is None else below)
    zR = _edge(_sh(f, 0, 1), 0, -1, f[-1])
    return xL, xR, zL, zR


def _grad(f, u, v, w, geo, nb, c=None):
    """Upwind-biased derivatives of f along x, y and z; `c`: the centre values."""
    c = f if c is None else c
    xL, xR, zL, zR = nb
    mx, mz = _inner(f.shape, 2, f.device), _inner(f.shape, 0, f.device)
    fx = (_face(_sh(f, 2, -1), c, _sh(f, 2, 1), _sh(f, 2, 2), u)
          - _face(_sh(f, 2, -2), _sh(f, 2, -1), c, _sh(f, 2, 1), u)) / DX
    fx = torch.where(mx, fx, torch.where(u >= 0.0, c - xL, xR - c) / DX)
    fy = (_face(_sh(f, 1, -1), c, _sh(f, 1, 1), _sh(f, 1, 2), v)
          - _face(_sh(f, 1, -2), _sh(f, 1, -1), c, _sh(f, 1, 1), v)) / DX
    hz = _zvec(0.5 * (geo.da + geo.db))
    fz = (_face(_sh(f, 0, -1), c, _sh(f, 0, 1), _sh(f, 0, 2), w)
          - _face(_sh(f, 0, -2), _sh(f, 0, -1), c, _sh(f, 0, 1), w)) / hz
    fz = torch.where(mz, fz, torch.where(w >= 0.0, (c - zL) / _zvec(geo.db),
                                         (zR - c) / _zvec(geo.da)))
    return fx, fy, fz


def _lap(f, geo, nb, c=None):
    c = f if c is None else c
    xL, xR, zL, zR = nb
    return ((xR - 2 * c + xL) / DX ** 2 + (_sh(f, 1, 1) - 2 * c + _sh(f, 1, -1)) / DX ** 2
            + ((zR - c) / _zvec(geo.da) - (c - zL) / _zvec(geo.db)) / _zvec(geo.dz))


def _exact_tentative(f, geo):
    u, v, w = f["u"], f["v"], f["w"]
    speed = torch.sqrt(u * u + v * v + w * w)
    a = f["alpha_s"]
    co = -(50.0 * 3.0e-5 * SAV ** 2 * a * a / (1.0 - a) ** 3 + C_D * SAV * a * 0.5 * f["rho"] * speed)
    out = []
    for q, inlet in ((u, f["u_inlet"]), (v, 0.0), (w, 0.0)):
        inlet = inlet if torch.is_tensor(inlet) else torch.zeros_like(f["u_inlet"])
        nb = _neighbours(q, inlet, torch.zeros_like(q[0]))
        gx, gy, gz = _grad(q, u, v, w, geo, nb)
        rate = -(u * gx + v * gy + w * gz) + 1.8e-5 / f["rho"] * _lap(q, geo, nb) + co * q / f["rho"]
        if q is w:
            rate = rate + 9.81 * (f["T_g"] - T_AMB) / T_AMB
        out.append(q + rate * DT)
    return out


def _exact_explicit(case, f):
    geo = _Geo(case, f["u"].device)
    u, v, w, T = f["u"], f["v"], f["w"], f["T_g"]
    un, vn, wn = _exact_tentative(f, geo)
    # k-epsilon
    g = {}
    idz = torch.where(torch.arange(case["nz"], device=u.device) == 0, 1.0 / geo.da,
                      1.0 / (geo.db + geo.da))
    idz[-1] = 1.0 / geo.db[-1]
    for n, q, inlet in (("u", u, f["u_inlet"]), ("v", v, torch.zeros_like(f["u_inlet"])),
                        ("w", w, torch.zeros_like(f["u_inlet"]))):
        xL, xR, zL, zR = _neighbours(q, inlet, torch.zeros_like(q[0]))
        g[n] = ((xR - xL) * 0.5 / DX, (_sh(q, 1, 1) - _sh(q, 1, -1)) * 0.5 / DX,
                (zR - zL) * _zvec(idz))
    (ux, uy, uz), (vx, vy, vz), (wx, wy, wz) = g["u"], g["v"], g["w"]
    S2 = 2 * (ux ** 2 + vy ** 2 + wz ** 2) + (uy + vx) ** 2 + (uz + wx) ** 2 + (vz + wy) ** 2
    O2 = (uy - vx) ** 2 + (uz - wx) ** 2 + (vz - wy) ** 2
    KT, ET = f["k_turb"], f["eps_turb"]
    kl, el = KT.clamp(min=1e-8), ET.clamp(min=1e-8)
    U = torch.sqrt(0.5 * (S2 + O2))
    nu = (kl * kl / el / (4.04 + 4.5 * U * kl / el)).clamp(min=0.0)
    P = torch.minimum(nu * S2, 10.0 * el)
    up, dn = _edge(_sh(T, 0, 1), 0, -1, T[-1]), _edge(_sh(T, 0, -1), 0, 0, T[0])
    Gk = ((nu / 0.85) * (9.81 / T.clamp(min=T_AMB)) * (up - dn) * _zvec(idz)).clamp(min=0.0)
    C3 = torch.tanh(w.abs() / torch.sqrt(u * u + v * v).clamp(min=0.01))
    speed = torch.sqrt(u * u + v * v + w * w)
    cds = SAV * f["alpha_s"] * speed
    Pc, Dc = cds * speed * speed, 4.0 * cds * kl
    inlet = torch.full_like(f["u_inlet"], 1e-8)
    wall = torch.full_like(KT[0], 1e-8)
    new = []
    for q, c, a, Sp, Sn in (
            (KT, kl, 1.5e-5 + nu, P + torch.minimum(Gk, P) + Pc, el + Dc),
            (ET, el, 1.5e-5 + nu / 1.3, None, None)):
        nb = list(_neighbours(q, inlet, wall))
        nb[1], nb[3] = _edge(nb[1], 2, -1, c[:, :, -1]), _edge(nb[3], 0, -1, c[-1])
        gx, gy, gz = _grad(q, u, v, w, geo, nb, c)
        if Sp is None:
            eta = torch.sqrt(S2) * kl / el
            rng = (0.09 * eta ** 3 * (1 - eta / 4.38) / (1 + 0.012 * eta ** 3)).clamp(min=0.0)
            Sp = (1.44 * (P + C3 * Gk) + 0.9 * Pc) * el / kl
            Sn = ((1.92 + rng) * el + 0.9 * Dc) * el / kl
        rate = -(u * gx + v * gy + w * gz) + a * _lap(q, geo, nb, c) + Sp
        new.append(((c + rate * DT) / (1.0 + Sn * DT / c)).clamp(min=1e-8))
    k, e = new
    nun = (k * k / e / (4.04 + 4.5 * U * k / e)).clamp(min=0.0)
    # gas temperature
    nb = _neighbours(T, torch.full_like(f["u_inlet"], T_AMB))
    gx, gy, gz = _grad(T, u, v, w, geo, nb)
    rate = -(u * gx + v * gy + w * gz) + 2.0e-5 * _lap(T, geo, nb)
    Tn = (T + rate * DT).clamp(T_AMB, T_CAP)
    return dict(zip(("u", "v", "w", "k", "eps", "nu_t", "T_g"), (un, vn, wn, k, e, nun, Tn)))


def _exact_pressure(case, f):
    geo = _Geo(case, f["u"].device)
    u, v, w = _exact_tentative(f, geo)
    rho = f["rho"]
    tgt = (f["S_pyro"] + f["S_drying"] - (rho - f["rho_prev"]) / DT) / rho.clamp(min=0.1)
    ir = 1.0 / rho.clamp(min=0.01)
    dz = _zvec(geo.dz)
    gx = dz * 0.5 * (ir + _sh(ir, 2, 1)) / DX ** 2
    gx[:, :, -1] = 0.0
    gy = dz * 0.5 * (ir + _sh(ir, 1, 1)) / DX ** 2
    gz = 0.5 * (ir + _sh(ir, 0, 1)) / _zvec(geo.da)
    gz[-1] = 0.0
    e = (-1.0e-6 * dz).expand_as(ir).clone()
    e[:, :, -1] += DZ * 2.0 * ir[:, :, -1] / DX ** 2
    e[-1] += DZ * 2.0 * ir[-1] / DZ ** 2

    def apply(x):
        tx, ty, tz = (x - _sh(x, 2, 1)) * gx, (x - _sh(x, 1, 1)) * gy, (x - _sh(x, 0, 1)) * gz
        return e * x + tx - _sh(tx, 2, -1) + ty - _sh(ty, 1, -1) + tz - _sh(tz, 0, -1)

    div = ((u - _edge(_sh(u, 2, -1), 2, 0, f["u_inlet"])) / DX + (v - _sh(v, 1, -1)) / DX
           + (w - _edge(_sh(w, 0, -1), 0, 0, torch.zeros_like(w[0]))) / dz)
    b = -dz * (div - tgt) / DT
    diag = e + gx + _sh(gx, 2, -1) + gy + _sh(gy, 1, -1) + gz + _sh(gz, 0, -1)
    x, r = torch.zeros_like(b), b.clone()
    z = r / diag
    p, rz, stop = z.clone(), (r * z).sum(), 1e-13 * b.norm()
    for it in range(6000):
        q = apply(p)
        a = rz / (p * q).sum()
        x += a * p
        r -= a * q
        if it % 50 == 49 and r.norm() < stop:
            break
        z = r / diag
        rn = (r * z).sum()
        p = z + (rn / rz) * p
        rz = rn
    out = x[:, :, -1]
    un = u - DT * (_sh(x, 2, 1) - x) / DX * 0.5 * (ir + _sh(ir, 2, 1))
    un[:, :, -1] = u[:, :, -1] + 2.0 * DT * out / DX * ir[:, :, -1]
    vn = v - DT * (_sh(x, 1, 1) - x) / DX * 0.5 * (ir + _sh(ir, 1, 1))
    wn = w - DT * (_sh(x, 0, 1) - x) / _zvec(geo.da) * 0.5 * (ir + _sh(ir, 0, 1))
    wn[-1] = w[-1] + 2.0 * DT * x[-1] / DZ * ir[-1]
    return {"u": un, "v": vn, "w": wn, "p": x, "target": tgt}


def _exact_substep(case, f):
    dev = f["u"].device
    geo = _Geo(case, dev)
    if case["form"] == "mixed":
        for k in ("T_g", "Y_fuel", "Y_O2", "Y_H2O", "rho", "u", "v", "w", "k_turb", "eps_turb",
                  "nu_t", "S_pyro", "S_drying", "Q_g_conv"):
            f[k] = f[k].float().double()
    T, Yf, Yo, Yh, rho = f["T_g"], f["Y_fuel"], f["Y_O2"], f["Y_H2O"], f["rho"]
    # EDC; a cell that does not react sees the quench flag of the last one that did
    react = (Yf > 1e-9) & (Yo > 1e-9)
    damp = (1.0 - Yh / 0.18).clamp(min=0.0)
    code = torch.where(react, 2 * torch.arange(T.numel(), device=dev).view(T.shape)
                       + ((Yh > 0.0) & (damp < 0.5)).long(), -1)
    flag = (torch.cummax(code.flatten(), 0).values.clamp(min=0) % 2 == 1).view(T.shape)
    kt, et = f["k_turb"].clamp(min=1e-4), f["eps_turb"].clamp(min=1e-6)
    gam = (2.1377 ** 3 * (1.5e-5 * et / kt ** 2).clamp(min=1e-30) ** 0.75).clamp(max=1.0)
    om = gam * rho * torch.minimum(Yf, Yo / S_ST) / (0.4083 * torch.sqrt(1.5e-5 / et))
    om = torch.where(react, om * torch.where(Yh > 0.0, damp, torch.ones_like(damp)), 0.0)
    heat = HOC * (1.0 - CHI)
    wet = flag & (T > 373.15) & (Yh > 0.0)
    relax = 1.0 - math.exp(-DT_SUB / 0.5)
    T = torch.where(wet, T - (T - 373.15) * relax * (Yh / 0.10).clamp(max=1.0), T)
    dY = -om * DT_SUB / rho
    Yf, Yo = (Yf + dY).clamp(min=0.0), (Yo + S_ST * dY).clamp(min=0.0)
    T = (T + om * heat * DT_SUB / rho / ((1.0 - Yh) * CP_G + Yh * 2000.0)).clamp(max=2400.0)
    # species with dilution sources
    sp, sd = f["S_pyro"], f["S_drying"]
    Y = []
    for y, inl, src, hi in ((Yf, 0.0, sp, 1.0), (Yo, 0.232, 0.0, 0.232), (Yh, 0.0, sd, 1.0)):
        nb = _neighbours(y, torch.full_like(f["u_inlet"], inl))
        gx, gy, gz = _grad(y, f["u"], f["v"], f["w"], geo, nb)
        rate = (-(f["u"] * gx + f["v"] * gy + f["w"] * gz) + 1.0e-5 * _lap(y, geo, nb)
                + (src - y * (sp + sd)) / rho)
        Y.append((y + rate * DT_SUB).clamp(0.0, hi))

    def diffuse(q, sc, lo, hi):
        nb = _neighbours(q, q[:, :, 0])
        return (q + f["nu_t"] / sc * _lap(q, geo, nb) * DT_SUB).clamp(lo, hi)

    Yf, Yo, Yh = (diffuse(y, SC_T, 0.0, hi) for y, hi in zip(Y, (1.0, 0.232, 1.0)))
    # gas energy, solid conduction
    Ts, a = f["T_s"], f["alpha_s"]
    qc = f["q_rad_gas"] / _zvec(geo.dz)
    qc[:NBED, :, 5:7] += 0.2 * 30000.0 / H_BED
    debit = (sp * (T - Ts).clamp(min=0.0) + sd * (T - 373.15).clamp(min=0.0)) * 2000.0
    cp = (1.0 - Yh) * 1100.0 + Yh * 2000.0
    Tn = (T + (qc - f["Q_g_conv"] - debit) * DT_SUB / (rho.clamp(min=1e-3) * cp)).clamp(min=T_AMB)
    flux = torch.zeros_like(Ts)
    for o, dist, end in ((1, geo.da, -1), (-1, geo.db, 0)):
        an = _edge(_sh(a, 0, o), 0, end, torch.zeros_like(a[0]))
        ok = (a > 0.0) & (an > 0.0)
        ae = torch.where(ok, 2.0 * a * an / (a + an).clamp(min=1e-30), 0.0)
        flux = flux + K_S * ae * (_sh(Ts, 0, o) - Ts) / _zvec(dist)
    dT = torch.where(a > 0.0, DT_SUB * flux / _zvec(geo.dz) / (RHO_S * CP_S) / a.clamp(min=1e-30),
                     0.0)
    return {"T_g": diffuse(Tn, PR_T, T_AMB, T_CAP), "Y_fuel": Yf, "Y_O2": Yo, "Y_H2O": Yh,
            "omega": om, "T_s": (Ts + dT).clamp(T_AMB, T_CAP), "Q_comb": qc}


def _exact_radiation(case, f):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    dev = f["u"].device
    om, wq = level_symmetric(case["order"])
    m = om.shape[0] // 8
    om = torch.tensor(om, device=dev).view(8, m, 3)
    wq = torch.tensor(wq, device=dev).view(8, m)
    ks = SAV * f["alpha_s"] * (1.0 + 5.0 * f["M_local"])
    kg = K_GAS * torch.maximum((f["omega"] / 1e-3).clamp(0.0, 1.0),
                               ((f["T_g"] - 600.0) / 400.0).clamp(0.0, 1.0))
    kg = kg + 30.0 * f["rho"] * f["Y_H2O"]
    kap = (ks + kg).clamp(min=1e-3)
    T4 = torch.where(ks + kg > 1e-9, (ks * f["T_s"] ** 4 + kg * f["T_g"] ** 4) / kap, T_AMB ** 4)
    B = SIGMA * T4 / math.pi
    amb = SIGMA * T_AMB ** 4 / math.pi
    soil = EPS_W * SIGMA * f["T_soil"] ** 4 / math.pi
    ig = soil.clone()
    sign = (om[:, 0] >= 0.0).tolist()
    flips = [[d for d, s in ((2, sx), (1, sy), (0, sz)) if not s] for sx, sy, sz in sign]
    K = torch.stack([kap.flip(d) for d in flips]).view(8, -1)
    E = torch.stack([(kap * B).flip(d) for d in flips]).view(8, -1)
    ax, ay, az = (om[..., q].abs()[:, :, None, None] / h for q, h in ((0, DX), (1, DX), (2, DZ)))
    w4 = wq[:, :, None, None]
    up = torch.tensor([s[2] for s in sign], device=dev)[:, None, None]
    mu = w4[..., 0] * om[..., 2].abs()[:, :, None]
    jj = torch.arange(ny, device=dev)[None, :]
    kk = torch.arange(nz, device=dev)[:, None]
    base = (kk * ny + jj) * nx
    planes = nx + ny + nz - 2
    i = torch.arange(nx, device=dev)
    wrap = torch.zeros((8, m, nz, nx), dtype=torch.float64, device=dev)
    G = torch.zeros((nz, ny, nx), dtype=torch.float64, device=dev)
    at = (i[None, None, :] + jj[..., None] + kk[..., None])  # the plane of each cell
    for it in range(30):
        X = torch.full((8, m, nz, ny), amb, dtype=torch.float64, device=dev)
        S = torch.zeros((planes, 8, nz, ny), dtype=torch.float64, device=dev)
        W = torch.zeros((planes, 8, m, nz), dtype=torch.float64, device=dev)
        Q = torch.zeros((planes, 8, ny), dtype=torch.float64, device=dev)
        igf = torch.stack([ig.flip([d - 1 for d in fl if d > 0]) for fl in flips])
        for d in range(planes):
            ip = d - jj - kk
            act = (ip >= 0) & (ip < nx)
            ic = ip.clamp(0, nx - 1)
            kb, eb = K[:, base + ic][:, None], E[:, base + ic][:, None]
            iy = torch.cat([wrap.gather(3, ic[:, :1].expand(8, m, nz, 1)), X[..., :-1]], 3)
            low = torch.where(up, igf.gather(2, ic[0].view(1, ny, 1).expand(8, ny, 1))[:, None, :, 0],
                              amb)
            iz = torch.cat([low[:, :, None, :].expand(8, m, 1, ny), X[:, :, :-1]], 2)
            v = (eb + ax * X + ay * iy + az * iz) / (kb + ax + ay + az)
            X = torch.where(act, v, X)
            S[d] = (w4 * v).sum(1)
            W[d] = v[..., -1]
            Q[d] = (mu * v[:, :, -1]).sum(1)
        prev, G, qin = G, torch.zeros_like(G), torch.zeros_like(ig)
        for o in range(8):
            G += S[:, o].gather(0, at.permute(2, 0, 1)).permute(1, 2, 0).flip(flips[o])
            edge = (i[:, None] + (ny - 1) + torch.arange(nz, device=dev)[None, :])
            wrap[o] = W[:, o].gather(0, edge[:, None, :].expand(nx, m, nz)).permute(1, 2, 0)
            if not sign[o][2]:
                low = Q[:, o].gather(0, i[:, None] + jj + (nz - 1)).T
                qin += low.flip([d - 1 for d in flips[o] if d > 0])
        ig = RELAX * (soil + (1.0 - EPS_W) / math.pi * qin) + (1.0 - RELAX) * ig
        if it > 0 and float((G - prev).abs().max() / G.max().clamp(min=1e-12)) < TOL:
            break
    net = (ks + kg) * (G - 4.0 * math.pi * B) * DZ
    return {"q_rad": net * ks / kap, "q_rad_gas": net * kg / kap, "q_in_soil": EPS_W * qin}


def exact(case, seed):
    if case["kind"] == "step":
        return None
    f = _fields(case, seed)
    return {"radiation": _exact_radiation, "pressure": _exact_pressure,
            "explicit": _exact_explicit, "substep": _exact_substep}[case["kind"]](case, f)
