"""Failure detection mirrored as status codes, driven from host-side inputs
(no GPU fault): non-finite fields, a pressure solve that cannot converge in
its iteration budget, and the learned solve's forced fallback."""
import ctypes as C

import numpy as np
import pytest
import torch

from firewebapp_b200._lib import FireStepError

pytestmark = pytest.mark.gpu


def test_nan_gas_temperature_raises_like_the_reference():
    """spread_3d.py:1927-1932: NaN/Inf in T_g raises RuntimeError at the dt check."""
    from firewebapp_b200.cases import TINY
    from firewebapp_b200.solver import Tier3Solver
    s = Tier3Solver(TINY)
    s.step()
    s.f["T_g"][3, 2, 5] = float("nan")
    with pytest.raises(RuntimeError, match="NaN/Inf"):
        s.step()
    s.close()


@pytest.mark.parametrize("fp32", [0, 1])
def test_dom_non_finite_input_returns_status_2(fp32):
    """NaN temperatures make G non-finite; the path-8 source iteration's
    device-side test reports it as FS_ENONFINITE, and the context stays usable."""
    from test_gpu_kernels import _dom_solves
    import test_gpu_kernels as K
    orig = K.dev
    calls = {"n": 0}

    def poisoned(a, dtype=torch.float64):
        t = orig(a, dtype)
        calls["n"] += 1
        if calls["n"] in (1, 2):  # T_s and T_g of the first solve, every 97th cell
            t.view(-1)[::97] = float("nan")
        return t

    K.dev = poisoned
    try:
        with pytest.raises(FireStepError) as ei:
            _dom_solves(8, fp32, 29, 40, 48, seed=5, calls=1)
    finally:
        K.dev = orig
    assert ei.value.status == 2
    # a clean solve on the same device afterwards works
    out = _dom_solves(8, fp32, 29, 40, 48, seed=5, calls=1)
    assert np.all(np.isfinite(out[0][0]))


def test_projection_iteration_cap_returns_status_3():
    """projection_3d.py:785-790 raises on BiCGSTAB failure; here a solve that
    cannot meet its tolerance within maxiter returns FS_ENOCONV (3)."""
    from firewebapp_b200.cases import TINY
    from firewebapp_b200.solver import Tier3Solver
    s = Tier3Solver(TINY)
    for _ in range(3):
        s.step()
    s.rtol, s.proj_maxiter = 1e-14, 1
    with pytest.raises(FireStepError) as ei:
        s.step()
    assert ei.value.status == 3
    s.close()


def test_learned_stall_falls_back_and_converges():
    """A network switched off (output scale 0) with a strict stall test falls
    back to the V-cycle within the solve and still reaches the tolerance."""
    from firewebapp_b200.cases import TINY
    from firewebapp_b200.learned import fcg_stats, init_params
    from firewebapp_b200.solver import Tier3Solver
    s = Tier3Solver(TINY, form="learned", learned_weights=init_params(2), learned_stall=0.5,
                    learned_max=50)
    s.net.set_output_scale(0.0)
    fell = 0
    for _ in range(5):
        assert s.step()
        st = fcg_stats(s)
        fell += int(st["fell_back"])
        if st["fell_back"]:
            assert st["learned_iters"] >= 3 and st["vcycle_iters"] >= 1
    assert fell >= 1 and fcg_stats(s)["fallbacks_total"] == fell
    s.close()


@pytest.mark.parametrize("kernel", [1, 2])
@pytest.mark.parametrize("fp32", [0, 1])
def test_dom_hand_off_wait_runs_out_with_status_4(fp32, kernel):
    """Path 8's CTAs wait for one another's rows with bounded waits.  With the
    test switch one CTA withholds a row (a fill that nothing else sends), the
    next CTA's wait runs out, the solve returns FS_ETIMEOUT (4) instead of
    hanging, and the same object then solves normally; with either sweep
    kernel (pencil per thread on 29 levels in CTAs of 3 rows, lane column on
    40 levels in CTAs of 4)."""
    from gpu_helpers import Grid, call, dev, host, lib, stream
    from firewebapp_b200._lib import dbl_array, ptr
    from firewebapp_b200.quadrature import level_symmetric
    om, wq = level_symmetric(8)
    nz, ny, nx = (29, 40, 48) if kernel == 1 else (40, 40, 48)
    rng = np.random.default_rng(3)
    g = Grid(nz, ny, nx, 0.5, 0.5, np.full(nz, 0.1))
    h = C.c_void_p()
    call("fs_dom_create", g.ref, om.shape[0], dbl_array(om[:, 0]), dbl_array(om[:, 1]),
         dbl_array(om[:, 2]), dbl_array(wq), 0.5, C.byref(h))
    shape = (nz, ny, nx)
    Ts = dev(300.0 + 900.0 * rng.random(shape) ** 4)
    Tg = dev(300.0 + 1500.0 * rng.random(shape) ** 6)
    a = dev(np.where(rng.random(shape) < 0.3, 0.002 * rng.random(shape), 0.0))
    zero = dev(np.zeros(shape))
    M = dev(0.05 + 0.1 * rng.random(shape))
    rho = dev(np.ones(shape))
    Tsoil = dev(np.full((ny, nx), 300.0))
    qs, qg = torch.zeros_like(Ts), torch.zeros_like(Ts)
    qsoil = torch.zeros((ny, nx), dtype=torch.float64, device="cuda")

    def solve():
        return lib().fs_dom_solve(h, ptr(Ts), ptr(Tg), ptr(a), ptr(zero), 5000.0, 300.0,
                                  ptr(Tsoil), ptr(zero), ptr(rho), ptr(M), ptr(qs), ptr(qg),
                                  ptr(qsoil), stream())
    try:
        if fp32:
            call("fs_dom_set_precision", h, 1)
        call("fs_dom_set_sweep_mode", h, 8, 0)
        call("fs_dom_set_sweep_kernel", h, kernel)
        assert solve() == 0
        assert lib().fs_dom_sweep_kernel(h) == kernel
        call("fs_dom_set_wait_test", h, 5)
        assert solve() == 4
        assert b"gave up" in lib().fs_last_error()
        call("fs_dom_set_wait_test", h, -1)
        assert solve() == 0
        assert np.all(np.isfinite(host(qs))) and np.all(np.isfinite(host(qg)))
    finally:
        lib().fs_dom_destroy(h)


@pytest.mark.parametrize("fp32", [0, 1])
@pytest.mark.parametrize("shape, ctas, threads", [((29, 40, 48), 0, None), ((16, 24, 48), 8, 32),
                                                  ((6, 40, 21), 3, 64)])
def test_dom_register_patch_wait_runs_out_and_leaves_nothing(shape, ctas, threads, fp32):
    """The default sweep kernel's waits end the same way: with a row withheld
    the solve returns FS_ETIMEOUT, twice in a row, and the next solve on that
    handle is a new handle's bit for bit (nothing of the abandoned sweep is
    left in the y-inflow rows or in G).  The second shape's CTAs are one warp
    that loads, sends and takes rows; the third's two warps."""
    from gpu_helpers import Grid, call, dev, host, lib, stream
    from firewebapp_b200._lib import dbl_array, ptr
    from firewebapp_b200.quadrature import level_symmetric
    om, wq = level_symmetric(8)
    nz, ny, nx = shape
    rng = np.random.default_rng(3)
    g = Grid(nz, ny, nx, 0.5, 0.5, np.full(nz, 0.1))
    Ts = dev(300.0 + 900.0 * rng.random(shape) ** 4)
    Tg = dev(300.0 + 1500.0 * rng.random(shape) ** 6)
    a = dev(np.where(rng.random(shape) < 0.3, 0.002 * rng.random(shape), 0.0))
    zero, rho = dev(np.zeros(shape)), dev(np.ones(shape))
    M = dev(0.05 + 0.1 * rng.random(shape))
    Tsoil = dev(np.full((ny, nx), 300.0))
    out = [torch.zeros_like(Ts), torch.zeros_like(Ts), torch.zeros_like(Tsoil)]

    def handle():
        h = C.c_void_p()
        call("fs_dom_create", g.ref, om.shape[0], dbl_array(om[:, 0]), dbl_array(om[:, 1]),
             dbl_array(om[:, 2]), dbl_array(wq), 0.5, C.byref(h))
        if fp32:
            call("fs_dom_set_precision", h, 1)
        call("fs_dom_set_sweep_mode", h, 0, ctas)
        return h

    def solve(h):
        return lib().fs_dom_solve(h, ptr(Ts), ptr(Tg), ptr(a), ptr(zero), 5000.0, 300.0,
                                  ptr(Tsoil), ptr(zero), ptr(rho), ptr(M), ptr(out[0]),
                                  ptr(out[1]), ptr(out[2]), stream())

    h, new = handle(), handle()
    try:
        assert solve(h) == 0
        assert lib().fs_dom_sweep_kernel(h) == 3
        s5 = (C.c_int * 5)()
        call("fs_dom_launch_shape", h, s5)
        assert threads in (None, s5[2]) and s5[0] > 1
        call("fs_dom_set_wait_test", h, 5)
        for _ in range(2):
            assert solve(h) == 4
            assert b"gave up" in lib().fs_last_error()
        call("fs_dom_set_wait_test", h, -1)
        assert solve(h) == 0
        got = [host(q).copy() for q in out]
        assert solve(new) == 0
        assert lib().fs_dom_iterations(h) == lib().fs_dom_iterations(new)
        for x, y in zip(got, out):
            assert np.array_equal(x, host(y))
    finally:
        lib().fs_dom_destroy(h)
        lib().fs_dom_destroy(new)


def test_dom_begin_of_a_new_handle_does_not_wait_for_its_stream():
    """fs_dom_begin queues its work and returns, on a handle's first solve too:
    behind 0.3 s or more of other work on the stream it comes back while that
    is still running, and the solve's results are a second handle's."""
    from gpu_helpers import Grid, call, dev, host, lib
    from firewebapp_b200._lib import dbl_array, ptr
    from firewebapp_b200.quadrature import level_symmetric
    om, wq = level_symmetric(4)
    shape = nz, ny, nx = 20, 24, 64
    rng = np.random.default_rng(5)
    g = Grid(nz, ny, nx, 0.5, 0.5, np.full(nz, 0.1))
    Ts = dev(300.0 + 900.0 * rng.random(shape) ** 4)
    Tg = dev(300.0 + 1500.0 * rng.random(shape) ** 6)
    a = dev(np.where(rng.random(shape) < 0.3, 0.002 * rng.random(shape), 0.0))
    zero, rho, M = dev(np.zeros(shape)), dev(np.ones(shape)), dev(np.full(shape, 0.1))
    Tsoil = dev(np.full((ny, nx), 300.0))
    st = torch.cuda.Stream()

    def handle():
        h = C.c_void_p()
        call("fs_dom_create", g.ref, om.shape[0], dbl_array(om[:, 0]), dbl_array(om[:, 1]),
             dbl_array(om[:, 2]), dbl_array(wq), 0.5, C.byref(h))
        return h

    def solve(h, busy):
        out = [torch.zeros_like(Ts), torch.zeros_like(Ts), torch.zeros_like(Tsoil)]
        torch.cuda.synchronize()
        e = torch.cuda.Event()
        with torch.cuda.stream(st):
            if busy:
                torch.cuda._sleep(600_000_000)  # cycles of at most 1.965 GHz
            e.record()
        call("fs_dom_begin", h, ptr(Ts), ptr(Tg), ptr(a), ptr(zero), 5000.0, 300.0, ptr(Tsoil),
             ptr(zero), ptr(rho), ptr(M), st.cuda_stream)
        running = not e.query()
        call("fs_dom_end", h, ptr(out[0]), ptr(out[1]), ptr(out[2]), st.cuda_stream)
        return [host(q) for q in out], running

    hs = [handle(), handle()]
    try:
        want, _ = solve(hs[0], False)
        got, running = solve(hs[1], True)
        assert running
        for x, y in zip(got, want):
            assert np.array_equal(x, y)
    finally:
        for h in hs:
            lib().fs_dom_destroy(h)


class _Dom:
    """A DOM handle on random fields of a 140 x 120 x 60 grid, S8: 48 MB of its
    own, 275 MB more for the register-patch kernel's first solve and 87 for the
    pencil kernel's."""

    def __init__(self, kernel=0, shape=(60, 120, 140)):
        from gpu_helpers import Grid, call, dev
        from firewebapp_b200._lib import dbl_array
        from firewebapp_b200.quadrature import level_symmetric
        om, wq = level_symmetric(8)
        rng = np.random.default_rng(8)
        nz, ny, nx = shape
        self.g = Grid(nz, ny, nx, 0.5, 0.5, np.full(nz, 0.1))
        self.Ts = dev(300.0 + 900.0 * rng.random(shape) ** 4)
        self.Tg = dev(300.0 + 1500.0 * rng.random(shape) ** 6)
        self.a = dev(np.where(rng.random(shape) < 0.3, 0.002 * rng.random(shape), 0.0))
        self.zero, self.rho = dev(np.zeros(shape)), dev(np.ones(shape))
        self.Tsoil = dev(np.full((ny, nx), 300.0))
        self.out = [torch.zeros_like(q) for q in (self.Ts, self.Ts, self.Tsoil)]
        self.h = C.c_void_p()
        call("fs_dom_create", self.g.ref, om.shape[0], dbl_array(om[:, 0]), dbl_array(om[:, 1]),
             dbl_array(om[:, 2]), dbl_array(wq), 0.5, C.byref(self.h))
        if kernel in (1, 2):
            call("fs_dom_set_sweep_mode", self.h, 8, 0)
        call("fs_dom_set_sweep_kernel", self.h, kernel)

    def solve(self):
        from gpu_helpers import lib, stream
        from firewebapp_b200._lib import ptr
        return lib().fs_dom_solve(self.h, ptr(self.Ts), ptr(self.Tg), ptr(self.a), ptr(self.zero),
                                  5000.0, 300.0, ptr(self.Tsoil), ptr(self.zero), ptr(self.rho),
                                  ptr(self.zero), *(ptr(q) for q in self.out), stream())

    def close(self):
        from gpu_helpers import lib
        lib().fs_dom_destroy(self.h)


def _leave_free(mb):
    """Tensors that hold all of the GPU's memory but some mb MB (untouched)."""
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    held, piece = [], 1 << 36
    while True:
        take = min(torch.cuda.mem_get_info()[0] - (mb << 20), piece)
        if take < (4 << 20):
            return held
        try:
            held.append(torch.empty(take >> 21 << 21, dtype=torch.uint8, device="cuda"))
        except torch.cuda.OutOfMemoryError:
            piece = take // 2


def test_dom_kernel_3_without_its_memory_says_so():
    """The register-patch kernel asked for by number where its layouts cannot be
    had: status 5 and a message about the memory (the shape is one it is built
    for); left automatic, the pencil kernel runs, with its results."""
    from gpu_helpers import host, lib
    small = [_Dom(k, (6, 5, 9)) for k in (1, 3)]
    assert [q.solve() for q in small] == [0, 0]  # both kernels' code is loaded
    asked, auto, pencil = _Dom(3), _Dom(0), _Dom(1)
    held = _leave_free(200)
    try:
        assert asked.solve() == 5
        assert b"out of memory" in lib().fs_last_error()
        assert auto.solve() == 0
        assert lib().fs_dom_sweep_kernel(auto.h) == 1
        held.clear()
        torch.cuda.empty_cache()
        assert asked.solve() == 0 and pencil.solve() == 0
        assert lib().fs_dom_sweep_kernel(asked.h) == 3
        for x, y, z in zip(auto.out, pencil.out, asked.out):
            assert np.array_equal(host(x), host(y)) and np.array_equal(host(x), host(z))
    finally:
        held.clear()
        for q in small + [asked, auto, pencil]:
            q.close()


@pytest.mark.parametrize("mode", [0, 8, 3])
def test_dom_first_solve_without_memory_can_be_repeated(mode):
    """No path's buffers can be had: status 5 each time the solve is tried, the
    handle unresolved, and a solve like a new handle's once there is memory."""
    from gpu_helpers import call, host, lib
    q, new = _Dom(), _Dom()
    for d in (q, new):
        call("fs_dom_set_sweep_mode", d.h, mode, 0)
    held = _leave_free(48)
    try:
        for _ in range(2):
            assert q.solve() == 5
            assert b"out of memory" in lib().fs_last_error()
            assert lib().fs_dom_sweep_mode(q.h) == 0
        held.clear()
        torch.cuda.empty_cache()
        assert q.solve() == 0 and new.solve() == 0
        for x, y in zip(q.out, new.out):
            assert np.array_equal(host(x), host(y))
    finally:
        held.clear()
        q.close()
        new.close()


def test_stencil_status_is_synchronous():
    """fs_stencil_status, kept for programs that check a step with it, returns
    after the work of the default stream has run."""
    from gpu_helpers import lib
    torch.cuda.synchronize()
    e = torch.cuda.Event()
    torch.cuda._sleep(200_000_000)
    e.record()
    assert not e.query()
    assert lib().fs_stencil_status(1) == 0
    assert e.query()


def test_proj_set_precision_without_memory_can_be_repeated():
    """Memory for part of the FP32 form only (49 MB at 140 x 120 x 60, of which the
    finest level's nine arrays take 36 and are the first): status 5 each time,
    and a solve like a new handle's once there is memory."""
    from gpu_helpers import Grid, call, dev, host, lib, stream
    from firewebapp_b200._lib import ptr
    shape = nz, ny, nx = 60, 120, 140
    rng = np.random.default_rng(4)
    g = Grid(nz, ny, nx, 0.5, 0.5, np.full(nz, 0.1))
    rho, u0, v0, w0 = (dev(0.3 + rng.random(shape)) for _ in range(4))
    ui = dev(np.full((nz, ny), 1.0))
    hs = [C.c_void_p(), C.c_void_p()]
    for h in hs:
        call("fs_proj_create", g.ref, C.byref(h))
    held = _leave_free(34)
    try:
        for _ in range(2):
            assert lib().fs_proj_set_precision(hs[0], 1) == 5
            assert b"out of memory" in lib().fs_last_error()
        held.clear()
        torch.cuda.empty_cache()
        got = []
        for h in hs:
            u, v, w = u0.clone(), v0.clone(), w0.clone()
            its = C.c_int()
            call("fs_proj_set_precision", h, 1)
            call("fs_proj_rebuild", h, ptr(rho), stream())
            call("fs_proj_project", h, ptr(u), ptr(v), ptr(w), ptr(ui), None, 0.01, 1e-8, 200,
                 C.byref(its), stream())
            got.append([host(q) for q in (u, v, w)])
        for x, y in zip(*got):
            assert np.array_equal(x, y)
    finally:
        held.clear()
        for h in hs:
            lib().fs_proj_destroy(h)
