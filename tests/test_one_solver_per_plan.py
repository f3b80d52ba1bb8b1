"""Setting a plan's solver: every second jja_plan_set_* call is refused and the first solver's results stay; a
setter that fails leaves the plan, and the device's memory, as they were."""
import ctypes
import itertools

import numpy as np
import pytest

from pyjjasim_gb300 import _native as N
from pyjjasim_gb300 import plan as P
from pyjjasim_gb300.circuit import SquareArray

SOLVERS = ["fast_poisson", "sine", "resident", "blocks", "top"]


def _set(pl, factor, c, solver):
    lib = N.lib()
    if solver in ("fast_poisson", "sine"):
        mx, my, grid, kappa = P.poisson_grid(c, P.face_matrix(c, 0.05)[1])
        pl._keep[solver] = grid
        call = lib.jja_plan_set_fast_poisson if solver == "fast_poisson" else lib.jja_plan_set_sine_solver
        return call(pl.handle, mx, my, N.ptr(grid, ctypes.c_int32), kappa)
    if solver == "resident":
        return lib.jja_plan_set_resident(pl.handle, factor.handle)
    if solver == "blocks":
        return lib.jja_plan_set_blocks(pl.handle, factor.handle, 0)
    return lib.jja_plan_set_top_block(pl.handle, factor.handle, 48)


@pytest.mark.gpu
@pytest.mark.parametrize("first,second", [p for p in itertools.permutations(SOLVERS, 2)])
def test_second_solver_is_refused(first, second):
    import torch
    c = SquareArray(8, 8)      # 49 faces: every solver takes it
    factor, A, _ = P.get_factor(c, 0.05)
    pl = P.DevicePlan(c, factor, A, 3, 0.05, 3, ((1.0, -1.0, 0.0), (1.0, -2.0, 1.0)))
    assert _set(pl, factor, c, first) == 0
    assert _set(pl, factor, c, second) == 1    # JJA_ERR_ARG
    b = np.random.default_rng(3).standard_normal((c._Nf(), 3))
    bd = torch.from_numpy(b).cuda()
    xd = torch.empty_like(bd)
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    pl.solve(bd.data_ptr(), xd.data_ptr(), s.cuda_stream)
    s.synchronize()
    pl.check()
    ref = factor.solve_host(b)
    assert np.abs(xd.cpu().numpy() - ref).max() <= 1e-11 * np.abs(ref).max()


@pytest.mark.gpu
@pytest.mark.parametrize("solver", ["sine", "resident", "blocks", "top"])
def test_a_setter_out_of_memory_leaves_the_plan_as_it_was(solver):
    import torch
    c = SquareArray(150, 140) if solver == "sine" else SquareArray(12, 12) if solver == "resident" else SquareArray(30, 24)
    factor, A, _ = P.get_factor(c, 0.05)
    W = 2
    b = np.random.default_rng(3).standard_normal((c._Nf(), W))
    bd = torch.from_numpy(b).cuda()
    xd = torch.empty_like(bd)
    ref = factor.solve_host(b)
    pl = P.DevicePlan(c, factor, A, W, 0.05, 3, ((1.0, -1.0, 0.0), (1.0, -2.0, 1.0)))
    lib = N.lib()

    def attempt():
        if solver == "top":
            return lib.jja_plan_set_top_block(pl.handle, factor.handle, 200)
        if solver == "blocks":
            return lib.jja_plan_set_blocks(pl.handle, factor.handle, 64)
        return _set(pl, factor, c, solver)

    before = lib.jja_plan_device_bytes(pl.handle)
    for limit in (0, 4000, 60000, 1 << 20):     # at the first allocation, between two, near the last
        assert lib.jja_plan_test_alloc_limit(pl.handle, limit) == 0
        code = attempt()
        if code == 0:
            assert limit > 0
            break
        assert code == 3 and b"out of memory" in lib.jja_last_error()
        assert lib.jja_plan_device_bytes(pl.handle) == before
        pl.solve(bd.data_ptr(), xd.data_ptr(), 0)
        torch.cuda.synchronize()
        assert np.abs(xd.cpu().numpy() - ref).max() <= 1e-11 * np.abs(ref).max(), limit
    else:
        assert lib.jja_plan_test_alloc_limit(pl.handle, -1) == 0
        assert attempt() == 0
    assert lib.jja_plan_device_bytes(pl.handle) > before
    pl.solve(bd.data_ptr(), xd.data_ptr(), 0)
    torch.cuda.synchronize()
    assert np.abs(xd.cpu().numpy() - ref).max() <= 1e-11 * np.abs(ref).max()


@pytest.mark.parametrize("code,message,kept", [(6, "too large", True), (3, "cudaMalloc: out of memory", True),
                                               (1, "factor order != Nf", False), (5, "supernodes", False)])
@pytest.mark.parametrize("solver", ["sine", "resident", "blocks", "top"])
def test_only_a_solver_that_does_not_fit_falls_back(monkeypatch, solver, code, message, kept):
    """The plan keeps its sweeps when the solver's setter says that it does not fit; other errors are raised
    (the library is a fake here)."""
    real = N.lib()

    class Fake:
        def __getattr__(self, name):
            if name in ("jja_plan_create", "jja_plan_destroy"):
                return lambda *a: 0
            if name == "jja_plan_device_bytes":
                return lambda *a: 7
            if name == "jja_last_error":
                return lambda: message.encode()
            if name.startswith("jja_plan_set_"):
                return lambda *a: code
            return getattr(real, name)

    c = SquareArray(8, 8)
    factor, A, _ = P.get_factor(c, 0.05)
    monkeypatch.setattr(N, "lib", lambda: Fake())
    option = {"sine": (7, 7, np.arange(49, dtype=np.int32), 1.0), "resident": True, "blocks": 0, "top": 48}[solver]
    make = lambda: P.DevicePlan(c, factor, A, 1, 0.05, 3, ((1.0, -1.0, 0.0), (1.0, -2.0, 1.0)), **{solver: option})
    if kept:
        pl = make()
        assert not pl.sine and not pl.resident and pl.blocks is None and pl.top is None
    else:
        with pytest.raises(N.JJAError):
            make()
