"""A plan takes one solver: every second jja_plan_set_* call is refused, and the first solver's results stay."""
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
