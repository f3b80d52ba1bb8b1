"""Tensor-core sine transforms + tridiagonal solve of uniform square arrays (jja_plan_set_sine_solver).

Against scipy's sparse direct solve at the edges of its tiles: sides around the multiples of 16
and 32 that the folded transforms are padded to, one face, odd and even sides, column counts
around the 128 of a tile, transforms along x and along y. Both solvers are backward stable, so
they differ by a small multiple of the condition number times the FP64 rounding; the condition
number of the Dirichlet Laplacian of n faces a side is below (n + 1)^2, 1.7e4 at 128, which gives
the bar 1e-11 that the other face solves of this package are held to."""
import numpy as np
import pytest
import scipy.sparse.linalg

from oracle import rcsj_oracle
from pyjjasim_gb300 import TimeEvolutionProblem, backend
from pyjjasim_gb300 import plan as P
from pyjjasim_gb300.circuit import HoneycombArray, SquareArray


def test_rule_takes_only_uniform_grids():
    c = SquareArray(20, 31)
    assert P.poisson_grid(c, P.face_matrix(c, 0.05)[1])[:2] == (19, 30)
    c.set_resistance(np.random.default_rng(0).uniform(1, 2, c.junction_count()))
    assert P.poisson_grid(c, P.face_matrix(c, 0.05)[1]) is None
    c = HoneycombArray(8, 8)
    assert P.poisson_grid(c, P.face_matrix(c, 0.05)[1]) is None
    assert P.untuned(None) and P.untuned({"schedule": 1}) and not P.untuned({"schedule": 2})
    assert not P.untuned({"subtree_rows": -1})


def _solve(c, b, sine):
    A, K = P.face_matrix(c, 0.05)
    factor, A, _ = P.get_factor(c, 0.05)
    st = (1.0, -1.0, 0.0), (1.0, -2.0, 1.0)
    pl = P.DevicePlan(c, factor, A, b.shape[1], 0.05, 3, st, sine=P.poisson_grid(c, K) if sine else None)
    import torch
    bd = torch.from_numpy(b).cuda()
    xd = torch.empty_like(bd)
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    pl.solve(bd.data_ptr(), xd.data_ptr(), s.cuda_stream)
    s.synchronize()
    pl.check()
    return xd.cpu().numpy(), K


SIZES = [(2, 2, 1), (2, 9, 3), (3, 4, 2), (18, 33, 7), (33, 34, 128), (34, 17, 129), (64, 64, 5), (66, 65, 33),
         (96, 97, 40), (98, 99, 2), (128, 128, 3), (129, 128, 65), (129, 300, 2), (300, 129, 2), (101, 60, 24),
         # both sides longer than 128 faces: strips of one and two widths, one and several separators
         (131, 130, 2), (130, 131, 17), (257, 257, 1), (140, 400, 3), (390, 135, 2), (300, 300, 5), (131, 131, 260),
         # more tiles than blocks, a last wave of half tiles
         (128, 128, 160), (40, 35, 610), (20, 33, 1300)]


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,W", SIZES)
def test_solve_matches_scipy(nx, ny, W):
    c = SquareArray(nx, ny)
    c.set_inductance(0.07)
    c.set_capacitance(0.3)
    rng = np.random.default_rng(nx + W)
    Nf = c._Nf()
    b = rng.standard_normal((Nf, W)) * 10.0 ** rng.uniform(-12, 12, (1, W))   # every problem its own scale
    b[:, 0] = 1.0                                                             # equal digits in every element
    if W > 1:
        b[:, 1] = 0.0
    x, K = _solve(c, b, True)
    ref = scipy.sparse.linalg.spsolve(K.tocsc(), b).reshape(x.shape)
    err = np.abs(x - ref).max(0) / np.maximum(np.abs(ref).max(0), 1e-300)
    assert float(err.max()) <= 1e-11, err.argmax()
    y, _ = _solve(c, b, False)
    # residuals against the sweeps': as accurate as the solve it stands in for
    rx, ry = (np.linalg.norm(K @ v - b, axis=0) / np.maximum(np.linalg.norm(b, axis=0), 1e-300) for v in (x, y))
    print(f"{nx}x{ny} W={W}: residual {rx.max():.2e}, sweeps {ry.max():.2e}")
    assert rx.max() <= max(4.0 * ry.max(), 1e-13)


@pytest.mark.gpu
def test_non_finite_values_stay_in_their_problem():
    c = SquareArray(40, 33)
    b = np.random.default_rng(1).standard_normal((c._Nf(), 6))
    good = _solve(c, b, True)[0]
    b[17, 2], b[900, 4] = np.nan, np.inf
    x = _solve(c, b, True)[0]
    assert not np.isfinite(x[:, [2, 4]]).all(0).any()
    np.testing.assert_array_equal(x[:, [0, 1, 3, 5]], good[:, [0, 1, 3, 5]])


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,W,width", [(60, 70, 64, 3), (40, 130, 40, 4), (25, 30, 300, 3), (150, 140, 3, 3)])
def test_trajectory_matches_sweeps_and_oracle(nx, ny, W, width):
    c = SquareArray(nx, ny)
    c.set_capacitance(0.4)
    c.set_inductance(0.1)
    Is = c.current_base(0.0)[:, None, None] * np.linspace(0.4, 1.6, W)[None, :, None]
    prob = TimeEvolutionProblem(c, time_step=0.05, time_step_count=120, current_sources=Is, external_flux=0.13,
                                store_time_steps=np.arange(0, 120, 25), stencil_width=width)
    m = prob.store_time_steps
    assert backend.GpuSimulation(prob).plan.sine
    th, I = backend.time_evolution_core(prob, m, m)
    th_s, I_s = backend.time_evolution_core(prob, m, m, fast_poisson=False)
    th_o, I_o = rcsj_oracle.evolve(prob, m, m)
    scale = max(1.0, float(np.abs(th_o).max()))
    assert float(np.abs(th - th_s).max()) <= 1e-10 * scale
    assert float(np.abs(th - th_o).max()) <= 1e-9 * scale
    assert float(np.abs(I - I_o).max()) <= 1e-9
