"""Face solves by dense blocks on the tensor cores (jja_plan_set_blocks) against scipy and the sweeps.

Sizes around its blocks of 128 x 64 entries and tiles of 16 to 64 problems. The bar against scipy is
the one of the other face solves (1e-11 of the largest value per problem); residuals are compared with
the triangular sweeps', which the blocks stand in for."""
import numpy as np
import pytest
import scipy.sparse.linalg

from oracle import rcsj_oracle
from pyjjasim_gb300 import TimeEvolutionProblem, backend
from pyjjasim_gb300 import plan as P
from pyjjasim_gb300.circuit import HoneycombArray, SquareArray, TriangularArray


def test_rule():
    assert P.block_leaf(HoneycombArray(24, 24), 61) == 0
    assert P.block_leaf(HoneycombArray(24, 24), 700) == 256
    c = SquareArray(230, 200)
    assert P.block_leaf(c, 8) == 384 and P.block_leaf(c, 4) is None and P.top_leaf(c, 4) == 3072
    assert P.block_leaf(c, 512) is None and P.block_leaf(TriangularArray(64, 48), 2048) is None
    c.components = 20
    assert P.top_leaf(c, 1) == 384


def _solve(c, b, leaf, top=None):
    import torch
    A, K = P.face_matrix(c, 0.05)
    factor, A, _ = P.get_factor(c, 0.05)
    pl = P.DevicePlan(c, factor, A, b.shape[1], 0.05, 3, ((1.0, -1.0, 0.0), (1.0, -2.0, 1.0)), blocks=leaf, top=top)
    assert (pl.blocks, pl.top) == (leaf, top)
    bd = torch.from_numpy(b).cuda()
    xd = torch.empty_like(bd)
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    pl.solve(bd.data_ptr(), xd.data_ptr(), s.cuda_stream)
    s.synchronize()
    pl.check()
    return xd.cpu().numpy(), K


@pytest.mark.gpu
@pytest.mark.parametrize("lattice,nx,ny,W,leaf", [
    (SquareArray, 2, 2, 1, 0), (SquareArray, 9, 9, 16, 0), (SquareArray, 14, 6, 17, 0), (SquareArray, 17, 9, 48, 0),
    (SquareArray, 44, 4, 49, 0), (SquareArray, 14, 15, 64, 0), (HoneycombArray, 12, 12, 65, 0),
    (TriangularArray, 10, 9, 15, 0), (TriangularArray, 24, 21, 130, 0), (HoneycombArray, 40, 40, 3, 0),
    (SquareArray, 9, 9, 5, 8), (SquareArray, 40, 33, 33, 64), (HoneycombArray, 30, 24, 61, 200),
    (TriangularArray, 40, 30, 20, 448), (SquareArray, 90, 70, 2, 300), (SquareArray, 12, 12, 3, 4000)])
def test_solve_matches_scipy(lattice, nx, ny, W, leaf):
    c = lattice(nx, ny)
    rng = np.random.default_rng(nx * ny + W)
    c.set_resistance(rng.lognormal(0.0, 0.4, c._Nj()))
    c.set_inductance(0.05)
    Nf = c._Nf()
    b = rng.standard_normal((Nf, W)) * 10.0 ** rng.uniform(-12, 12, (1, W))
    b[:, 0] = 1.0
    if W > 1:
        b[:, 1] = 0.0
    x, K = _solve(c, b, leaf)
    ref = scipy.sparse.linalg.spsolve(K.tocsc(), b).reshape(x.shape)
    err = np.abs(x - ref).max(0) / np.maximum(np.abs(ref).max(0), 1e-300)
    assert float(err.max()) <= 1e-11, err.argmax()
    y, _ = _solve(c, b, None)
    rx, ry = (np.linalg.norm(K @ v - b, axis=0) / np.maximum(np.linalg.norm(b, axis=0), 1e-300) for v in (x, y))
    print(f"Nf={Nf} W={W}: residual {rx.max():.2e}, sweeps {ry.max():.2e}")
    assert rx.max() <= max(4.0 * ry.max(), 1e-13)


@pytest.mark.gpu
@pytest.mark.parametrize("lattice,nx,ny,W,top", [(SquareArray, 9, 9, 1, 4), (SquareArray, 60, 55, 1, 300),
                                                 (TriangularArray, 30, 24, 3, 500), (HoneycombArray, 30, 24, 40, 128),
                                                 (SquareArray, 90, 70, 17, 1000), (SquareArray, 12, 12, 2, 4000), (TriangularArray, 25, 22, 300, 768)])
def test_top_block_matches_scipy(lattice, nx, ny, W, top):
    c = lattice(nx, ny)
    rng = np.random.default_rng(nx * ny + W)
    c.set_resistance(rng.lognormal(0.0, 0.4, c._Nj()))
    b = rng.standard_normal((c._Nf(), W)) * 10.0 ** rng.uniform(-12, 12, (1, W))
    x, K = _solve(c, b, None, top)
    ref = scipy.sparse.linalg.spsolve(K.tocsc(), b).reshape(x.shape)
    err = np.abs(x - ref).max(0) / np.maximum(np.abs(ref).max(0), 1e-300)
    assert float(err.max()) <= 1e-11, err.argmax()
    y, _ = _solve(c, b, None)
    rx, ry = (np.linalg.norm(K @ v - b, axis=0) / np.linalg.norm(b, axis=0) for v in (x, y))
    assert rx.max() <= max(4.0 * ry.max(), 1e-13)


@pytest.mark.gpu
def test_non_finite_values_stay_in_their_problem():
    c = HoneycombArray(14, 13)
    b = np.random.default_rng(1).standard_normal((c._Nf(), 20))
    good = _solve(c, b, 0)[0]
    b[17, 2], b[200, 4] = np.nan, np.inf
    x = _solve(c, b, 0)[0]
    rest = [w for w in range(20) if w not in (2, 4)]
    assert np.isnan(x[:, [2, 4]]).all()
    np.testing.assert_allclose(x[:, rest], good[:, rest], rtol=1e-13, atol=1e-15 * np.abs(good).max())


@pytest.mark.gpu
@pytest.mark.parametrize("lattice,nx,ny,W,width", [(HoneycombArray, 16, 12, 33, 3), (TriangularArray, 15, 14, 5, 4)])
def test_trajectory_matches_sweeps_and_oracle(lattice, nx, ny, W, width):
    c = lattice(nx, ny)
    c.set_capacitance(0.4)
    Is = c.current_base(0.0)[:, None, None] * np.linspace(0.4, 1.4, W)[None, :, None]
    prob = TimeEvolutionProblem(c, time_step=0.05, time_step_count=120, current_sources=Is, external_flux=0.13,
                                store_time_steps=np.arange(0, 120, 25), stencil_width=width)
    m = prob.store_time_steps
    assert backend.GpuSimulation(prob).plan.blocks is not None
    th, I = backend.time_evolution_core(prob, m, m)
    th_s, I_s = backend.time_evolution_core(prob, m, m, fast_poisson=False)
    th_o, I_o = rcsj_oracle.evolve(prob, m, m)
    scale = max(1.0, float(np.abs(th_o).max()))
    assert float(np.abs(th - th_s).max()) <= 1e-10 * scale
    assert float(np.abs(th - th_o).max()) <= 1e-9 * scale
    assert float(np.abs(I - I_o).max()) <= 1e-9


@pytest.mark.gpu
def test_too_many_blocks_keep_the_sweeps():
    """More blocks than the limit (131 x 261 of one inverse): the plan solves by its sweeps, as without blocks."""
    import torch
    c = SquareArray(130, 130)
    c.set_resistance(np.random.default_rng(0).lognormal(0.0, 0.2, c._Nj()))
    A, K = P.face_matrix(c, 0.05)
    factor, A, _ = P.get_factor(c, 0.05)
    pl = P.DevicePlan(c, factor, A, 2, 0.05, 3, ((1.0, -1.0, 0.0), (1.0, -2.0, 1.0)), blocks=0)
    assert pl.blocks is None
    b = np.random.default_rng(1).standard_normal((c._Nf(), 2))
    bd = torch.from_numpy(b).cuda()
    xd = torch.empty_like(bd)
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    pl.solve(bd.data_ptr(), xd.data_ptr(), s.cuda_stream)
    s.synchronize()
    ref = scipy.sparse.linalg.spsolve(K.tocsc(), b)
    assert np.abs(xd.cpu().numpy() - ref).max() <= 1e-11 * np.abs(ref).max()


@pytest.mark.gpu
@pytest.mark.parametrize("top,taken", [(8, False), (16, False), (64, True)])
def test_top_block_does_not_cut_a_fused_subtree(top, taken):
    """Supernodes that the sweeps solve inside a fused subtree (up to 32 rows) cannot go to the product."""
    import torch
    c = SquareArray(60, 55)
    c.set_resistance(np.random.default_rng(0).lognormal(0.0, 0.4, c._Nj()))
    W, tuning = 64, dict(subtree_rows=32)
    factor, A, _ = P.get_factor(c, 0.05)
    assert factor.schedule_stats(W, tuning)["n_subtrees"] > 0
    pl = P.DevicePlan(c, factor, A, W, 0.05, 3, ((1.0, -1.0, 0.0), (1.0, -2.0, 1.0)), tuning=tuning, top=top)
    assert (pl.top is not None) == taken
    b = np.random.default_rng(1).standard_normal((c._Nf(), W))
    bd = torch.from_numpy(b).cuda()
    xd = torch.empty_like(bd)
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    pl.solve(bd.data_ptr(), xd.data_ptr(), s.cuda_stream)
    s.synchronize()
    ref = scipy.sparse.linalg.spsolve(P.face_matrix(c, 0.05)[1].tocsc(), b)
    assert np.abs(xd.cpu().numpy() - ref).max() <= 1e-11 * np.abs(ref).max()


def _exact(K, b):
    """K^-1 b in extended precision (refined with long double residuals)."""
    K = scipy.sparse.csr_matrix(K)
    lu, val, x = scipy.sparse.linalg.splu(K.tocsc()), K.data.astype(np.longdouble)[:, None], np.zeros(b.shape, np.longdouble)
    for _ in range(5):
        r = b.astype(np.longdouble) - np.add.reduceat(val * x[K.indices], K.indptr[:-1], axis=0)
        x = x + lu.solve(r.astype(np.float64))
    return x


@pytest.mark.gpu
@pytest.mark.parametrize("lattice,nx,ny,leaf,top", [(HoneycombArray, 24, 24, 0, None), (TriangularArray, 24, 22, 0, None),
                                                    (TriangularArray, 24, 22, 256, None), (SquareArray, 64, 64, 256, None),
                                                    (SquareArray, 90, 70, None, 768)])
@pytest.mark.parametrize("sigma", [0.0, 0.2, 0.4, 1.0])
def test_phase_increments_are_as_accurate_as_the_sweeps(lattice, nx, ny, leaf, top, sigma):
    """The increments A^T x / c0 of a step of random phases against extended precision, for junctions of a lognormal
    spread of resistances: over all of them (rms) no further off than the sweeps', but for 5 % that the order of
    the atomic sums of either may move."""
    c = lattice(nx, ny)
    rng = np.random.default_rng(nx + int(10 * sigma))
    R = rng.lognormal(0.0, sigma, c._Nj())
    c.set_resistance(R)
    W, c0 = 64, (1.0 / (0.05 * R))[:, None]
    th = rng.uniform(-3.0, 3.0, (c._Nj(), W))
    A, K = P.face_matrix(c, 0.05)
    b = np.ascontiguousarray(A @ ((np.sin(th) - rng.uniform(-1.0, 1.0, th.shape)) / c0 - th) - 0.2 * np.pi)
    exact = _exact(K, b)
    x, _ = _solve(c, b, leaf, top)
    y, _ = _solve(c, b, None)
    rms = [float(np.sqrt((((A.T @ (v - exact).astype(np.float64)) / c0) ** 2).mean())) for v in (x, y)]
    print(f"increments: {rms[0]:.2e}, sweeps {rms[1]:.2e}")
    assert rms[0] <= 1.05 * rms[1]


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,W,top", [(262, 262, 2, 24576), (240, 235, 3, 12288)])
def test_top_block_over_large_subtrees(nx, ny, W, top):
    c = SquareArray(nx, ny)
    rng = np.random.default_rng(nx)
    c.set_resistance(rng.lognormal(0.0, 0.2, c._Nj()))
    b = rng.standard_normal((c._Nf(), W))
    x, K = _solve(c, b, None, top)
    ref = scipy.sparse.linalg.spsolve(K.tocsc(), b)
    assert np.abs(x - ref).max() <= 1e-11 * np.abs(ref).max()
