"""Whole runs of small circuits in one launch (jja_plan_set_resident) against the oracle and the sweeps.

The trajectory bars are those of the other paths (1e-9 relative against the oracle, 1e-10 between
solvers); the product's error bound stands in csrc/jja_resident.cuh, its size beside the sweeps' is tested here."""
import numpy as np
import pytest

from oracle import rcsj_oracle
from pyjjasim_gb300 import TimeEvolutionProblem, backend
from pyjjasim_gb300 import plan as P
from pyjjasim_gb300.circuit import HoneycombArray, SquareArray, TriangularArray


def test_rule():
    assert P.resident_fits(SquareArray(10, 10), 1) and P.resident_fits(SquareArray(13, 13), P.RESIDENT_MAX_W)
    assert not P.resident_fits(SquareArray(10, 10), P.RESIDENT_MAX_W + 1)
    assert not P.resident_fits(SquareArray(14, 14), 1)


CASES = [(SquareArray, 2, 2, 1, 3), (SquareArray, 2, 5, 3, 4), (SquareArray, 9, 5, 1, 3),    # 1, 4 and 32 faces
         (SquareArray, 12, 4, 2, 5), (SquareArray, 10, 10, 5, 3), (SquareArray, 9, 17, 2, 4),  # 33, 81, 128 faces
         (SquareArray, 9, 21, 1, 3), (HoneycombArray, 4, 4, 7, 3), (TriangularArray, 5, 4, 3, 5)]   # 160 faces


@pytest.mark.gpu
@pytest.mark.parametrize("lattice,nx,ny,W,width", CASES)
@pytest.mark.parametrize("sources", ["constant", "timedep"])
def test_trajectory(lattice, nx, ny, W, width, sources):
    c = lattice(nx, ny)
    rng = np.random.default_rng(nx * ny + W)
    c.set_resistance(rng.uniform(0.8, 1.3, c._Nj()))
    c.set_critical_current(rng.uniform(0.5, 1.5, c._Nj()))
    if width > 3:
        c.set_capacitance(0.6)
    c.set_inductance(0.1)
    Nt = 60
    Is = rng.uniform(-0.6, 0.6, (c._Nj(), W, 1))
    f, kw = rng.uniform(-0.4, 0.4, (c._Nf(), W, 1)), {}
    if sources == "timedep":
        Is = Is * np.sin(0.1 * np.arange(Nt))
        f = lambda i: 0.01 * i
        kw = dict(voltage_sources=rng.uniform(-0.2, 0.2, (c._Nj(), 1, 1)))
    prob = TimeEvolutionProblem(c, time_step=0.05, time_step_count=Nt, current_sources=Is, external_flux=f,
                                store_time_steps=[0, 7, 8, 9, 30, Nt - 1], stencil_width=width,
                                config_at_minus_1=rng.uniform(-1, 1, (c._Nj(), W)), **kw)
    m, mI = prob.store_time_steps, np.arange(Nt) % 3 == 0
    sim = backend.GpuSimulation(prob)
    assert sim.plan.resident
    th, I = backend.time_evolution_core(prob, m, mI, sim=sim)
    th_s, I_s = backend.time_evolution_core(prob, m, mI, fast_poisson=False)
    th_o, I_o = rcsj_oracle.evolve(prob, m, mI)
    scale = max(1.0, float(np.abs(th_o).max()))
    assert float(np.abs(th - th_s).max()) <= 1e-10 * scale and float(np.abs(I - I_s).max()) <= 1e-9
    assert float(np.abs(th - th_o).max()) <= 1e-9 * scale and float(np.abs(I - I_o).max()) <= 1e-9


@pytest.mark.gpu
def test_calls_chain_and_noise_is_the_same_as_step_by_step():
    c = SquareArray(8, 7)
    W, Nt = 4, 50
    Is = c.current_base(0.0)[:, None, None] * np.linspace(0.3, 1.4, W)[None, :, None]
    prob = TimeEvolutionProblem(c, time_step=0.05, time_step_count=Nt, current_sources=Is, external_flux=0.1,
                                temperature=0.05)
    import torch
    a, b = backend.GpuSimulation(prob, seed=5), backend.GpuSimulation(prob, seed=5, fast_poisson=False)
    assert a.plan.resident and not b.plan.resident
    for n in (1, 7, 20, 3):
        a.run(n)
        b.run(n)
    all_a = torch.empty((19, c._Nj(), W), dtype=torch.float64, device="cuda")
    all_b = torch.empty_like(all_a)
    a.run(19, None, None, all_a, None, store_all=True)
    b.run(19, None, None, all_b, None, store_all=True)
    a.synchronize()
    b.synchronize()
    assert float((all_a - all_b).abs().max()) <= 1e-10
    for x, y in zip(a.history(), b.history()):
        assert float((x - y).abs().max()) <= 1e-10


@pytest.mark.gpu
def test_non_finite_phases_are_reported():
    from pyjjasim_gb300 import _native as N
    c = SquareArray(6, 6)
    Is = np.zeros((c._Nj(), 2, 1))
    Is[3, 1] = np.nan
    prob = TimeEvolutionProblem(c, time_step=0.05, time_step_count=5, current_sources=Is, external_flux=0.1)
    sim = backend.GpuSimulation(prob)
    assert sim.plan.resident
    sim.run(5)
    with pytest.raises(N.JJAError):
        sim.synchronize()
    sim.synchronize()   # reported once


# faces, junctions, width, fits: both sides of the 227 KB of shared memory, which the history shares
LIMITS = [(41, 5, 3, True), (41, 5, 4, True), (41, 5, 5, False), (81, 3, 5, False), (54, 4, 5, True), (80, 3, 5, True)]


@pytest.mark.parametrize("nx,ny,width,fits", LIMITS)
def test_rule_counts_the_history(nx, ny, width, fits):
    for c in (SquareArray(nx, ny), SquareArray(ny, nx)):
        assert P.resident_fits(c, 1, width) == fits


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,width,fits", LIMITS)
def test_default_plan_at_the_limit(nx, ny, width, fits):
    c = SquareArray(nx, ny)
    c.set_capacitance(0.6)
    Is = c.current_base(0.0)[:, None, None] * np.linspace(0.4, 1.4, 2)[None, :, None]
    prob = TimeEvolutionProblem(c, time_step=0.05, time_step_count=30, current_sources=Is, external_flux=0.13,
                                store_time_steps=[10, 29], stencil_width=width)
    m = prob.store_time_steps
    sim = backend.GpuSimulation(prob)
    assert sim.plan.resident == fits
    th, _ = backend.time_evolution_core(prob, m, m, sim=sim)
    th_o, _ = rcsj_oracle.evolve(prob, m, m)
    assert float(np.abs(th - th_o).max()) <= 1e-9 * max(1.0, float(np.abs(th_o).max()))


@pytest.mark.gpu
@pytest.mark.parametrize("lattice,nx,ny", [(SquareArray, 10, 10), (SquareArray, 13, 13), (HoneycombArray, 4, 4),
                                           (TriangularArray, 6, 6)])
@pytest.mark.parametrize("sigma", [0.0, 0.4, 0.7])
def test_steps_are_as_accurate_as_the_sweeps(lattice, nx, ny, sigma):
    """One step of random phases against extended precision, for junctions of a lognormal spread of resistances:
    over all junctions and problems (rms) no further off than the sweeps. Width 3 without capacitance:
    theta = A^T K^-1 (A q - 2 pi f) / c0 - q, c0 q = Ic sin(2 th1 - th2) - Is - c0 th1."""
    c = lattice(nx, ny)
    rng = np.random.default_rng(nx + int(10 * sigma))
    R, W = rng.lognormal(0.0, sigma, c._Nj()), 64
    c.set_resistance(R)
    th1, th2 = rng.uniform(-3.0, 3.0, (2, c._Nj(), W))
    Is = rng.uniform(-1.0, 1.0, (c._Nj(), W))
    prob = TimeEvolutionProblem(c, time_step=0.05, time_step_count=1, current_sources=Is[:, :, None], external_flux=0.1,
                                config_at_minus_1=th1, config_at_minus_2=th2)
    A, K = P.face_matrix(c, 0.05)
    ld = np.longdouble
    c0 = (1.0 / (0.05 * R))[:, None].astype(ld)
    q = (np.sin(2.0 * th1.astype(ld) - th2.astype(ld)) - Is) / c0 - th1
    A, K = A.toarray().astype(ld), K.toarray()
    b, x = A @ q - 2.0 * ld(np.pi) * ld(0.1), 0.0
    for _ in range(5):
        x = x + np.linalg.solve(K, (b - K.astype(ld) @ x if np.ndim(x) else b).astype(np.float64))
    exact = (A.T @ x) / c0 - q
    rms = []
    for fast_poisson in ("auto", False):
        sim = backend.GpuSimulation(prob, fast_poisson=fast_poisson)
        assert sim.plan.resident == (fast_poisson == "auto")
        sim.run(1)
        sim.synchronize()
        rms.append(float(np.sqrt(((sim.theta().cpu().numpy() - exact) ** 2).mean())))
    print(f"step: {rms[0]:.2e}, sweeps {rms[1]:.2e}")
    assert rms[0] <= rms[1]


@pytest.mark.gpu
@pytest.mark.parametrize("steps", [50, 60000])
def test_output_slots_are_read_before_the_call_returns(steps):
    """The caller may reuse its slot arrays at once, also while earlier steps are still running."""
    import torch
    c = SquareArray(4, 4)
    prob = TimeEvolutionProblem(c, time_step=0.05, time_step_count=200000, external_flux=0.1,
                                current_sources=0.5 * c.current_base(0.0)[:, None, None])
    want = None
    for overwrite in (False, True):
        sim = backend.GpuSimulation(prob)
        assert sim.plan.resident
        out = torch.zeros((5, c._Nj(), 1), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        slots = np.full(steps, -1, np.int64)
        slots[::steps // 5] = np.arange(5)
        sim.run(100000)          # a quarter of a second of steps before them
        sim.run(steps, th_slot=slots, th_dev=out)
        if overwrite:
            slots[:] = -1
        sim.synchronize()
        want = out.clone() if want is None else want
        assert torch.equal(out, want) and float(out.abs().min(dim=1).values.max()) > 0.0
