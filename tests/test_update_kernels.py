"""The usual-step kernels (k_update_fast, k_face_rhs_fast) against the general ones.

A run that stores every step takes the general update kernel, one that stores none the fast one,
both on the same plan: odd and even problem counts (one or two problems per thread), with and
without capacitance, Philox noise, currents, per-problem critical currents and flux. The two
differ in the order of at most two roundings per junction and step, which 40 steps of these
subcritical arrays do not amplify beyond a few hundred units in the last place: 1e-12."""
import numpy as np
import pytest

from pyjjasim_gb300 import TimeEvolutionProblem, backend
from pyjjasim_gb300.circuit import HoneycombArray, SquareArray, TriangularArray


@pytest.mark.gpu
@pytest.mark.parametrize("W", [1, 2, 3, 32, 34, 65])
@pytest.mark.parametrize("C,T,driven,per_w,flux", [(0.0, 0.0, True, False, "face"), (0.5, 0.0, True, True, "all"),
                                                   (0.0, 0.02, True, True, "none"), (0.5, 0.02, False, False, "w")])
def test_fast_steps_match_general_steps(W, C, T, driven, per_w, flux):
    import torch
    c = HoneycombArray(9, 8) if W % 2 else SquareArray(15, 14)
    rng = np.random.default_rng(W)
    c.set_capacitance(C)
    c.set_resistance(rng.uniform(0.8, 1.2, c._Nj()))     # the sweeps solve: no special solver
    Nj, Nf, n = c._Nj(), c._Nf(), 40
    f = {"face": rng.uniform(-0.3, 0.3, (Nf, 1, 1)), "all": rng.uniform(-0.3, 0.3, (Nf, W, 1)), "none": 0.0,
         "w": rng.uniform(-0.3, 0.3, (1, W, 1))}[flux]
    Is = c.current_base(0.0)[:, None, None] * rng.uniform(0.1, 0.6, (1, W, 1)) if driven else 0.0
    prob = TimeEvolutionProblem(c, time_step=0.05, time_step_count=n, current_sources=Is, external_flux=f,
                                temperature=T)
    Ic = rng.uniform(0.7, 1.3, (Nj, W)) if per_w else None
    a, b = (backend.GpuSimulation(prob, seed=9, Ic=Ic, fast_poisson=False) for _ in range(2))
    th = torch.empty((n, Nj, W), dtype=torch.float64, device="cuda")
    cur = torch.empty_like(th)
    a.run(n)
    a.synchronize()
    b.run(n, np.arange(n), np.arange(n), th, cur)
    b.synchronize()
    for x, y in zip(a.history(), b.history()):
        assert float((x - y).abs().max()) <= 1e-12 * max(1.0, float(y.abs().max()))
    assert torch.equal(th[-1], b.theta())


@pytest.mark.gpu
@pytest.mark.parametrize("lattice", [TriangularArray, SquareArray, HoneycombArray])
@pytest.mark.parametrize("W", [1, 34])
def test_face_sums_of_each_degree(lattice, W):
    """The fast face kernel (flux constant in time) against the general one (the same flux as a function of time):
    the same operations in the same order."""
    import torch
    c = lattice(14, 11)
    c.set_resistance(np.random.default_rng(W).uniform(0.8, 1.2, c._Nj()))
    f = np.random.default_rng(W).uniform(-0.3, 0.3, (c._Nf(), W, 1))
    out = []
    for flux in (f, lambda i: f[:, :, 0]):
        prob = TimeEvolutionProblem(c, time_step=0.05, time_step_count=20, external_flux=flux,
                                    current_sources=0.3 * np.ones((c._Nj(), W, 1)))
        sim = backend.GpuSimulation(prob, fast_poisson=False)
        sim.run(20)
        sim.synchronize()
        out.append(sim.theta().clone())
    assert float((out[0] - out[1]).abs().max()) <= 1e-13


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,W,per_face", [(4, 4, 1, True), (16, 32, 1, False), (32, 8, 2, True), (64, 32, 3, True),
                                              (64, 64, 8, False), (256, 64, 1, True), (32, 32, 9, True)])
def test_face_sums_in_the_first_transform(nx, ny, W, per_face):
    """Radix-2 plans form the face sums in their first transform, except in timed runs (and beyond 8 problems): the
    same operations in the same order."""
    import torch
    c = SquareArray(nx, ny)
    rng = np.random.default_rng(nx + W)
    f = rng.uniform(-0.3, 0.3, (c._Nf(), W, 1)) if per_face else rng.uniform(-0.3, 0.3, (1, W, 1))
    prob = TimeEvolutionProblem(c, time_step=0.05, time_step_count=40, external_flux=f,
                                current_sources=0.4 * np.ones((c._Nj(), W, 1)))
    a, b = (backend.GpuSimulation(prob, fast_poisson=True) for _ in range(2))
    assert a.plan.fast_poisson
    a.run(40)
    a.synchronize()
    b.run_timed(40)
    b.synchronize()
    assert torch.equal(a.theta(), b.theta())
