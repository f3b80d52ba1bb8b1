"""Which solver the default plan takes, where that is decided by accuracy."""
import numpy as np
import pytest

from pyjjasim_gb300 import TimeEvolutionProblem, backend
from pyjjasim_gb300 import plan as P
from pyjjasim_gb300.circuit import HoneycombArray, SquareArray


def _spread(c, sigma):
    c.set_resistance(np.random.default_rng(7).lognormal(0.0, sigma, c._Nj()))
    return c


def _one_junction(c, factor, what):
    v = np.ones(c._Nj())
    v[c._Nj() // 3] = factor
    (c.set_resistance if what == "R" else c.set_inductance)(v)
    return c


# circuit, products allowed
WEIGHTS = [(lambda: SquareArray(10, 10), True), (lambda: _spread(SquareArray(10, 10), 0.4), True),
           (lambda: _spread(SquareArray(10, 10), 3.0), False), (lambda: _spread(HoneycombArray(24, 24), 0.4), True),
           (lambda: _spread(HoneycombArray(24, 24), 3.0), False),
           (lambda: _one_junction(SquareArray(10, 10), 200.0, "R"), True),
           (lambda: _one_junction(SquareArray(10, 10), 1e3, "R"), False),
           (lambda: _one_junction(SquareArray(40, 30), 1e-3, "R"), False),
           (lambda: _one_junction(SquareArray(40, 30), 1e3, "L"), False)]


@pytest.mark.parametrize("make,even", WEIGHTS)
def test_even_weights(make, even):
    assert P.even_weights(make(), 0.05) == even


@pytest.mark.gpu
@pytest.mark.parametrize("make,even", WEIGHTS)
def test_uneven_circuits_keep_the_sweeps(make, even):
    c = make()
    prob = TimeEvolutionProblem(c, time_step=0.05, time_step_count=20, external_flux=0.1,
                                current_sources=c.current_base(0.0)[:, None, None] * np.array([0.4, 0.9])[None, :, None])
    sim = backend.GpuSimulation(prob)
    assert (sim.plan.resident or sim.plan.blocks is not None) == even and not sim.plan.sine and sim.plan.top is None
    if not even:
        assert backend.GpuSimulation(prob, fast_poisson=False).plan is sim.plan
