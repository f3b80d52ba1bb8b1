"""Which solver the default plan takes, where accuracy or repeatability decides."""
import types

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


# nodes, problems, solver: power-of-two grids of few problems had the radix-2 transforms, whose runs repeat bit for bit
REPEATS = [(16, 16, 1, "fast_poisson"), (32, 32, 1, "fast_poisson"), (32, 32, 8, "fast_poisson"),
           (64, 32, 3, "fast_poisson"), (64, 64, 2, "fast_poisson"), (64, 64, 8, "fast_poisson"),
           (256, 256, 4, "fast_poisson"), (512, 512, 1, "fast_poisson"), (128, 128, 8, "sine"), (10, 10, 8, "resident")]


@pytest.mark.parametrize("nx,ny,W,solver", REPEATS)
def test_power_of_two_grids_of_few_problems_take_what_repeats(monkeypatch, nx, ny, W, solver):
    asked = {}
    monkeypatch.setattr(P, "HostFactor", lambda *a, **k: None)
    monkeypatch.setattr(P, "DevicePlan", lambda *a, **k: types.SimpleNamespace(asked=asked.update(k)))
    P.clear_cache()
    P.get_plan(SquareArray(nx, ny), 0.05, W, 3, ((1.0, -1.0, 0.0), (1.0, -2.0, 1.0)))
    P.clear_cache()
    assert [k for k in ("fast_poisson", "sine", "resident", "blocks", "top") if asked[k] not in (None, False)] == [solver]


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,W,solver", REPEATS)
def test_their_runs_repeat_bit_for_bit(nx, ny, W, solver):
    import torch
    base = np.zeros((nx - 1) * ny + nx * (ny - 1))
    base[:(nx - 1) * ny] = 1.0
    prob = TimeEvolutionProblem(SquareArray(nx, ny), time_step=0.05, time_step_count=30, external_flux=0.1,
                                current_sources=base[:, None, None] * np.linspace(0.3, 1.5, W)[None, :, None])
    sim = backend.GpuSimulation(prob)
    start, first = [h.clone() for h in sim.history()], None
    for _ in range(4):
        sim.set_history(start, 0)
        sim.run(30)
        sim.synchronize()
        first = sim.theta().clone() if first is None else first
        assert torch.equal(sim.theta(), first)


@pytest.mark.parametrize("trees,leaf", [
    ([3353] * 12, 384), ([14520] + [5006] * 10, 384), ([14520, 14520] + [3949] * 9, 768),   # equal means, larger squares
    ([34782] + [3878] * 7, 1536), ([34782, 20000] + [4679] * 6, 3072), ([29756, 25000] + [4856] * 10, 6144),
    ([25122, 20000] + [2675] * 25, 12288), ([14520] * 4 + [2868] * 21, None), ([34782, 30000] + [5140] * 12, 12288),
    ([11444] * 24, 6144), ([200_000, 30_000], None)])                                       # a tree above 2^17: by its size alone
def test_a_unions_top_block_by_its_trees(trees, leaf):
    """The separators' blocks of a union are read once a step: the rule keeps them within the L2 cache, whatever
    the trees' mean (one large lattice among small ones counts by its square)."""
    class Union:
        components, tree_faces = len(trees), tuple(trees)

        def _Nf(self):
            return sum(trees)

    assert P.top_leaf(Union(), 1) == leaf


def test_a_ragged_batch_says_its_trees():
    from pyjjasim_gb300.ragged import RaggedBatch
    circuits = [SquareArray(4, 5), HoneycombArray(3, 3), SquareArray(7, 3)]
    Is = [np.zeros((c._Nj(), 2, 1)) for c in circuits]
    probs = [TimeEvolutionProblem(c, time_step=0.05, time_step_count=3, current_sources=i) for c, i in zip(circuits, Is)]
    u = RaggedBatch(probs).circuit
    assert sorted(P.tree_sizes(u)) == sorted(2 * [c._Nf() for c in circuits]) and sum(P.tree_sizes(u)) == u._Nf()


@pytest.mark.parametrize("n,W,leaf", [
    (32768, 1, 768), (32769, 1, 3072), (46000, 7, 3072), (46001, 1, 6144), (54000, 7, 6144), (54001, 2, 12288), (66000, 7, 12288),
    (66001, 1, 24576), (100000, 3, 24576), (66001, 4, 6144), (100001, 1, 6144), (1 << 17, 1, 6144), (60000, 512, 3072),
    (200000, 8, None), (200000, 16, 6144), (400001, 16, None), (400001, 32, 6144), ((1 << 19) + 1, 64, None)])
def test_a_single_trees_top_block(n, W, leaf):
    class One:
        def _Nf(self):
            return n

    assert P.top_leaf(One(), W) == leaf
