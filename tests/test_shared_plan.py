"""Simulations of one cached plan on streams and threads of their own: the plan's work vectors are shared, so the
calls follow one another and each simulation gets what it gets alone."""
import threading

import numpy as np
import pytest

from pyjjasim_gb300 import TimeEvolutionProblem, backend
from pyjjasim_gb300.circuit import HoneycombArray, SquareArray

# circuit, W, fast_poisson, the plan's solver
PLANS = {"resident": (lambda: SquareArray(10, 10), 3, "auto"), "sweeps": (lambda: SquareArray(24, 20), 5, False),
         "radix2": (lambda: SquareArray(64, 64), 1, "auto"), "sine": (lambda: SquareArray(64, 64), 64, "auto"),
         "strips": (lambda: SquareArray(150, 140), 8, "auto"), "blocks": (lambda: HoneycombArray(24, 24), 8, "auto"),
         "top": (lambda: SquareArray(190, 180), 2, "auto")}


def _solver(pl):
    return "resident" if pl.resident else "radix2" if pl.fast_poisson else "sine" if pl.sine else \
        "blocks" if pl.blocks is not None else "top" if pl.top is not None else "sweeps"


@pytest.mark.gpu
@pytest.mark.parametrize("name", PLANS)
@pytest.mark.parametrize("threads", [False, True])
def test_simulations_that_share_a_plan(name, threads):
    import torch
    make, W, fast_poisson = PLANS[name]
    c = make()
    if name == "top":
        c.set_resistance(np.random.default_rng(0).lognormal(0.0, 0.2, c._Nj()))
    base = c.current_base(0.0)

    def problem(k):     # the plan does not depend on the sources: all of these share one
        Is = base[:, None, None] * np.linspace(0.3 + 0.2 * k, 0.9, W)[None, :, None]
        return TimeEvolutionProblem(c, time_step=0.05, time_step_count=60, current_sources=Is,
                                    external_flux=0.05 * (k + 1), temperature=0.01 * (k + 1))

    probs = [problem(k) for k in range(3)]
    alone = []
    for k, p in enumerate(probs):
        s = backend.GpuSimulation(p, seed=k, fast_poisson=fast_poisson)
        s.run(45)
        s.synchronize()
        alone.append(s.theta().cpu())
    sims = [backend.GpuSimulation(p, seed=k, fast_poisson=fast_poisson) for k, p in enumerate(probs)]
    assert all(s.plan is sims[0].plan for s in sims)
    assert _solver(sims[0].plan) == {"strips": "sine"}.get(name, name)
    slots = np.full(15, -1)
    slots[::4] = np.arange(4)

    kept = []     # written on the simulations' streams: alive until those are done

    def steps(s):
        out = torch.empty((4,) + tuple(s.theta().shape), dtype=torch.float64, device="cuda")
        kept.append(out)
        for _ in range(3):
            s.run(15, th_slot=slots, th_dev=out)

    torch.cuda.synchronize()
    if threads:
        ts = [threading.Thread(target=steps, args=(s,)) for s in sims]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
    else:
        for _ in range(3):
            for s in sims:
                s.run(15)
    for s, ref in zip(sims, alone):
        s.synchronize()
        assert float((s.theta().cpu() - ref).abs().max()) <= 1e-10 * max(1.0, float(ref.abs().max()))
