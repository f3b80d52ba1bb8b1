"""Performance cases: what users of this package have it do, through its public entry points.

A case is a dict of plain values. ``prepare(case, seed)`` makes what a program has in hand before
the call (the array, the bias and flux values drawn from the seed, the problem or the simulation it
keeps), ``run(state)`` is one pass, ``exact(case, seed)`` the same outputs from plain torch in 64
bits, ``work(case)`` the bytes and operations a pass cannot do without.

Kinds of calls:
  evolve   TimeEvolutionProblem(...).compute(), the whole drop-in call: host inputs, host results
  advance  a GpuSimulation that the program keeps: restart from its phases, step, read the phases
  adjoint  TimeAveragedVoltageLoss: loss and gradients of disordered arrays
  ragged   a RaggedBatch of different lattices stepped together
  static   a batch of StaticProblems solved by Newton's method
"""
import functools
import math

import numpy as np
import torch

import pyjjasim_gb300 as jja

LATTICES = {"square": jja.SquareArray, "honeycomb": jja.HoneycombArray, "triangular": jja.TriangularArray}
DT = 0.05

# the options of a time evolution that a case may leave out
DEFAULTS = dict(stencil=3, C=0.0, L=0.0, R_sigma=0.0, T=0.0, ac=0.0, vs=0.0, f=0.1, bias_lo=0.0, bias_hi=2.0, keep="last")


def listed():
    return [
        # the smallest call and the package's first example: one 10x10 array at a constant bias,
        # 2000 steps, phases, voltages and currents of every step kept (the API's defaults)
        dict(name="plain_10x10", kind="evolve", lattice="square", nx=10, ny=10, W=1, steps=2000, bias_lo=0.4,
             bias_hi=0.6, keep="all"),
        # an IV curve of a small honeycomb array: an odd number of bias points in one call
        dict(name="iv_honeycomb_24_w61", kind="evolve", lattice="honeycomb", nx=24, ny=24, W=61, steps=300, f=0.2),
        # one ordinary square array followed for a thousand steps
        dict(name="square_128_w1", kind="evolve", lattice="square", nx=128, ny=128, W=1, steps=1000, f=0.25,
             bias_lo=0.8, bias_hi=1.2),
        # one AC-driven array with capacitance, inductance and thermal noise: time-dependent sources
        dict(name="ac_driven_256_w1", kind="evolve", lattice="square", nx=256, ny=256, W=1, steps=600, C=1.0, L=0.1,
             T=0.01, ac=0.3, bias_lo=0.75, bias_hi=0.85),
        # the headline: an IV sweep of 512 problems on 128x128 arrays
        dict(name="iv_sweep_128_w512", kind="advance", lattice="square", nx=128, ny=128, W=512, steps=256, f=0.25),
        # spread in the junction resistances on a triangular array: no fast solver applies
        dict(name="triangular_disorder_w96", kind="advance", lattice="triangular", nx=64, ny=48, W=96, steps=200,
             R_sigma=0.2, f=0.15),
        # a rectangular array of odd sizes, higher-order stencil, C and L, driven by voltage sources
        dict(name="stencil4_101x60_w24", kind="evolve", lattice="square", nx=101, ny=60, W=24, steps=300, stencil=4,
             C=0.7, L=0.2, vs=0.3, bias_lo=0.2, bias_hi=1.5),
        # gradients: 64 disorder draws of a 64x64 array, loss and its derivatives in Ic, f and bias
        dict(name="adjoint_64_w64", kind="adjoint", lattice="square", nx=64, ny=64, W=64, steps=256),
        # the largest array: 2.1 million junctions, 8 bias values, C, L and on-device noise
        dict(name="large_1024_w8", kind="advance", lattice="square", nx=1024, ny=1024, W=8, steps=32, C=0.5, L=0.05,
             T=0.005, bias_lo=0.5, bias_hi=1.2),
        # a batch of different lattices and sizes stepped as one system
        dict(name="ragged_24", kind="ragged", count=24, side_lo=32, side_hi=128, steps=200, f=0.25),
        # stationary states: 64 problems of a 64x64 array by Newton's method
        dict(name="static_64_w64", kind="static", lattice="square", nx=64, ny=64, W=64, L=0.1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


MOST_WORK = 128 * 127 * 2 * 512 * 256   # junction-steps of the largest listed case


def draw(rng):
    kind = rng.choice(["evolve", "evolve", "evolve", "advance", "advance", "advance", "adjoint", "ragged", "static"])
    if kind == "ragged":
        return dict(kind=kind, count=rng.randint(6, 28), side_lo=rng.randint(16, 40), side_hi=rng.randint(56, 128),
                    steps=2 * rng.randint(50, 120), f=round(rng.uniform(0.05, 0.4), 3))
    if kind == "static":
        return dict(kind=kind, lattice="square", nx=_log(rng, 12, 72), ny=_log(rng, 12, 72), W=_log(rng, 1, 64), L=0.1)
    if kind == "adjoint":
        return dict(kind=kind, lattice="square", nx=_log(rng, 16, 72), ny=_log(rng, 16, 64), W=_log(rng, 1, 64),
                    steps=rng.randint(100, 256))
    lattice = rng.choice(["square", "square", "square", "honeycomb", "triangular"])
    most = 40 if lattice == "honeycomb" else 80 if lattice == "triangular" else 400 if kind == "advance" else 140
    nx = _log(rng, 6, most)
    ny = max(6, min(most, int(nx * rng.uniform(0.6, 1.4))))
    W = _log(rng, 1, 512 if kind == "advance" else 100)
    junctions = {"square": 2, "honeycomb": 6, "triangular": 6}[lattice] * nx * ny
    while junctions * W > 1.2e7:
        W = (W + 1) // 2
    steps = 2 * max(16, min(150 if kind == "evolve" else 128, MOST_WORK // (4 * junctions * W)))
    case = dict(kind=kind, lattice=lattice, nx=nx, ny=ny, W=W, steps=steps, f=round(rng.uniform(0.02, 0.4), 3))
    if rng.random() < 0.4:
        case.update(C=round(rng.uniform(0.2, 1.0), 2))
    if rng.random() < 0.4:
        case.update(L=round(rng.uniform(0.05, 0.5), 2))
    if rng.random() < 0.25:
        case.update(T=round(rng.uniform(0.002, 0.05), 3))
    if rng.random() < 0.25:
        case.update(R_sigma=0.2)
    if kind == "evolve":
        if rng.random() < 0.25:
            case.update(stencil=rng.choice([4, 5]), C=round(rng.uniform(0.5, 1.0), 2))
        if rng.random() < 0.2:
            case.update(vs=0.3)
        if rng.random() < 0.2:
            case.update(ac=0.3)
        if nx * ny * W < 2000:
            case.update(keep="all")
    return case


# ---------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=64)
def _array(lattice, nx, ny, C=0.0, L=0.0, R_sigma=0.0):
    """The array of a case (a program builds it once) and its uniform bias pattern."""
    a = LATTICES[lattice](nx, ny)
    if R_sigma:
        a.set_resistance(np.random.default_rng(7).lognormal(0.0, R_sigma, a.junction_count()))
    if C:
        a.set_capacitance(C)
    if L:
        a.set_inductance(L)
    if lattice == "square":   # unit current along x: what current_base(0) gives on a square array
        base = np.zeros(a.junction_count())
        base[:(nx - 1) * ny] = 1.0
    else:
        base = a.current_base(0.0)
    return a, base


def _full(case):
    return {**DEFAULTS, **case}


def _circuit(c):
    return _array(c["lattice"], c["nx"], c["ny"], c["C"], c["L"], c["R_sigma"])


def _values(c, seed):
    """The seed's bias amplitudes (sorted, as along an IV curve), flux and voltage amplitudes."""
    rng = np.random.default_rng(seed)
    bias = np.sort(rng.uniform(c["bias_lo"], c["bias_hi"], c["W"]))
    return bias, c["f"] * rng.uniform(0.9, 1.1), c["vs"] * rng.uniform(0.9, 1.1)


def _problem(c, seed):
    a, base = _circuit(c)
    bias, f, vs = _values(c, seed)
    if c["ac"]:
        pattern = base[:, None] * bias[None, :]

        def current(i):
            return pattern * (1.0 + c["ac"] * np.sin(2 * np.pi * 0.05 * i * DT))
    else:
        current = base[:, None, None] * bias[None, :, None]
    opts = dict(store_voltage=True, store_current=c["keep"] == "all",
                store_time_steps=None if c["keep"] == "all" else [c["steps"] // 2, c["steps"] - 1])
    if c["vs"]:
        opts["voltage_sources"] = _voltage_pattern(base, vs)[:, None, None]
    if c["T"]:
        opts["temperature"] = c["T"]
    return jja.TimeEvolutionProblem(a, time_step=DT, time_step_count=c["steps"], external_flux=f,
                                    current_sources=current, stencil_width=c["stencil"], **opts)


def _voltage_pattern(base, vs):
    """A voltage source in every 16th driven junction."""
    v = np.zeros(len(base))
    v[np.flatnonzero(base)[::16]] = vs
    return v


def _ragged_spec(case, seed):
    """Lattice kinds and sides of the batch (fixed by the case) and the seed's bias values."""
    rng = np.random.default_rng(case["count"] * 1000 + case["side_hi"])
    kinds = [("square", "honeycomb", "triangular")[k] for k in rng.integers(0, 3, case["count"])]
    sides = rng.integers(case["side_lo"], case["side_hi"] + 1, case["count"])
    bias = np.random.default_rng(seed).uniform(0.0, 2.0, case["count"])
    # honeycomb and triangular unit cells hold 4 and 2 nodes: the same side means that many more
    return [(k, max(4, int(n) // {"square": 1, "honeycomb": 2, "triangular": 1}[k]), b)
            for k, n, b in zip(kinds, sides, bias)]


def _adjoint_inputs(case, seed):
    a, base = _array(case["lattice"], case["nx"], case["ny"])
    rng = np.random.default_rng(seed)
    W = case["W"]
    Ic = rng.lognormal(0.0, 0.2, (a.junction_count(), W))
    f = np.full((a.face_count(), W), 0.1) * rng.uniform(0.95, 1.05, (1, W))
    bias = np.full(W, 1.2) * rng.uniform(0.95, 1.05, W)
    setup = dict(circuit=a, dt=DT, Nt=case["steps"], base=base, t1=case["steps"] // 2, t2=case["steps"] - 1,
                 junctions=np.flatnonzero(base))
    return Ic, f, bias, setup


def _static_inputs(case, seed):
    a, base = _array(case["lattice"], case["nx"], case["ny"], 0.0, case["L"])
    rng = np.random.default_rng(seed)
    vertical = (base == 0.0).astype(float)
    out = []
    for w in range(case["W"]):
        ang = rng.uniform(0.0, np.pi)
        amp = rng.uniform(0.05, 0.3)
        out.append((amp * (np.cos(ang) * base + np.sin(ang) * vertical), 0.01 * rng.uniform(0.0, 0.5)))
    return a, out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "evolve":
        return dict(kind=kind, problem=_problem(_full(case), seed), seed=seed)
    if kind == "advance":
        from pyjjasim_gb300.backend import GpuSimulation
        c = _full(case)
        sim = GpuSimulation(_problem(c, seed), seed=seed)
        return dict(kind=kind, sim=sim, steps=c["steps"], start=[h.clone() for h in sim.history()])
    if kind == "adjoint":
        dev = "cuda"
        Ic, f, bias, setup = _adjoint_inputs(case, seed)
        t = [torch.tensor(v, device=dev, requires_grad=True) for v in (Ic, f, bias)]
        return dict(kind=kind, inputs=t, setup=setup)
    if kind == "ragged":
        from pyjjasim_gb300.ragged import RaggedBatch
        probs = []
        for lattice, n, b in _ragged_spec(case, seed):
            a, base = _array(lattice, n, n)
            probs.append(jja.TimeEvolutionProblem(a, time_step=DT, time_step_count=case["steps"],
                                                  current_sources=base[:, None, None] * b, external_flux=case["f"],
                                                  store_time_steps=[case["steps"] - 1]))
        sims = RaggedBatch(probs).simulations()
        return dict(kind=kind, sims=sims, steps=case["steps"], start=[[h.clone() for h in s.history()] for s in sims])
    a, specs = _static_inputs(case, seed)
    return dict(kind=kind, problems=[jja.StaticProblem(a, current_sources=Is, external_flux=f) for Is, f in specs])


# ---------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind == "evolve":
        r = state["problem"].compute(seed=state["seed"])
        out = {"theta": r.get_theta(), "voltage": r.get_voltage()}
        if r.current is not None:
            out["current"] = r.get_current()
        return out
    if kind == "advance":
        sim = state["sim"]
        sim.set_history(state["start"], 0)
        sim.run(state["steps"])
        sim.synchronize()     # the check for diverged phases that a reader of the results needs
        return dict(zip(("theta", "previous"), sim.history()))
    if kind == "ragged":
        from pyjjasim_gb300.ragged import RaggedBatch
        sims = state["sims"]
        for sim, start in zip(sims, state["start"]):
            sim.set_history(start, 0)
        RaggedBatch.run_simulations(sims, state["steps"])
        for sim in sims:
            sim.synchronize()
        return [s.theta() for s in sims]
    if kind == "adjoint":
        from pyjjasim_gb300.adjoint import TimeAveragedVoltageLoss
        Ic, f, bias = state["inputs"]
        for t in state["inputs"]:
            t.grad = None
        loss = TimeAveragedVoltageLoss.apply(Ic, f, bias, state["setup"])
        loss.sum().backward()
        return {"loss": loss.detach(), "Ic": Ic.grad, "f": f.grad, "bias": bias.grad}
    from pyjjasim_gb300.static import compute_many
    got = compute_many(state["problems"])
    return {"theta": np.stack([s.get_theta() for s, _, _ in got]),
            "status": np.array([st for _, st, _ in got]),
            "iterations": np.array([i.get_number_of_iterations() for _, _, i in got])}


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------
def _counts(lattice, nx, ny):
    if lattice == "square":
        return (nx - 1) * ny + nx * (ny - 1), (nx - 1) * (ny - 1)
    a, _ = _array(lattice, nx, ny)
    return a.junction_count(), a.face_count()


ON_CHIP = 128 << 20   # a state larger than the L2 cache moves through memory on every step


def _steps_work(Nj, Nf, W, steps, width, stored):
    state = 8.0 * Nj * W * width          # the phase history in, the new phase out
    moved = state * steps if state > ON_CHIP else state
    # per step: current balance and update of every junction, a fast elliptic solve of the faces
    flops = steps * W * (24.0 * Nj + 10.0 * Nf * math.log2(Nf + 1))
    return moved + 8.0 * Nj * W * stored, flops


def work(case):
    kind = case["kind"]
    if kind == "ragged":
        b = fl = 0.0
        Nj = Nf = 0
        for lattice, n, _ in _ragged_spec(case, 0):
            j, f = _counts(lattice, n, n)
            Nj, Nf = Nj + j, Nf + f
        b, fl = _steps_work(Nj, Nf, 1, case["steps"], 3, 1)
        return {"bytes": b, "flops": fl}
    Nj, Nf = _counts(case["lattice"], case["nx"], case["ny"])
    if kind == "adjoint":
        b, fl = _steps_work(Nj, Nf, case["W"], case["steps"], 3, 3)
        return {"bytes": 3 * b, "flops": 3 * fl}
    if kind == "static":
        # about six iterations, each a sparse factorisation of the faces
        return {"bytes": 8.0 * case["W"] * (4 * Nj + 2 * Nf), "flops": 6.0 * case["W"] * 10.0 * Nf ** 1.5}
    c = _full(case)
    stored = 3 * c["steps"] if c["keep"] == "all" else (4 if kind == "evolve" else 2)
    b, fl = _steps_work(Nj, Nf, c["W"], c["steps"], c["stencil"], stored)
    return {"bytes": b, "flops": fl}


# ---------------------------------------------------------------------------------------------
# the same in plain torch, 64 bits
# ---------------------------------------------------------------------------------------------
class _Faces:
    """K^-1 b and the products with A for one array, in plain torch."""

    def __init__(self, a, diag, uniform, dev):
        A = a.get_cycle_matrix().tocoo()
        at = torch.tensor(np.stack([A.row, A.col]).astype(np.int64), device=dev)
        val = torch.tensor(A.data.astype(np.float64), device=dev)
        self.A = torch.sparse_coo_tensor(at, val, A.shape).coalesce()
        self.At = self.A.t().coalesce()
        self.sine = None
        if uniform:
            # a square array of equal junctions: K is kappa times the five-point Laplacian on the
            # grid of faces, diagonal in sine transforms
            x, y = (np.asarray(v, float) for v in a.get_node_coordinates())
            n1, n2 = a.get_junction_nodes()
            cnt = np.bincount(A.row, minlength=A.shape[0])
            fx = np.bincount(A.row, 0.5 * (x[n1] + x[n2])[A.col], A.shape[0]) / cnt
            fy = np.bincount(A.row, 0.5 * (y[n1] + y[n2])[A.col], A.shape[0]) / cnt
            mx, my = a.count_x - 1, a.count_y - 1
            cell = (np.round(fy - 0.5) * mx + np.round(fx - 0.5)).astype(np.int64)
            self.cell = torch.tensor(cell, device=dev)
            one = lambda m: torch.arange(1, m + 1, dtype=torch.float64, device=dev)
            S = lambda m: math.sqrt(2.0 / (m + 1)) * torch.sin(torch.remainder(
                one(m)[:, None] * one(m)[None, :], 2 * (m + 1)) * (math.pi / (m + 1)))
            lam = lambda m: 2.0 - 2.0 * torch.cos(one(m) * (math.pi / (m + 1)))
            self.sine = (mx, my, S(mx), S(my), float(diag[0]) * (lam(my)[:, None] + lam(mx)[None, :]))
        else:
            d = torch.tensor(diag, device=dev)
            dense = self.A.to_dense()
            self.chol = torch.linalg.cholesky((dense * d) @ dense.T)

    def mul(self, v):
        return torch.sparse.mm(self.A, v)

    def mul_t(self, v):
        return torch.sparse.mm(self.At, v)

    def solve(self, b):
        if self.sine is None:
            return torch.cholesky_solve(b, self.chol)
        mx, my, Sx, Sy, lam = self.sine
        W = b.shape[1]
        g = torch.empty((my * mx, W), dtype=b.dtype, device=b.device).index_copy(0, self.cell, b)
        g = g.T.reshape(W, my, mx)
        g = Sy @ ((Sy @ g @ Sx) / lam) @ Sx
        return g.reshape(W, my * mx).T[self.cell]


STENCILS = {3: ((1.0, -1.0, 0.0), (1.0, -2.0, 1.0)),
            4: ((1.5, -2.0, 0.5, 0.0), (2.0, -5.0, 4.0, -1.0)),
            5: ((11.0 / 6, -3.0, 1.5, -1.0 / 3, 0.0), (35.0 / 12, -26.0 / 3, 9.5, -14.0 / 3, 11.0 / 12))}
EXTRAPOLATE = {3: (2.0, -1.0), 4: (3.0, -3.0, 1.0), 5: (4.0, -6.0, 4.0, -1.0)}
DENSE_FACES = 13000


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _seconds(Nj, Nf, W, steps, uniform, mx, my):
    """A rough time of the plain computation on this GPU's 64-bit units."""
    solve = 4.0 * mx * my * (mx + my) * W if uniform else 2.0 * Nf * Nf * W
    return steps * (solve / 0.8e12 + 60.0 * 8 * Nj * W / 4e12 + 1e-3) + (0 if uniform else 1.5 * Nf ** 3 / 0.8e12)


def _evolve_exact(c, seed):
    a, base = _circuit(c)
    Nj, Nf, W, steps, width = a.junction_count(), a.face_count(), c["W"], c["steps"], c["stencil"]
    uniform = c["lattice"] == "square" and not c["R_sigma"]
    if c["T"] or (not uniform and Nf > DENSE_FACES) or \
            _seconds(Nj, Nf, W, steps, uniform, c["nx"] - 1, c["ny"] - 1) > 15:
        return None
    dev = _device()
    R = np.random.default_rng(7).lognormal(0.0, c["R_sigma"], Nj) if c["R_sigma"] else np.ones(Nj)
    Rv, Cv = 1.0 / (DT * R), np.full(Nj, c["C"] / DT ** 2)
    faces = _Faces(a, c["L"] + 1.0 / (Cv + Rv), uniform, dev)
    s1, s2 = STENCILS[width]
    coef = [torch.tensor(s1[k] * Rv + s2[k] * Cv, device=dev)[:, None] for k in range(width)]
    bias, f, vs = _values(c, seed)
    pattern = torch.tensor(base[:, None] * bias[None, :], device=dev)
    Vs = torch.tensor(_voltage_pattern(base, vs), device=dev)[:, None]
    theta_s = torch.zeros((Nj, 1), dtype=torch.float64, device=dev)
    hist = [torch.zeros((Nj, W), dtype=torch.float64, device=dev) for _ in range(width - 1)]
    past_I = [torch.zeros_like(hist[0]) for _ in range(width - 1)]
    keep = set(range(steps)) if c["keep"] == "all" else {steps // 2, steps - 1}
    th_out, v_out, i_out = [], [], []
    for i in range(steps):
        Is = pattern * (1.0 + c["ac"] * math.sin(2 * math.pi * 0.05 * i * DT)) if c["ac"] else pattern
        x = torch.sin(sum(e * h for e, h in zip(EXTRAPOLATE[width], hist))) - Is
        for k in range(1, width):
            x = x + coef[k] * hist[k - 1]
        y = faces.mul_t(faces.solve(faces.mul(x / coef[0] - theta_s) - 2 * math.pi * f))
        th = (y - x) / coef[0]
        if c["vs"]:
            theta_s = theta_s + Vs * DT
        I = y + Is
        if i in keep and c["kind"] == "evolve":
            th_out.append(th)
            V = sum(s * h for s, h in zip(s1[:-1], [th] + hist[:-1])) / DT
            if c["L"]:
                V = V + c["L"] * sum(s * h for s, h in zip(s1[:-1], [I] + past_I[:-1])) / DT
            v_out.append(V)
            i_out.append(I)
        hist = [th] + hist[:-1]
        past_I = [I] + past_I[:-1]
    if c["kind"] == "advance":
        return {"theta": hist[0], "previous": hist[1]}
    out = {"theta": torch.stack(th_out, 2), "voltage": torch.stack(v_out, 2)}
    if c["keep"] == "all":
        out["current"] = torch.stack(i_out, 2)
    return out


def _adjoint_exact(case, seed):
    Ic, f, bias, setup = _adjoint_inputs(case, seed)
    a, base = setup["circuit"], setup["base"]
    Nj, Nf, W, steps = a.junction_count(), a.face_count(), case["W"], case["steps"]
    if _seconds(Nj, Nf, W, 3 * steps, True, case["nx"] - 1, case["ny"] - 1) > 15 or steps * Nj * W * 80 > 60e9:
        return None
    dev = _device()
    faces = _Faces(a, np.full(Nj, DT), True, dev)
    Ic, f, bias = (torch.tensor(v, device=dev, requires_grad=True) for v in (Ic, f, bias))
    pattern = torch.tensor(base, device=dev)[:, None]
    c0 = 1.0 / DT
    h1 = h2 = torch.zeros((Nj, W), dtype=torch.float64, device=dev)
    at = {}
    for i in range(steps):
        x = Ic * torch.sin(2.0 * h1 - h2) - c0 * h1 - pattern * bias
        y = faces.mul_t(faces.solve(faces.mul(x / c0) - 2 * math.pi * f))
        h1, h2 = (y - x) / c0, h1
        if i in (setup["t1"], setup["t2"]):
            at[i] = h1[torch.tensor(setup["junctions"], device=dev)]
    loss = ((at[setup["t2"]] - at[setup["t1"]]) / (DT * (setup["t2"] - setup["t1"]))).mean(0)
    loss.sum().backward()
    return {"loss": loss.detach(), "Ic": Ic.grad, "f": f.grad, "bias": bias.grad}


def exact(case, seed):
    if case["kind"] in ("evolve", "advance"):
        return _evolve_exact(_full(case), seed)
    if case["kind"] == "adjoint":
        return _adjoint_exact(case, seed)
    return None   # ragged unions and Newton iterations: no plain counterpart in reasonable time
