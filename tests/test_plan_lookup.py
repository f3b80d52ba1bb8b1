"""Set-up of a plan on the host: a kept plan is found without choosing its solver again, and a square array's
grid of faces is recognised once per matrix (no GPU: the device plan is a stand-in)."""
import numpy as np
import pytest

from pyjjasim_gb300 import plan as P
from pyjjasim_gb300.circuit import Circuit, HoneycombArray, SquareArray

STENCIL = ((1.0, -1.0, 0.0), (1.0, -2.0, 1.0))


@pytest.fixture
def counted(monkeypatch):
    """Counts recognitions, factorisations and plans; plans are the options they were asked for with."""
    counts = dict(grid=0, factor=0, plan=0)

    def count(name, f):
        def g(*a, **k):
            counts[name] += 1
            return f(*a, **k)
        return g

    class FakePlan:
        def __init__(self, *a, **k):
            counts["plan"] += 1
            self.options = k

    P.clear_cache()
    monkeypatch.setattr(P, "poisson_grid", count("grid", P.poisson_grid))
    monkeypatch.setattr(P, "HostFactor", count("factor", P.HostFactor))
    monkeypatch.setattr(P, "DevicePlan", FakePlan)
    yield counts
    P.clear_cache()


@pytest.mark.parametrize("make,W", [(lambda: SquareArray(40, 40), 200), (lambda: SquareArray(64, 64), 1),
                                    (lambda: HoneycombArray(8, 8), 3), (lambda: SquareArray(9, 9), 2)])
def test_a_kept_plan_is_found_at_once(counted, make, W):
    c = make()
    p = P.get_plan(c, 0.05, W, 3, STENCIL)
    after = dict(counted)
    assert after["plan"] == 1 and after["factor"] == 1
    assert P.get_plan(c, 0.05, W, 3, STENCIL) is p and P.get_plan(make(), 0.05, W, 3, STENCIL) is p
    assert counted == after
    # other critical currents: another plan, the same matrix
    c.set_critical_current(1.1)
    q = P.get_plan(c, 0.05, W, 3, STENCIL)
    assert q is not p and counted == dict(after, plan=2) and (q.options["sine"] is None) == (p.options["sine"] is None)
    # what was asked for counts too
    assert P.get_plan(c, 0.05, W, 3, STENCIL, fast_poisson=False) is not q
    assert P.get_plan(c, 0.05, W, 3, STENCIL, tuning=dict(groups=1)) is not q


def test_evicted_plans_are_made_again(counted):
    c = SquareArray(20, 20)
    first = P.get_plan(c, 0.05, 1, 3, STENCIL)
    for W in range(2, 2 + P.MAX_PLANS):
        P.get_plan(c, 0.05, W, 3, STENCIL)
    again = P.get_plan(c, 0.05, 1, 3, STENCIL)
    assert again is not first and len(P._PLANS) == P.MAX_PLANS
    assert P.get_plan(c, 0.05, 1, 3, STENCIL) is again


def test_a_circuit_without_coordinates_does_not_hide_a_grid(counted):
    a = SquareArray(40, 40)
    bare = Circuit(a.get_cycle_matrix())
    assert P.get_plan(bare, 0.05, 200, 3, STENCIL).options["sine"] is None
    assert P._kept_grid(a, P.face_matrix(a, 0.05)[1], "some digest") is not None


@pytest.mark.parametrize("nx,ny", [(3, 3), (3, 6), (7, 4), (12, 9), (2, 6), (6, 2)])
@pytest.mark.parametrize("swap,sx,sy", [(False, 1, 1), (False, -1, 1), (True, 1, -1), (True, -1, -1)])
def test_numbered_grids_are_those_of_the_coordinates(monkeypatch, nx, ny, swap, sx, sy):
    a = SquareArray(nx, ny)
    x, y = (np.asarray(v, float) for v in a.get_node_coordinates())
    n1, n2 = a.get_junction_nodes()
    x, y = sx * x, sy * y
    c = Circuit(a.get_cycle_matrix(), node_x=y if swap else x, node_y=x if swap else y, node1=n1, node2=n2)
    K = P.face_matrix(c, 0.05)[1]
    fast = P.poisson_grid(c, K)
    monkeypatch.setattr(P, "_numbered_grid", lambda *a: None)
    slow = P.poisson_grid(c, K)
    assert fast[:2] == slow[:2] and fast[3] == slow[3]
    np.testing.assert_array_equal(fast[2], slow[2])


def test_numbered_grid_wants_every_neighbour():
    """A 5 x 6 grid's matrix with the couplings of two faces moved is no grid, whatever its counts."""
    c = SquareArray(6, 7)
    K = P.face_matrix(c, 0.05)[1].tolil()
    v = K[0, 1]
    m = int(P.face_matrix(c, 0.05)[1].indices[2])
    K[7, 8] = K[8, 7] = 0.0
    K[7, 20] = K[20, 7] = v
    K = K.tocsc()
    K.eliminate_zeros()
    K.sort_indices()
    assert P._numbered_grid(c, K) is None and P.poisson_grid(c, K) is None
    assert m in (5, 6)


def test_digests_tell_contents_types_and_shapes_apart(monkeypatch):
    monkeypatch.setattr(P, "_DIGEST_PIECE", 1 << 10)
    a = np.arange(5000, dtype=np.int64)
    b = a.copy()
    seen = {P._digest(a)}
    assert P._digest(b) in seen
    for k in (0, 127, 128, 4999):     # either side of a piece's end
        b[k] ^= 1
        d = P._digest(b)
        assert d not in seen
        seen.add(d)
    for other in ((a.view(np.float64),), (a.reshape(50, 100),), (a[:2500], a[2500:]), (a, a[:0]), (a[::-1],), ()):
        d = P._digest(*other)
        assert d not in seen
        seen.add(d)


@pytest.mark.parametrize("make,W,ordering,want", [
    (lambda: HoneycombArray(24, 24), 4096, "auto", "nd"),     # blocks, with more work than minimum degree is taken from
    (lambda: HoneycombArray(24, 24), 4096, "mmd", "mmd"), (lambda: SquareArray(90, 90), 600, "auto", "mmd"),
    (lambda: SquareArray(9, 9), 1, "auto", "nd")])
def test_a_plan_says_the_order_of_its_factor(counted, monkeypatch, make, W, ordering, want):
    got = []
    order = P.fill_reducing_order
    monkeypatch.setattr(P, "fill_reducing_order", lambda K, o, c=None: got.append(o) or order(K, o, c))
    p = P.get_plan(make(), 0.05, W, 3, STENCIL, ordering=ordering)
    assert p.ordering == want and got == [want]
