"""Host-side plan: the face-space matrix, its factor and the device plan, cached.

The reference rebuilds and refactorises K = A (L + diag(1/Cnext)) A^T inside every
time_evolution_core call (time_evolution.py:504-506). Here the factor (host, FP64,
nested dissection + supernodal Cholesky in libjja_gb300) and the device plan (factor
blocks + circuit tables uploaded once) are cached by the content that determines them:
the cycle matrix, R, C, L, dt and the stencil width (and W for the device plan), so
repeated compute() calls on the same circuit (e.g. an annealing schedule or a sweep)
pay the factorisation once.
"""
import ctypes
import hashlib
import threading
from collections import OrderedDict
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import scipy.sparse

from . import _native as N

_FACTORS = OrderedDict()
_PLANS = OrderedDict()
_ROUTES = OrderedDict()   # what was asked for -> key of its plan: a kept plan is found without choosing its solver
_GRIDS = OrderedDict()    # digest of K -> poisson_grid
MAX_FACTORS = 4
MAX_PLANS = 4
MAX_ROUTES = 64
MAX_GRIDS = 8
_CACHE_LOCK = threading.Lock()   # the caches are shared by host threads (ragged parts build in parallel);
                                 # the lock covers lookups and insertions, not the factorisations

# Extrapolation weights of the CPR argument on theta(t-1), theta(t-2), ... (time_evolution.py:547-553)
EXTRAP = {3: (2.0, -1.0), 4: (3.0, -3.0, 1.0), 5: (4.0, -6.0, 4.0, -1.0)}
# launch-shape fields of the triangular solves (jja_solve_tuning)
TUNING_FIELDS = ("rhs_block", "rows_per_lane", "target_warps", "min_piece", "schedule", "rows_per_lane_fwd",
                 "pack_rows", "pack_min_warps", "pdl", "groups", "coop_blocks", "dst_lines",
                 "pack_lanes", "subtree_rows")
SCHEDULES = {"levels": 1, "dataflow": 2, "cooperative": 3}


_DIGEST_PIECE = 4 << 20   # bytes hashed by one thread (hashlib lets go of the interpreter); 1024x1024: 250 -> 40 ms


def _digest(*arrays):
    """Digest of the arrays' types, shapes and contents, in pieces of a fixed size (large ones by several threads)."""
    h = hashlib.blake2b(digest_size=16)
    pieces = []
    for a in arrays:
        a = np.ascontiguousarray(a)
        h.update(str(a.dtype).encode() + str(a.shape).encode())
        flat = a.view(np.uint8).ravel() if a.size else np.empty(0, np.uint8)
        pieces += [flat[k:k + _DIGEST_PIECE] for k in range(0, len(flat), _DIGEST_PIECE)]
    one = lambda piece: hashlib.blake2b(piece, digest_size=16).digest()
    if len(pieces) > len(arrays):
        with ThreadPoolExecutor(8) as pool:
            parts = list(pool.map(one, pieces))
    else:
        parts = map(one, pieces)
    for part in parts:
        h.update(part)
    return h.hexdigest()


def coefficients(circuit, dt, stencil):
    """Per-junction stencil coefficients (time_evolution.py:472-478, 489, 495, 501)."""
    s1, s2 = stencil
    Rv = 1.0 / (dt * np.asarray(circuit._R(), np.float64))
    Cv = np.asarray(circuit._C(), np.float64) / dt ** 2
    coef = [s1[k] * Rv + s2[k] * Cv for k in range(len(s1))]
    return Rv, Cv, coef


def face_matrix(circuit, dt):
    """K = A (L + diag(1/(Cv + Rv))) A^T as CSC with sorted indices (time_evolution.py:504-505)."""
    A = scipy.sparse.csc_matrix(circuit.get_cycle_matrix()).astype(np.float64)
    Rv = 1.0 / (dt * np.asarray(circuit._R(), np.float64))
    Cv = np.asarray(circuit._C(), np.float64) / dt ** 2
    L = circuit._L()
    L = scipy.sparse.csc_matrix(L) if not scipy.sparse.issparse(L) else L
    K = (A @ (L + scipy.sparse.diags(1.0 / (Cv + Rv), 0)) @ A.T).tocsc()
    K.sum_duplicates()
    K.sort_indices()
    return A, K


class HostFactor:
    """Ordered supernodal Cholesky of K (owned C object)."""

    def __init__(self, K, coords=None, perm=None, nd_leaf=8, max_supernode=0, keep_factor=False, relax_zeros=-1,
                 relax_frac=-1.0):
        L = N.lib()
        n = K.shape[0]
        self.n = n
        colptr = np.ascontiguousarray(K.indptr, np.int64)
        rowind = np.ascontiguousarray(K.indices, np.int32)
        val = np.ascontiguousarray(K.data, np.float64)
        cx = cy = None
        if coords is not None:
            cx = np.ascontiguousarray(coords[0], np.float64)
            cy = np.ascontiguousarray(coords[1], np.float64)
        pm = None if perm is None else np.ascontiguousarray(perm, np.int32)
        opts = N.FactorOpts(nd_leaf, max_supernode, int(keep_factor), int(relax_zeros), float(relax_frac))
        h = ctypes.c_void_p()
        N.check(L.jja_factor_create(n, N.ptr(colptr, ctypes.c_int64), N.ptr(rowind, ctypes.c_int32), N.ptr(val),
                                    N.ptr(cx), N.ptr(cy), N.ptr(pm, ctypes.c_int32), ctypes.byref(opts),
                                    ctypes.byref(h)))
        self.handle = h
        st = N.FactorStats()
        N.check(L.jja_factor_get_stats(h, ctypes.byref(st)))
        self.stats = {k: getattr(st, k) for k, _ in N.FactorStats._fields_}

    def perm(self):
        out = np.empty(self.n, np.int32)
        N.check(N.lib().jja_factor_get_perm(self.handle, N.ptr(out, ctypes.c_int32)))
        return out

    def supernodes(self):
        """dict of per-supernode arrays: col0, k, m, level, parent."""
        ns = self.stats["n_supernodes"]
        out = {k: np.empty(ns, np.int32) for k in ("col0", "k", "m", "level", "parent")}
        N.check(N.lib().jja_factor_get_supernodes(self.handle, *(N.ptr(out[k], ctypes.c_int32)
                                                                for k in ("col0", "k", "m", "level", "parent"))))
        return out

    def check_schedule(self, W, tuning=None):
        """Build the GPU work-item schedule for W problems on the host and check its dataflow
        order (raises JJAError otherwise); returns the item counts (forward, backward)."""
        t = dict(tuning or {})
        tu = N.SolveTuning(*(int(t.get(f, 0)) for f in TUNING_FIELDS))
        nf, nb = ctypes.c_int64(0), ctypes.c_int64(0)
        N.check(N.lib().jja_factor_check_schedule(self.handle, int(W), ctypes.byref(tu), ctypes.byref(nf),
                                                  ctypes.byref(nb)))
        return nf.value, nb.value

    def schedule_stats(self, W, tuning=None):
        """dict: the shape of the GPU schedule for W problems (levels, bottom subtrees, subtree
        packs, work items), built on the host as the plan builds it."""
        t = dict(tuning or {})
        tu = N.SolveTuning(*(int(t.get(f, 0)) for f in TUNING_FIELDS))
        st = N.ScheduleStats()
        N.check(N.lib().jja_factor_schedule_stats(self.handle, int(W), ctypes.byref(tu), ctypes.byref(st)))
        return {k: getattr(st, k) for k, _ in N.ScheduleStats._fields_}

    def solve_host(self, b):
        """Host solve (diagnostic). b: (n,) or (n, nrhs)."""
        b = np.array(b, dtype=np.float64, order="C", copy=True)
        nrhs = 1 if b.ndim == 1 else b.shape[1]
        N.check(N.lib().jja_factor_solve_host(self.handle, N.ptr(b), nrhs))
        return b

    def __del__(self):
        h = getattr(self, "handle", None)
        if h is not None and N._lib is not None:
            N._lib.jja_factor_destroy(h)
            self.handle = None


def poisson_grid(circuit, K):
    """(mx, my, grid_face, kappa) when the face-space matrix is K = kappa (4 I - adjacency) on an
    mx x my grid of faces: a square array with equal R and C and a uniform self-inductance, whose K
    is kappa times the 5-point Laplacian with Dirichlet boundaries. Checked entry by entry (relative
    1e-12); None otherwise."""
    # the entries first: most circuits fail there, without their geometry
    K = scipy.sparse.csc_matrix(K)
    Nf = K.shape[0]
    diag = K.diagonal()
    kappa = float(diag[0]) / 4.0
    if not kappa > 0.0:
        return None
    tol = 1e-12 * kappa
    if np.abs(diag - 4.0 * kappa).max() > tol:
        return None
    if np.count_nonzero(np.abs(K.data + kappa) <= tol) != K.nnz - Nf:
        return None
    grid = _numbered_grid(circuit, K)
    if grid is not None:
        return grid + (kappa,)
    try:
        cx, cy = _face_midpoints(circuit)
    except Exception:
        return None
    if not (np.isfinite(cx).all() and np.isfinite(cy).all()):
        return None
    ix, iy = _grid_index(K, cx), _grid_index(K, cy)
    mx, my = int(ix.max()) + 1, int(iy.max()) + 1
    if mx * my != Nf or K.nnz - Nf != 2 * (mx * (my - 1) + my * (mx - 1)):
        return None
    cell = iy * mx + ix
    grid = np.full(Nf, -1, np.int32)
    grid[cell] = np.arange(Nf, dtype=np.int32)
    if np.any(grid < 0):
        return None
    # every off-diagonal entry couples neighbours: the same row one cell on, or one row on
    r, c = cell[K.indices], np.repeat(cell, np.diff(K.indptr))
    step = np.abs(r - c)
    along = (step == 1) & (np.minimum(r, c) % mx != mx - 1)
    if np.count_nonzero(along | (step == mx) | (step == 0)) != K.nnz:
        return None
    return mx, my, grid, kappa


def _numbered_grid(circuit, K):
    """(mx, my, grid_face) when the faces are numbered line by line (as SquareArray numbers them), from the
    pattern of K alone but for the two faces that tell x from y; else None. 1024x1024: 110 -> 20 ms."""
    Nf = K.shape[0]
    first = K.indices[:K.indptr[1]]     # sorted: face 0, the next one of its line, the next line's
    if not (len(first) == 3 and first[0] == 0 and first[1] == 1):
        return None
    m = int(first[2])
    lines = Nf // m
    if m < 2 or lines * m != Nf or K.nnz - Nf != 2 * (lines * (m - 1) + (lines - 1) * m):
        return None
    i = np.arange(Nf, dtype=K.indices.dtype)
    at = np.empty((Nf, 5), K.indices.dtype)
    there = np.ones((Nf, 5), bool)
    for k, step in enumerate((-m, -1, 0, 1, m)):
        np.add(i, K.indices.dtype.type(step), out=at[:, k])
    there[:m, 0] = there[-m:, 4] = False
    there[::m, 1] = there[m - 1::m, 3] = False
    count = np.full(Nf, 5, K.indptr.dtype)
    count[:m] -= 1
    count[-m:] -= 1
    count[::m] -= 1
    count[m - 1::m] -= 1
    if not (np.array_equal(np.diff(K.indptr), count) and np.array_equal(at[there], K.indices)):
        return None
    try:
        x, y = (np.asarray(v, np.float64) for v in circuit.get_node_coordinates())
        n1, n2 = circuit.get_junction_nodes()
        A = scipy.sparse.csc_matrix(circuit.get_cycle_matrix())

        def middle(f):   # mean of the junction midpoints of face f
            j = np.searchsorted(A.indptr, np.flatnonzero(A.indices == f), side="right") - 1
            return 0.5 * np.array([(v[n1[j]] + v[n2[j]]).mean() for v in (x, y)])

        along, across = middle(1) - middle(0), middle(m) - middle(0)
    except Exception:    # no node coordinates
        return None
    cell = np.arange(Nf, dtype=np.int32).reshape(lines, m)
    for axis in (0, 1):   # the lines along x, or along y
        if abs(along[axis]) > 1e-9 and abs(along[1 - axis]) <= 1e-9 and \
                abs(across[1 - axis]) > 1e-9 and abs(across[axis]) <= 1e-9:
            if along[axis] < 0.0:
                cell = cell[:, ::-1]
            if across[1 - axis] < 0.0:
                cell = cell[::-1]
            if axis == 0:
                return m, lines, np.ascontiguousarray(cell).ravel()
            return lines, m, np.ascontiguousarray(cell.T).ravel()
    return None


def _grid_index(K, v):
    """Index of every face along one axis (int32): on an equally spaced grid from the spacing, the smallest
    difference between coupled faces (without a sort), else by rank."""
    some = K.indptr[min(K.shape[0], 4096)]
    d = np.abs(v[K.indices[:some]] - v[np.repeat(np.arange(min(K.shape[0], 4096)), np.diff(K.indptr[:4097]))])
    d = d[d > 1e-9]
    lo, h = v.min(), d.min(initial=np.inf)
    if np.isfinite(h):
        i = np.rint((v - lo) / h)
        if np.abs(v - (lo + i * h)).max() <= 1e-6 * h:
            return i.astype(np.int32)
    return np.unique(np.round(v, 9), return_inverse=True)[1].astype(np.int32)


def _face_midpoints(circuit):
    """Mean of each face's junction midpoints (for a square, its centre), or of its corners where the
    circuit gives no junction nodes."""
    try:
        x, y = (np.asarray(v, np.float64) for v in circuit.get_node_coordinates())
        n1, n2 = circuit.get_junction_nodes()
        A = scipy.sparse.csc_matrix(circuit.get_cycle_matrix())
        faces, per = A.indices, np.diff(A.indptr)
        count = np.bincount(faces, minlength=A.shape[0])
        mean = lambda v: np.bincount(faces, np.repeat(0.5 * (v[n1] + v[n2]), per), A.shape[0]) / count
        return mean(x), mean(y)
    except Exception:
        cx, cy = circuit.get_face_centroids()
        return np.asarray(cx, np.float64), np.asarray(cy, np.float64)


def _kept_grid(circuit, K, digest):
    """poisson_grid, kept by the digest of K (a grid holds for every circuit with that K; that none was found may
    be for want of coordinates, and is not kept)."""
    with _CACHE_LOCK:
        if digest in _GRIDS:
            _GRIDS.move_to_end(digest)
            return _GRIDS[digest]
    g = poisson_grid(circuit, K)
    if g is not None:
        with _CACHE_LOCK:
            _GRIDS[digest] = g
            while len(_GRIDS) > MAX_GRIDS:
                _GRIDS.popitem(last=False)
    return g


def fast_poisson_grid(circuit, K, digest=None):
    """``poisson_grid`` for the radix-2 transforms: mx + 1 and my + 1 powers of two, up to 1024."""
    g = poisson_grid(circuit, K) if digest is None else _kept_grid(circuit, K, digest)
    return None if g is None or any(m + 1 > 1024 or (m + 1) & m for m in g[:2]) else g


# "auto" uses the radix-2 sine transforms for at most this many problems and face-problems (W x Nf) when
# the caller tunes the sweeps. Measured on GB300 (device ms per step, transforms / sweeps): 256x256 W = 1
# 0.066 / 0.158, 128x128 W = 1 0.031 / 0.082, W = 8 0.092 / 0.142, W = 16 0.168 / 0.163, W = 64
# 0.60 / 0.30; 512x512 W = 1 0.23 / 0.36; 1024x1024 W = 1 0.85 / 0.79, W = 8 6.3 / 2.9; 64x64 W = 64
# 0.150 / 0.129
FAST_POISSON_MAX_W = 8
FAST_POISSON_MAX_WORK = 1 << 18

# Uniform square arrays otherwise (us per step: radix-2 transforms / tensor-core transforms (cut into
# strips above 128 faces a side) / dense blocks; the radix-2 steps take 1.6 us less since their first
# transform forms the face sums):
#   33x33    W = 16   - / 28 / 14      W = 64   - / 29 / 20       W = 256  - / 37 / 42
#   64x64    W = 1   24 / 30 / 22      W = 16  37 / 32 / 28       W = 64  92 / 39 / 43
#   101x60   W = 1    - / 40 / 22      W = 16   - / 38 / 30       W = 64   - / 51 / 54
#   110x110  W = 4    - / 43 / 38      W = 16   - / 44 / 54       W = 64   - / 72 / 116
#   128x128  W = 1   27 / 66 / 49      W = 4   39 / 46 / 53       W = 16 102 / 48 / 65
#   150x150  W = 1    - / 76 / 76      W = 8    - / 82 / 90       W = 64   - / 167 / 238
#   256x256  W = 1   44 / 115 / -      W = 4  124 / 103 / -
# so: dense blocks up to SINE_FROM_WORK face-problems on up to SINE_FROM_FACES faces, tensor-core
# transforms above, radix-2 transforms for a few problems on power-of-two grids.
# The sums of blocks (of the separators between strips too) are added atomically in any order, as the sweeps' split
# dot products are; the transforms repeat bit for bit. So power-of-two grids within FAST_POISSON_MAX_WORK keep
# transforms there, also where the others take less time (radix-2 / others: 32x32 W = 1 20 / 10, W = 8 22 / 12; 64x64
# W = 8 25 / 24; 256x256 W = 4 119 / 100; 512x512 W = 1 133 / 150); from 8192 faces in one strip, where radix2_fits
# ends, the tensor-core ones (128x128 W = 8 60 / 48).
SINE_FROM_WORK = 150000
SINE_FROM_FACES = 1 << 14
SINE_MIN_SIDE = 8
SINE_MAX_SIDE = 4096
SINE_ONE_STRIP = 128     # a side up to which no strips are cut


def radix2_fits(n_faces, W):
    """Whether "auto" tries the radix-2 transforms for W problems (the grid permitting)."""
    return 2048 <= n_faces <= 1 << 17 and W <= (1 if n_faces < 8192 else 4 if n_faces < 1 << 15 else 3)


def sine_solver_fits(grid):
    """Whether "auto" takes the tensor-core sine transforms on this poisson_grid (for any number of problems)."""
    mx, my = grid[:2]
    return SINE_MIN_SIDE <= min(mx, my) and max(mx, my) <= SINE_MAX_SIDE


# Circuits whose state and inverse fit one SM run whole calls in one launch, a block per problem, while
# the problems need few rounds of blocks (304 a round). Measured on GB300 (us per step, one launch per call /
# dense inverse / sweeps): 5x5 nodes W = 1 2.3 / 8.6 / 11.6, W = 512 5.3 / 11.4 / 15.8; 10x10 W = 64 3.2 / 10.9 / 19.3,
# W = 512 8.1 / 12.5 / 39.4, W = 1024 14.5 / 13.3 / 41.4; 13x13 W = 152 5.0 / 11.8 / 31.3, W = 304 10.0 / 12.6 / 57.4,
# W = 512 19.4 / 14.8 / 58.8: the largest circuits are past the crossing with the dense inverse there, the others not
RESIDENT_MAX_FACES = 160
RESIDENT_MAX_JUNCTIONS = 512
RESIDENT_MAX_W = 512


def resident_fits(circuit, W, stencil_width=3):
    """Whether the default plan steps W problems of this circuit in one launch per call. The phase history is
    in shared memory too: with 160 faces and width 5 at most 360 junctions fit, with 158 faces 468."""
    n_faces, n_junctions = circuit._Nf(), circuit._Nj()
    return n_faces <= RESIDENT_MAX_FACES and n_junctions <= RESIDENT_MAX_JUNCTIONS and W <= RESIDENT_MAX_W and \
        bool(N.lib().jja_resident_fits(n_faces, n_junctions, stencil_width))


# Other circuits solve by products with dense blocks on the tensor cores: the whole inverse (leaf 0),
# or the inverses of subtrees of up to `leaf` faces with the separators' Schur complement (3 launches).
# Measured on GB300 (us per step, W problems; sweeps / inverse / leaves of 256):
#   honeycomb 24x24 (1081 faces)   W = 1  48 / 14 / 20    W = 24  58 / 20 / 25    W = 96  103 / 34 / 31
#   honeycomb 31x31 (1830 faces)   W = 1  55 / 17 / 21    W = 24  70 / 27 / 28    W = 96  115 / 63 / 40
#   triangular 64x48 (11970 faces) W = 1  89 / - / 33     W = 24  145 / - / 61    W = 96  240 / - / 145
#   triangular 80x80 (25122 faces) W = 1  97 / - / 66     W = 24  188 / - / 111   W = 256 906 / - / 734
# Larger circuits: leaves of 384 while the problems pay for reading the blocks, else sweeps over subtrees
# with one product for the separators above them (sweeps / leaves of 384 / subtrees of 3072 / of 6144):
#   square 230x200, R spread (45571)   W = 1  142 / 136 / 114 / 121   W = 16  270 / 193 / 227 / 238
#   square 300x300, R spread (89401)   W = 1  201 / 317 / 201 / 190   W = 16  419 / 451 / 365 / 373
#                                                                     W = 64 1213 / 1164 / 985 / 1021
#   square 500x500, R spread (249001)  W = 1  345 / - / 463 / 343     W = 16  984 / - / 1014 / 897
#   24 arrays in one union (274672)    W = 1  351 / - / 320 / 312     8 of them (90876) 167 / - / 155 / 151
# and for many problems, or many small arrays in one union (sweeps / leaves of 256 or 384 / subtrees of 384 /
# of 768 / of 3072):
#   triangular 64x48 (11970)           W = 512  745 / 586 / 631 / 642 / 746     W = 2048 2461 / 2485 / 2121 / 2104 / 2326
#   square 230x200, R spread (45571)   W = 128 1144 / 899 / - / - / 996         W = 512  3220 / 3379 / - / - / 2917
#   28 arrays (73184)                  W = 1  145 / - / 115 / 129 / 139         60 (151102) 196 / - / 215 / 209 / 198
INVERSE_MAX_FACES = 2048
INVERSE_MAX_WORK = 11000    # 128 x 64 blocks of the inverse x problems


def block_leaf(circuit, W):
    """The leaf size of the block solver that the default plan takes for W problems, or None."""
    n = circuit._Nf()
    if n <= INVERSE_MAX_FACES and -(-n // 128) * -(-n // 64) * W <= INVERSE_MAX_WORK:
        return 0
    if n * W > 1 << 24:     # as much data as blocks: their products cost what the sweeps cost
        return None
    if n <= 1 << 15:
        return 256
    return 384 if W >= 8 and n <= 1 << 16 else None


# Unions of many trees: the smallest subtrees with which a step's data stay within the L2 cache: some 0.77 kB a face
# (the sweeps' factor and vectors) and the separators' blocks, 12 bytes an entry or 85 MB x 384 / leaf per 1e9 of the
# trees' squared sizes. us per step of one problem, sweeps / 384 / 768 / 1536 / 3072 / 6144 / 12288 (the sum of squares):
#   35636 faces (0.54e9) 148 / 98 / 106 / 115 / 126 / 134 / 143      64600 (0.70e9) 157 / 154 / 125 / 133 / 134 / 143 / 152
#   61929 (1.45e9) 156 / 192 / 175 / 126 / 134 / 142 / 152            82859 (1.98e9) 158 / 196 / 192 / 175 / 135 / 153 / 155
#   103317 (1.81e9) 168 / 224 / 221 / 191 / 158 / 152 / 168           111999 (1.42e9) 189 / 228 / 225 / 186 / 172 / 186 / 170
# Where none does, a product still pays for large trees (126470 faces, mean 9033: 212 / - / - / 228 / 214 / 197 / 188; 263822,
# mean 10147: 345 / - / - / 310 / 332 / 331 / 329), not for small ones (118320, mean 4732: 168 / - / - / 191 / 181 / 188 / 199).
UNION_LEAVES = (384, 768, 1536, 3072, 6144, 12288)
UNION_CACHE = 90.0       # MB
UNION_LARGE_TREES = 6144

# One tree and few problems, likewise (sweeps / 3072 / 6144 / 12288 / 24576, us per step):
#   45369 faces  W = 1 136 / 113 / 120 / 128 / 136                     53536  W = 1 144 / 172 / 117 / 122 / 131
#   56355        W = 2 146 / 179 / 160 / 125 /  -   W = 4 192 / 183 / 174 / 162
#   65025        W = 1 148 / 187 / 151 / 125 / 134  W = 7 242 / 218 / 207 / 215 / 226
#   68121        W = 1 148 / 200 / 155 / 153 / 136  W = 7 249 / 230 / 218 / 222 / 226
#   89401        W = 1 182 / 197 / 189 / 187 / 175  W = 7 295 / 253 / 250 / 262 / 270
#   128881       W = 1 275 / 243 / 236 / 234 / 243  W = 16 583 / 516 / 514 / 524 / 542
#   358801       W = 16 1348 / 1425 / 1240 / 1212   488601  W = 16 1862 / - / 1967 / 1722   W = 48 6502 / - / 5792
SINGLE_LEAVES = ((46_000, 3072), (54_000, 6144), (66_000, 12288), (100_000, 24576))


def tree_sizes(circuit):
    """Faces of the trees of the circuit's elimination forest: of a ragged union its circuits', else one tree."""
    n = circuit._Nf()
    components = getattr(circuit, "components", 1)
    return getattr(circuit, "tree_faces", None) or (n // components,) * components


def top_leaf(circuit, W):
    """The subtree size below which the default plan keeps the sweeps when block_leaf takes none (a
    product solves the faces above), or None."""
    n, trees = circuit._Nf(), tree_sizes(circuit)
    if n > 1 << 19:
        return None
    if len(trees) > 1 and max(trees) <= 1 << 17:
        squares = sum(t * t for t in trees)
        for leaf in UNION_LEAVES:
            if 0.77e-3 * n + 85e-9 * squares * 384 / leaf <= UNION_CACHE:
                return leaf
        return None if n // len(trees) <= UNION_LARGE_TREES else 12288 if n < 150_000 else 6144
    if n <= 1 << 15:
        return 768
    if n <= 100_000 and W < 8:
        return next(leaf for most, leaf in SINGLE_LEAVES if n <= most) if n <= 66_000 or W < 4 else 6144
    if max(trees) <= 1 << 17:
        return 3072 if n <= 1 << 16 else 6144
    return 6144 if W >= (16 if n <= 400_000 else 32) else None


# Products with explicit inverses (resident steps, dense blocks) are at least as accurate as the sweeps while the
# junctions' weights in K are within this factor of each other. Error of the phase increments (rms, of the sweeps')
# at lognormal spreads of the resistances of 1 (factor 200 to 3000) / 2 (1e6) / 3 (1e8): whole inverse of
# honeycomb 24x24 0.6 / 0.8 / 3.7, leaves of 64x64 0.5 / 0.8 / 6, 10x10 resident 0.4 / 1.0 / 6; one junction of 1e3
# times the others' resistance on 10x10: 3.3.
EVEN_WEIGHTS = 256.0


def even_weights(circuit, dt):
    """Whether no junction's weight 1 / (Cv + Rv), nor that plus its inductance, is more than EVEN_WEIGHTS times
    another's."""
    w = 1.0 / (np.asarray(circuit._C(), np.float64) / dt ** 2 + 1.0 / (dt * np.asarray(circuit._R(), np.float64)))
    L = circuit._L()
    w_L = w + (np.asarray(L.diagonal()) if scipy.sparse.issparse(L) else np.diag(np.asarray(L)))
    return all(bool(v.min() > 0.0 and v.max() <= EVEN_WEIGHTS * v.min()) for v in (w, w_L))


def untuned(tuning):
    """True when ``tuning`` asks for nothing but the level schedule (the library's default)."""
    t = dict(tuning or {})
    return int(t.pop("schedule", 0)) in (0, 1) and not any(int(v) for v in t.values())


class DevicePlan:
    """Circuit tables + factor uploaded for W problems (owned C object)."""

    def __init__(self, circuit, factor, A, W, dt, stencil_width, stencil, Ic_w=None, tuning=None, fast_poisson=None,
                 sine=None, resident=False, blocks=None, top=None):
        """``tuning``: dict with any of rhs_block, rows_per_lane, target_warps, min_piece (the
        launch shape of the triangular solves; missing or 0 = library default)."""
        Nj, Nf = circuit._Nj(), circuit._Nf()
        Rv, Cv, coef = coefficients(circuit, dt, stencil)
        Acsr = scipy.sparse.csr_matrix(A)
        Acsr.sort_indices()
        self._keep = dict(
            rowptr=np.ascontiguousarray(Acsr.indptr, np.int64),
            col=np.ascontiguousarray(Acsr.indices, np.int32),
            val=np.ascontiguousarray(Acsr.data, np.float64),
            Ic=np.ascontiguousarray(circuit._Ic(), np.float64),
            Ic_w=None if Ic_w is None else np.ascontiguousarray(Ic_w, np.float64),
            inv_c0=np.ascontiguousarray(1.0 / coef[0], np.float64),
            coef=np.ascontiguousarray(np.stack(coef[1:]), np.float64),
            Rv=np.ascontiguousarray(Rv, np.float64))
        k = self._keep
        ex = (ctypes.c_double * 4)(*(list(EXTRAP[stencil_width]) + [0.0] * (4 - len(EXTRAP[stencil_width]))))
        d = N.PlanDesc(Nj, Nf, W, stencil_width, N.ptr(k["rowptr"], ctypes.c_int64), N.ptr(k["col"], ctypes.c_int32),
                       N.ptr(k["val"]), N.ptr(k["Ic"]), N.ptr(k["inv_c0"]), N.ptr(k["coef"]), N.ptr(k["Rv"]), ex, dt,
                       N.ptr(k["Ic_w"]))
        tuning = dict(tuning or {})
        unknown = set(tuning) - set(TUNING_FIELDS)
        if unknown:
            raise ValueError(f"unknown tuning fields {sorted(unknown)}; expected {TUNING_FIELDS}")
        d.tuning = N.SolveTuning(*(int(tuning.get(f, 0)) for f in TUNING_FIELDS))
        self.tuning = {f: int(tuning.get(f, 0)) for f in TUNING_FIELDS}
        h = ctypes.c_void_p()
        N.check(N.lib().jja_plan_create(ctypes.byref(d), factor.handle, ctypes.byref(h)))
        self.handle = h
        self.Nj, self.Nf, self.W = Nj, Nf, W
        self.inv_c0 = k["inv_c0"]
        self.fast_poisson = False
        if fast_poisson is not None:
            mx, my, grid, kappa = fast_poisson
            self._keep["grid"] = grid
            N.check(N.lib().jja_plan_set_fast_poisson(h, int(mx), int(my), N.ptr(grid, ctypes.c_int32), float(kappa)))
            self.fast_poisson = True
        # a solver that is too large for the circuit, or for the memory left, leaves the plan with its sweeps
        self.sine = self.resident = False
        self.blocks = self.top = None
        try:
            if sine is not None:
                mx, my, grid, kappa = sine
                self._keep["grid"] = grid
                N.check(N.lib().jja_plan_set_sine_solver(h, int(mx), int(my), N.ptr(grid, ctypes.c_int32), float(kappa)))
                self.sine = True
            elif resident:
                N.check(N.lib().jja_plan_set_resident(h, factor.handle))
                self.resident = True
            elif blocks is not None:
                N.check(N.lib().jja_plan_set_blocks(h, factor.handle, int(blocks)))
                self.blocks = blocks
            elif top is not None:
                N.check(N.lib().jja_plan_set_top_block(h, factor.handle, int(top)))
                self.top = top
        except N.JJAError as e:
            if e.code != N.ERR_UNFIT and "out of memory" not in str(e):
                raise
        self.device_bytes = N.lib().jja_plan_device_bytes(h)

    def solve(self, b_dev, x_dev, stream=0):
        N.check(N.lib().jja_solve(self.handle, ctypes.c_void_p(b_dev), ctypes.c_void_p(x_dev), ctypes.c_void_p(stream)))

    def check(self):
        """Synchronise the device; raise JJAError if a wait of a dataflow sweep ran out of its
        bound since the last check (the steps since then are invalid)."""
        t = ctypes.c_int(0)
        N.check(N.lib().jja_plan_check(self.handle, ctypes.byref(t)))
        if t.value:
            raise N.JJAError(5, "a bounded wait of a dataflow or cooperative sweep ran out of its bound; "
                                "results are invalid")

    def eval_sin(self, x_dev, out_dev, n, stream=0):
        N.check(N.lib().jja_eval_sin(self.handle, ctypes.c_void_p(x_dev), ctypes.c_void_p(out_dev), int(n),
                                     ctypes.c_void_p(stream)))

    def __del__(self):
        h = getattr(self, "handle", None)
        if h is not None and N._lib is not None:
            N._lib.jja_plan_destroy(h)
            self.handle = None


def _coords(circuit):
    try:
        cx, cy = circuit.get_face_centroids()
        return np.asarray(cx, np.float64), np.asarray(cy, np.float64)
    except Exception:
        return None


MMD_MIN_WORK = 1 << 22     # "auto" picks minimum degree from this many face-problems (W x Nf) ...
MMD_MAX_FACES = 1 << 18    # ... on up to this many faces (its order comes from a host SuperLU run)


def resolve_ordering(ordering, W, n_faces):
    """The fill-reducing order "auto" stands for. When a step has a lot of work (W x Nf >= 2^22)
    the sweeps are FP64-bound, and minimum degree's factor has about 30 % fewer values than
    nested dissection's on 2D lattices (measured on GB300: 4 % less time per step for
    512 x SquareArray(128, 128)). With less work they are latency-bound, and nested dissection's
    tree has half the levels (64 x SquareArray(64, 64): minimum degree 54 % slower)."""
    if ordering == "auto":
        return "mmd" if W * n_faces >= MMD_MIN_WORK and n_faces <= MMD_MAX_FACES else "nd"
    return ordering


SMALL_STEP_FACES = 1 << 15   # W x Nf up to which "auto" factors with large leaves and strong amalgamation


def resolve_factor_shape(nd_leaf, relax, ordering, W, n_faces):
    """(nd_leaf, relax) that ``nd_leaf=None`` stands for. A step of few face-problems
    (W x Nf <= 2^15, nested dissection, default amalgamation) is bound by the elimination tree's
    depth: every level of each sweep is a chain of dependent memory round trips (about 3.5 us on
    GB300), and the flops are negligible. Such steps factor with nested-dissection leaves of 128
    faces and merge supernodes that add at most 256 zeros or 50 %: fewer, denser levels. Measured
    (W = 1, graph-replayed steps): SquareArray(10,10) 0.029 -> 0.014 ms/step (one dense
    supernode), SquareArray(128,128) 0.113 -> 0.081 ms; at 256x256 the larger factor costs more
    than the levels it saves (0.165 -> 0.205 ms), so larger steps keep leaves of 8."""
    if nd_leaf is not None:
        return nd_leaf, relax
    if ordering == "nd" and tuple(relax) == (-1, -1.0) and W * n_faces <= SMALL_STEP_FACES:
        return 128, (256, 0.5)
    return 8, relax


def fill_reducing_order(K, ordering, circuit=None):
    """(coords, perm) for HostFactor. "nd": the library's nested dissection on face centroids;
    "mmd": the multiple-minimum-degree column order scipy's SuperLU computes on A + A^T
    (less fill on 2D lattices, deeper elimination tree)."""
    if ordering == "nd":
        return (_coords(circuit) if circuit is not None else None), None
    if ordering == "mmd":
        import scipy.sparse.linalg
        lu = scipy.sparse.linalg.splu(K.tocsc(), permc_spec="MMD_AT_PLUS_A", diag_pivot_thresh=0.0,
                                      options=dict(SymmetricMode=True))
        return None, np.argsort(lu.perm_c).astype(np.int32)
    raise ValueError(f"ordering must be 'nd' or 'mmd', not {ordering!r}")


def get_factor(circuit, dt, nd_leaf=8, ordering="nd", relax=(-1, -1.0), matrices=None, digest=None):
    """(factor, A, cache key); ``matrices``: face_matrix(circuit, dt), ``digest``: of its K, when the caller has them."""
    A, K = face_matrix(circuit, dt) if matrices is None else matrices
    key = (_digest(K.indptr, K.indices, K.data) if digest is None else digest, nd_leaf, ordering, tuple(relax))
    with _CACHE_LOCK:
        hit = _FACTORS.get(key)
        if hit is not None:
            _FACTORS.move_to_end(key)
            return hit[0], A, key
    coords, perm = fill_reducing_order(K, ordering, circuit)
    f = HostFactor(K, coords=coords, perm=perm, nd_leaf=nd_leaf, relax_zeros=relax[0], relax_frac=relax[1])
    with _CACHE_LOCK:
        _FACTORS[key] = (f, A)
        while len(_FACTORS) > MAX_FACTORS:
            _FACTORS.popitem(last=False)
    return f, A, key


def get_plan(circuit, dt, W, stencil_width, stencil, nd_leaf=None, ordering="auto", relax=(-1, -1.0), Ic_w=None,
             tuning=None, fast_poisson="auto"):
    """Device plan for W problems; ``Ic_w`` (Nj, W) gives each problem its own critical currents;
    ``ordering`` "nd", "mmd" or "auto" (see resolve_ordering); ``nd_leaf`` None: by the step's
    size (see resolve_factor_shape); ``tuning`` the launch shape of the triangular solves (see
    DevicePlan); ``fast_poisson``: solve with sine transforms when the face-space matrix allows it
    (fast_poisson_grid): True (radix-2 grids), False (the sweeps), or "auto": unless ``tuning`` asks for
    sweeps of some shape, whichever of the resident steps (resident_fits), the radix-2 or tensor-core
    transforms, the dense blocks (block_leaf) and the dense top block (top_leaf) is fastest for the circuit
    and W (resident steps and blocks for circuits of even_weights only)."""
    matrices = A, K = face_matrix(circuit, dt)
    digest = _digest(K.indptr, K.indices, K.data)
    n_faces = circuit._Nf()
    Rv, Cv, coef = coefficients(circuit, dt, stencil)
    if Ic_w is not None:
        Ic_w = np.ascontiguousarray(np.broadcast_to(np.asarray(Ic_w, np.float64), (circuit._Nj(), W)))
    ic = np.asarray(circuit._Ic(), np.float64) if Ic_w is None else Ic_w
    tkey = tuple(int((tuning or {}).get(f, 0)) for f in TUNING_FIELDS)
    tables = (W, stencil_width, Ic_w is None, tkey, _digest(ic, *coef, Rv, A.indptr, A.indices, A.data))
    asked = (digest, nd_leaf, ordering, tuple(relax), fast_poisson, tree_sizes(circuit)) + tables
    with _CACHE_LOCK:
        p = _PLANS.get(_ROUTES.get(asked))
        if p is not None:
            _PLANS.move_to_end(_ROUTES[asked])
            return p
    fp = sine = blocks = top = None
    auto = fast_poisson == "auto" and untuned(tuning)
    resident = auto and resident_fits(circuit, W, stencil_width) and even_weights(circuit, dt)
    if fast_poisson is True or (auto and not resident and radix2_fits(n_faces, W)) or \
            (fast_poisson == "auto" and not auto and W <= FAST_POISSON_MAX_W and W * n_faces <= FAST_POISSON_MAX_WORK):
        fp = fast_poisson_grid(circuit, K, digest)
    if auto and not resident and fp is None:
        if W * n_faces > SINE_FROM_WORK or n_faces > SINE_FROM_FACES:
            sine = _kept_grid(circuit, K, digest)
            if sine is not None and not sine_solver_fits(sine):
                sine = None
        if sine is None:
            blocks = block_leaf(circuit, W)
            top = top_leaf(circuit, W) if blocks is None else None
            if blocks is not None and not even_weights(circuit, dt):
                blocks = None
        repeats = sine is not None and min(sine[:2]) <= SINE_ONE_STRIP
        if not repeats and W <= FAST_POISSON_MAX_W and W * n_faces <= FAST_POISSON_MAX_WORK:
            grid = fast_poisson_grid(circuit, K, digest)
            if grid is not None:
                blocks = top = None
                strips = min(grid[:2]) > SINE_ONE_STRIP
                fp, sine = (grid, None) if strips or n_faces < 8192 else (None, grid)
    if blocks is not None:     # the block solver cuts the tree itself: nested dissection with small leaves
        nd_leaf = 8 if nd_leaf is None else nd_leaf
        ordering = "nd" if ordering == "auto" else ordering
    ordering = resolve_ordering(ordering, W, n_faces)
    nd_leaf, relax = resolve_factor_shape(nd_leaf, relax, ordering, W, n_faces)
    factor, A, fkey = get_factor(circuit, dt, nd_leaf, ordering=ordering, relax=relax, matrices=matrices, digest=digest)
    key = (fkey, fp is not None, sine is not None, resident, blocks, top) + tables
    with _CACHE_LOCK:
        p = _PLANS.get(key)
        if p is not None:
            _PLANS.move_to_end(key)
    if p is None:
        p = DevicePlan(circuit, factor, A, W, dt, stencil_width, stencil, Ic_w=Ic_w, tuning=tuning, fast_poisson=fp,
                       sine=sine, resident=resident, blocks=blocks, top=top)
        p.ordering = ordering     # the order its factor has
    with _CACHE_LOCK:
        _PLANS[key] = p
        _ROUTES[asked] = key
        while len(_PLANS) > MAX_PLANS:
            _PLANS.popitem(last=False)
        while len(_ROUTES) > MAX_ROUTES:
            _ROUTES.popitem(last=False)
    return p


def clear_cache():
    with _CACHE_LOCK:
        _PLANS.clear()
        _ROUTES.clear()
        _FACTORS.clear()
        _GRIDS.clear()
