"""Timed cases of the sparse LU engine: what a circuit or power-grid simulator has it do.

Each case is one call sequence of the C ABI (include/glu_b200.h, through the
package's ctypes binding) on a synthetic matrix of the repository's generators:

* ``nodal``:  nodal analysis, two band links (|i-j| <= 16) and one uniform long
  link per node, 5 % unsymmetric rows; after a minimum-degree ordering its fill
  ends in a dense trailing block of about a third of the columns;
* ``linked``: the wider one of the batches, band 32, two long links per node,
  10 % unsymmetric rows; half of its columns end in the dense block;
* ``mesh``:   a side x side resistive power grid with long couplings, ordered
  by nested dissection, the couplings' nodes last; many levels of small
  supernodes, then a moderate dense block.

The pattern of a case is fixed by its family and size, as a simulator's netlist
is; values and right-hand sides come from the seed.  Host-side analysis of a
pattern (ordering, symbolic phase) is kept for the process, a handle belongs to
one state.  The matrices are scaled symmetrically by the first values'
diagonal, with scales that later values of the pattern keep, as a
refactorization does.
"""
import ctypes
import functools
import heapq
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "glu-hcu_b200"))
from pyglu import _capi, synth  # noqa: E402

HOST, DEVICE = _capi.GLU_HOST, _capi.GLU_DEVICE
STREAMS = 16  # of a call over many systems, pyglu.UnevenBatch's default


# ------------------------------------------------------------------- cases --
def listed():
    return [
        # The smallest call in earnest: a sub-circuit inside a transient loop,
        # new values and one FP32 solve per time step, everything on the GPU.
        dict(name="step_small", family="nodal", size=300, task="step", sets=1, nrhs=1),
        # The plain form's headline circuit: new values, FP32 factors handed
        # back (what LUonDevice gives its caller), no solve.
        dict(name="refactor_nodal", family="nodal", size=4960, task="refactor", sets=1, perturb=0),
        # The same with the perturbation of tiny pivots, at an odd size.
        dict(name="refactor_perturb", family="nodal", size=2777, task="refactor", sets=1, perturb=1),
        # A Newton iteration through host arrays, as pyglu's refactor and
        # solve(refine=True) make it.
        dict(name="newton_host", family="nodal", size=4960, task="newton", sets=1, nrhs=1, host=1, tol=1e-10),
        # Many right-hand sides against kept factors (transfer functions, port
        # by port), FP32.
        dict(name="solve_ports", family="nodal", size=4960, task="solve", nrhs=32),
        # One right-hand side against kept factors of a power grid (the time
        # step of a linear transient analysis), FP32.
        dict(name="solve_grid", family="mesh", size=251, task="solve", nrhs=1),
        # The adjoint solve behind pyglu.sparse_solve's backward: A^T, refined.
        dict(name="adjoint", family="nodal", size=9973, task="adjoint", nrhs=1, tol=1e-10),
        # A medium power grid: refactor and refined solve.
        dict(name="newton_grid", family="mesh", size=300, task="newton", sets=1, nrhs=1, host=0, tol=1e-10),
        # The largest power grid, n = 490,000.
        dict(name="newton_grid_large", family="mesh", size=700, task="newton", sets=1, nrhs=1, host=0, tol=1e-10),
        # A parameter sweep: many value sets of a small circuit at once.
        dict(name="sweep_small", family="nodal", size=1500, task="newton", sets=96, nrhs=1, host=0, tol=1e-10),
        # The batch's pattern, n = 20,000, four right-hand sides per value set.
        dict(name="sweep_linked", family="linked", size=20000, task="newton", sets=12, nrhs=4, host=0, tol=1e-10),
        # Independent circuits of uneven sizes with 1 to 64 right-hand sides,
        # through host arrays.
        dict(name="systems", family="nodal", size=9000, least=2000, count=10, task="systems", tol=1e-10),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the same tasks over the ranges between the listed ones."""
    task = rng.choice(["step", "refactor", "newton", "newton", "solve", "adjoint", "sweep", "sweep", "systems"])
    family = rng.choice(["nodal", "mesh"])
    size = _log_int(rng, 300, 9973) if family == "nodal" else _log_int(rng, 20, 700)
    if task == "step":
        return dict(family=family, size=size, task="step", sets=1, nrhs=rng.choice([1, 1, 2, 3]))
    if task == "refactor":
        return dict(family=family, size=size, task="refactor", sets=1, perturb=rng.randint(0, 1))
    if task == "newton":
        return dict(family=family, size=size, task="newton", sets=1, nrhs=rng.choice([1, 1, 2, 5]),
                    host=rng.randint(0, 1), tol=1e-10)
    if task == "solve":
        return dict(family=family, size=size, task="solve", nrhs=_log_int(rng, 1, 64))
    if task == "adjoint":
        return dict(family=family, size=size, task="adjoint", nrhs=rng.randint(1, 3),
                    tol=1e-10)
    if task == "sweep":
        family = rng.choice(["nodal", "linked"])
        size = _log_int(rng, 500, 4960)
        return dict(family=family, size=size, task="newton", sets=rng.randint(2, max(3, min(96, 150000 // size))),
                    nrhs=rng.randint(1, 4), host=0, tol=1e-10)
    return dict(family="nodal", size=_log_int(rng, 4000, 9000), least=2000, count=rng.randint(3, 10), task="systems",
                tol=1e-10)


def _systems(case):
    """(size, right-hand sides) of every system: sizes spread over their logarithm."""
    k = case["count"]
    return [(int(round(case["least"] * (case["size"] / case["least"]) ** (i / max(1, k - 1)))), 1 + (37 * i) % 64)
            for i in range(k)]


# ---------------------------------------------------------------- patterns --
def _min_degree(n, rows, cols):
    """Minimum-degree order of the symmetrised pattern (quotient graph, bounds
    of the degrees); stops where the rest is about to be dense."""
    off = rows != cols
    edge = np.unique(np.concatenate([cols[off] * n + rows[off], rows[off] * n + cols[off]]))
    ptr = np.searchsorted(edge, np.arange(n + 1, dtype=np.int64) * n).tolist()
    nbr = (edge % n).tolist()
    var = [set(nbr[ptr[i]:ptr[i + 1]]) for i in range(n)]  # uneliminated neighbours
    elt = [set() for _ in range(n)]                        # eliminated cliques it is in
    clique = {}
    deg = [len(v) for v in var]
    heap = [(d, i) for i, d in enumerate(deg)]
    heapq.heapify(heap)
    order, left = [], n
    while heap:
        d, p = heapq.heappop(heap)
        if var[p] is None or d != deg[p]:
            continue
        if 2 * d >= left:
            break
        lp, gone = var[p], elt[p]
        for e in gone:
            lp |= clique.pop(e)
        lp.discard(p)
        outside = {}
        for i in lp:
            elt[i] -= gone
            for e in elt[i]:
                outside[e] = outside.get(e, len(clique[e])) - 1
        order.append(p)
        left -= 1
        for i in lp:
            var[i] -= lp
            var[i].discard(p)
            d = len(lp) - 1 + len(var[i]) + sum(outside[e] for e in elt[i])
            elt[i].add(p)
            d = min(d, left - 1, deg[i] + len(lp) - 1)
            if d != deg[i]:
                deg[i] = d
                heapq.heappush(heap, (d, i))
        clique[p] = lp
        var[p] = elt[p] = None
    rest = sorted((i for i in range(n) if var[i] is not None), key=lambda i: (deg[i], i))
    return np.array(order + rest, dtype=np.int64)


def _dissection(side, rows, cols):
    """Nested dissection of a side x side grid; one node of each long coupling goes last."""
    gap = np.abs(rows - cols)
    last = np.unique(np.minimum(rows, cols)[(gap > 1) & (gap != side)])
    out = []

    def cut(a):
        h, w = a.shape
        if h < w:
            a, h, w = a.T, w, h
        if h <= 3:
            out.append(a.ravel())
            return
        m = h // 2
        cut(a[:m])
        cut(a[m + 1:])
        out.append(a[m])

    cut(np.arange(side * side, dtype=np.int64).reshape(side, side))
    o = np.concatenate(out)
    keep = np.ones(side * side, bool)
    keep[last] = False
    return np.concatenate([o[keep[o]], last])


class Pattern:
    """A netlist's pattern: first values, ordering, scaling, symbolic phase."""

    def __init__(self, family, size):
        if family == "mesh":
            A = synth.grid_mesh(size, seed=0, n_long=max(1, 2000 * size * size // 490000))
        elif family == "linked":
            A = synth.config2_pattern(seed=0, n=size)
        else:
            A = synth.nodal(size, seed=0)
        self.data, self.indices, self.indptr, n = A
        self.n = n
        self.rows = self.indices.astype(np.int64)
        self.cols = np.repeat(np.arange(n, dtype=np.int64), np.diff(self.indptr))
        order = (_dissection(size, self.rows, self.cols) if family == "mesh"
                 else _min_degree(n, self.rows, self.cols))
        self.new = np.empty(n, np.int64)
        self.new[order] = np.arange(n)
        diag = np.ones(n)
        on = self.rows == self.cols
        diag[self.rows[on]] = self.data[on]
        d = 1.0 / np.sqrt(np.abs(diag))
        self.scale = d[self.rows] * d[self.cols]
        self.d = d
        # the permuted matrix, and every entry's place in it
        place = np.lexsort((self.new[self.rows], self.new[self.cols]))
        self.ai = np.ascontiguousarray(self.new[self.rows][place], dtype=np.uint32)
        self.ap = np.zeros(n + 1, np.uint32)
        self.ap[1:] = np.cumsum(np.bincount(self.new[self.cols], minlength=n))
        eng, ptr = _capi.engine(), _capi.ptr
        self.sym = ctypes.c_void_p()
        _capi.check(eng.glu_symbolic_analyze(n, self.ai.size, ptr(self.ap), ptr(self.ai), ctypes.byref(self.sym)))
        nnz = ctypes.c_uint32()
        eng.glu_symbolic_sizes(self.sym, None, ctypes.byref(nnz))
        self.nnz_lu = nnz.value
        slots = np.empty(self.ai.size, np.uint32)
        eng.glu_symbolic_slots(self.sym, ptr(slots))
        self.slot = np.empty_like(slots)
        self.slot[place] = slots
        self.transform = (order.astype(np.uint32), self.new.astype(np.uint32), np.arange(n, dtype=np.int32),
                          np.ascontiguousarray(d[order]), d)

    def layout(self):
        """(row, column) of every LU value, in the permuted matrix."""
        cp, ri = np.empty(self.n + 1, np.uint32), np.empty(self.nnz_lu, np.uint32)
        _capi.engine().glu_symbolic_export(self.sym, _capi.ptr(cp), _capi.ptr(ri), None, None, None, None)
        return ri.astype(np.int64), np.repeat(np.arange(self.n, dtype=np.int64), np.diff(cp.astype(np.int64)))

    def handle(self, sets):
        eng, ptr = _capi.engine(), _capi.ptr
        h = ctypes.c_void_p()
        _capi.check(eng.glu_create(self.sym, 0, sets, ctypes.byref(h)))
        _capi.check(eng.glu_set_transform(h, *(ptr(a) for a in self.transform), 1))
        ap, ai = self.indptr.astype(np.uint32), self.indices.astype(np.uint32)
        _capi.check(eng.glu_set_source(h, self.indices.size, ptr(ap), ptr(ai), ptr(self.slot), ptr(self.scale)))
        return h

    @functools.lru_cache(maxsize=1)
    def flops(self):
        """Of one factorization: sum over the columns of |L| + 2 |L| |U|."""
        cp, rp, dp, rd = (np.empty(self.n + 1, np.uint32), np.empty(self.n + 1, np.uint32),
                          np.empty(self.n, np.uint32), np.empty(self.n, np.uint32))
        _capi.engine().glu_symbolic_export(self.sym, _capi.ptr(cp), None, _capi.ptr(dp), _capi.ptr(rp), None,
                                           _capi.ptr(rd))
        low = cp[1:].astype(np.float64) - dp - 1
        up = rp[1:].astype(np.float64) - rd - 1
        return float((low + 2 * low * up).sum())


@functools.lru_cache(maxsize=24)
def _pattern(family, size):
    return Pattern(family, size)


def _values(pat, sets, seed, transient=False):
    """Value sets of the pattern; ``transient``: with the capacitors' companion conductances of
    a time step (1 to 10 % of the diagonal), without: the DC matrix of a Newton iteration,
    whose FP32 solutions need the refinement."""
    v = synth.perturb_values(pat.data, pat.indices, pat.indptr, pat.n, sets, seed=seed)
    if transient:
        on = pat.rows == pat.cols  # every diagonal entry is there
        v[:, on] *= 1.0 + np.exp(np.random.default_rng(seed + 5).uniform(np.log(1e-2), np.log(1e-1), (sets, pat.n)))
    return v


def _transient(case):
    return case["task"] in ("step", "solve", "refactor")


def _rhs(case, n, sets, nrhs, seed):
    """Right-hand sides (sets, nrhs, n): loads on a grid, uniform in [-1, 1] on a circuit."""
    if case["family"] == "mesh":
        return np.stack([synth.rhs_loads(n, seed=seed + 1000 * k) for k in range(sets * nrhs)]).reshape(sets, nrhs, n)
    return synth.rhs_uniform(n, sets * nrhs, seed=seed).reshape(sets, nrhs, n)


# ------------------------------------------------------------------ states --
class State:
    """Handles, inputs and output buffers of one case; the handles end with it."""

    def __init__(self, **kw):
        self.__dict__.update(kw)

    def __del__(self):
        for h in getattr(self, "handles", ()):
            _capi.engine().glu_destroy(h)


def _address(a):
    return ctypes.c_void_p(a.data_ptr()) if isinstance(a, torch.Tensor) else _capi.ptr(a)


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def prepare(case, seed):
    task = case["task"]
    if task == "systems":
        sysd = _systems(case)
        pats = [_pattern(case["family"], n) for n, _ in sysd]
        values = [_values(p, 1, seed + 7 * i)[0] for i, p in enumerate(pats)]
        b = [_rhs(case, p.n, 1, k, seed + 7 * i + 3)[0] for i, (p, (_, k)) in enumerate(zip(pats, sysd))]
        return State(task=task, handles=[p.handle(1) for p in pats], values=values, b=b, tol=case["tol"],
                     streams=[torch.cuda.Stream() for _ in range(min(STREAMS, len(pats)))])
    pat = _pattern(case["family"], case["size"])
    sets, nrhs, host = case.get("sets", 1), case.get("nrhs", 1), case.get("host", 0)
    s = State(task=task, handles=[pat.handle(sets)], sets=sets, nrhs=nrhs, host=host, tol=case.get("tol", 0.0),
              perturb=case.get("perturb", 0))
    s.values = _values(pat, sets, seed, _transient(case))
    s.b = _rhs(case, pat.n, sets, nrhs, seed + 1)
    if not host:
        s.values, s.b = torch.from_numpy(s.values).cuda(), torch.from_numpy(s.b).cuda()
        if task in ("step", "solve"):
            s.b = s.b.float()
        s.x = torch.empty_like(s.b)
    if task == "refactor":
        s.lu = torch.empty(sets, pat.nnz_lu, dtype=torch.float32, device="cuda")
    if task in ("solve", "adjoint"):  # the factors are there already
        _refactor(s)
    return s


def _refactor(s):
    eng, where = _capi.engine(), HOST if s.host else DEVICE
    _capi.check(eng.glu_load_source_values(s.handles[0], 0, s.sets, _address(s.values), where, _stream()))
    _capi.check(eng.glu_factor(s.handles[0], 0, s.sets, s.perturb, _stream()))


def _run_systems(s):
    eng, k, ns = _capi.engine(), len(s.handles), len(s.streams)
    streams = (ctypes.c_void_p * ns)(*[q.cuda_stream for q in s.streams])
    for i, (h, v) in enumerate(zip(s.handles, s.values)):
        _capi.check(eng.glu_load_source_values(h, 0, 1, _capi.ptr(v), HOST, ctypes.c_void_p(streams[i % ns])))
    handles = (ctypes.c_void_p * k)(*[h.value for h in s.handles])
    _capi.check(eng.glu_factor_many(k, handles, 0, streams, ns))
    x = [np.empty_like(b) for b in s.b]
    _capi.check(eng.glu_solve_refined_many(
        k, handles, (ctypes.c_uint32 * k)(*[b.shape[0] for b in s.b]),
        (ctypes.c_void_p * k)(*[b.ctypes.data for b in s.b]), (ctypes.c_void_p * k)(*[a.ctypes.data for a in x]),
        s.tol, 10, HOST, (_capi.RefineStats * k)(), streams, ns))
    return x


def run(s):
    eng = _capi.engine()
    if s.task == "systems":
        return _run_systems(s)
    h = s.handles[0]
    if s.task in ("step", "refactor", "newton"):
        _refactor(s)
    if s.task == "refactor":
        _capi.check(eng.glu_store_lu_values(h, 0, s.sets, _address(s.lu), DEVICE, _stream()))
        return s.lu
    if s.task in ("step", "solve"):
        _capi.check(eng.glu_solve(h, 0, s.nrhs, _address(s.b), _address(s.x), DEVICE, _stream()))
        return s.x
    x = np.empty_like(s.b) if s.host else s.x
    stats = _capi.RefineStats()
    _capi.check(eng.glu_solve_refined(h, 0, s.sets, s.nrhs, _address(s.b), _address(x), s.tol, 10,
                                      int(s.task == "adjoint"), HOST if s.host else DEVICE, ctypes.byref(stats),
                                      _stream()))
    return x


# -------------------------------------------------------------- comparison --
def work(case):
    """Values, factors, right-hand sides and solutions once; a refined solve is
    one FP32 solve, one FP64 residual and one correction."""
    one = [(_pattern(case["family"], n), k) for n, k in _systems(case)] if case["task"] == "systems" else \
        [(_pattern(case["family"], case["size"]), case.get("nrhs", 0))]
    task, sets = case["task"], case.get("sets", 1)
    byt = flo = 0.0
    for p, k in one:
        if task not in ("solve", "adjoint"):
            byt += 8.0 * p.data.size + 4.0 * p.nnz_lu
            flo += p.flops()
        if task in ("solve", "adjoint"):
            byt += 4.0 * p.nnz_lu
        if task in ("step", "solve"):
            byt += 8.0 * k * p.n
            flo += 2.0 * k * p.nnz_lu
        elif task != "refactor":
            byt += 16.0 * k * p.n + 8.0 * p.data.size
            flo += k * (4.0 * p.nnz_lu + 2.0 * p.data.size)
    return {"bytes": byt * sets, "flops": flo * sets}


def _dense(pat, values, scaled):
    """The matrix as a dense FP64 tensor: as given, or scaled and permuted."""
    r, c = (pat.new[pat.rows], pat.new[pat.cols]) if scaled else (pat.rows, pat.cols)
    A = torch.zeros(pat.n, pat.n, dtype=torch.float64, device="cuda")
    v = values * pat.scale if scaled else values
    A[torch.from_numpy(r).cuda(), torch.from_numpy(c).cuda()] = torch.from_numpy(v).cuda()
    return A


def _solve_grid(pat, side, values, b):
    """The grid's rows are a block tridiagonal matrix once the nodes that the long couplings end
    in are set apart: block elimination with those nodes' columns as further right-hand sides,
    then their Schur complement."""
    n, dev = pat.n, "cuda"
    rows, cols, v = (torch.from_numpy(a).to(dev) for a in (pat.rows, pat.cols, values))
    gap = np.abs(pat.rows - pat.cols)
    last = torch.from_numpy(np.unique(np.minimum(pat.rows, pat.cols)[(gap > 1) & (gap != side)])).to(dev)
    k = last.numel()
    at = torch.full((n,), -1, dtype=torch.long, device=dev)
    at[last] = torch.arange(k, device=dev)
    inner = (at[rows] < 0) & (at[cols] < 0)
    blocks = torch.zeros(3, side, side, side, dtype=torch.float64, device=dev)  # left, diagonal, right of each row
    r, c = rows[inner], cols[inner]
    blocks[c // side - r // side + 1, r // side, r % side, c % side] = v[inner]
    blocks[1, last // side, last % side, last % side] = 1.0
    rhs = torch.zeros(n, k + b.shape[0], dtype=torch.float64, device=dev)
    up = (at[rows] < 0) & (at[cols] >= 0)
    rhs[rows[up], at[cols[up]]] = v[up]
    rhs[:, k:] = torch.from_numpy(b).to(dev).T
    rhs[last, k:] = 0.0
    rhs = rhs.reshape(side, side, -1)
    factors = []
    for i in range(side):
        d = blocks[1, i]
        if i:
            w = torch.linalg.lu_solve(*factors[-1], blocks[0, i], left=False)
            d = d - w @ blocks[2, i - 1]
            rhs[i] -= w @ rhs[i - 1]
        factors.append(torch.linalg.lu_factor(d))
    for i in reversed(range(side)):
        if i + 1 < side:
            rhs[i] -= blocks[2, i] @ rhs[i + 1]
        rhs[i] = torch.linalg.lu_solve(*factors[i], rhs[i])
    rhs = rhs.reshape(n, -1)
    low = at[rows] >= 0
    border = torch.zeros(k, n, dtype=torch.float64, device=dev)
    border[at[rows[low]], cols[low]] = v[low]
    full = torch.from_numpy(b).to(dev).T[last]
    y = border.clone()
    y[:, last] = 0.0
    schur = border[:, last] - y @ rhs[:, :k]
    xl = torch.linalg.solve(schur, full - y @ rhs[:, k:])
    x = rhs[:, k:] - rhs[:, :k] @ xl
    x[last] = xl
    return x.T.contiguous().cpu().numpy()


def _exact_x(case, pat, values, b):
    if case["family"] == "mesh" and pat.n > 8000 and case["task"] == "adjoint":
        return None
    if case["family"] == "mesh" and pat.n > 8000:
        return _solve_grid(pat, case["size"], values, b)
    A = _dense(pat, values, False)
    if case["task"] == "adjoint":
        A = A.T
    return torch.linalg.solve(A, torch.from_numpy(b).cuda().T).T.contiguous().cpu().numpy()


def exact(case, seed):
    task = case["task"]
    if task == "systems":
        pats = [_pattern(case["family"], n) for n, _ in _systems(case)]
        return [_exact_x(case, p, _values(p, 1, seed + 7 * i)[0], _rhs(case, p.n, 1, k, seed + 7 * i + 3)[0])
                for i, (p, (_, k)) in enumerate(zip(pats, _systems(case)))]
    pat = _pattern(case["family"], case["size"])
    sets, nrhs = case.get("sets", 1), case.get("nrhs", 1)
    values = _values(pat, sets, seed, _transient(case))
    if task == "refactor":
        if pat.n > 10000:
            return None
        r, c = pat.layout()
        A = _dense(pat, values[0], True)
        lu = torch.linalg.lu_factor(A, pivot=False)[0]
        if case["perturb"] and lu.diagonal().abs().min() < 1e-3 * A.abs().sum(0).max():
            return None  # a pivot as small as the perturbation
        return lu[torch.from_numpy(r).cuda(), torch.from_numpy(c).cuda()].reshape(sets, -1).cpu().numpy()
    b = _rhs(case, pat.n, sets, nrhs, seed + 1)
    if task in ("step", "solve"):
        b = b.astype(np.float32).astype(np.float64)
    x = [_exact_x(case, pat, values[k], b[k]) for k in range(sets)]
    return None if x[0] is None else np.stack(x)
