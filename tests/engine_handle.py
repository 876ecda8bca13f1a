"""A handle of the C ABI on a given matrix, for tests that need no preprocessing library."""
import contextlib
import ctypes as C

import numpy as np


def pattern(A):
    """(column pointers, row indices, columns) of the entries of A in column order."""
    cols, rows = np.nonzero(A.T)
    ap = np.zeros(A.shape[0] + 1, np.uint32)
    ap[1:] = np.cumsum(np.bincount(cols, minlength=A.shape[0]))
    return ap, rows.astype(np.uint32), cols


class Handle:
    """Factor and solve with dense matrices of one pattern."""

    def __init__(self, A, sets, dense):
        from pyglu import _capi

        self.capi, self.eng, self.ptr = _capi, _capi.engine(), _capi.ptr
        self.n = A.shape[0]
        self.ap, self.rows, self.cols = pattern(A)
        self.sym, self.h = C.c_void_p(), C.c_void_p()
        _capi.check(self.eng.glu_symbolic_analyze(self.n, self.rows.size, self.ptr(self.ap), self.ptr(self.rows),
                                                  C.byref(self.sym)))
        _capi.check(self.eng.glu_create(self.sym, 0, sets, C.byref(self.h)))
        if not dense:
            self.tune(dense_tail_min=1 << 31)
            assert self.stats().dense_tail == 0

    def tune(self, **kw):
        t = self.capi.Tuning()
        self.capi.check(self.eng.glu_get_tuning(self.h, C.byref(t)))
        for k, v in kw.items():
            setattr(t, k, v)
        self.capi.check(self.eng.glu_set_tuning(self.h, C.byref(t)))

    def stats(self):
        st = self.capi.Stats()
        self.capi.check(self.eng.glu_get_stats(self.h, C.byref(st)))
        return st

    def load(self, z, A):
        """A's values for value set z, in FP32."""
        val = np.empty(self.stats().nnz_lu, np.float32)
        self.eng.glu_predict_lu(self.sym, self.ptr(np.ascontiguousarray(A.T[self.cols, self.rows], np.float64)),
                                self.ptr(val))
        self.capi.check(self.eng.glu_load_lu_values(self.h, z, 1, self.ptr(val), self.capi.GLU_HOST, None))

    def source(self, mats):
        """The matrices as sources of all value sets: for refined solves."""
        slots = np.empty(self.rows.size, np.uint32)
        self.eng.glu_symbolic_slots(self.sym, self.ptr(slots))
        self.capi.check(self.eng.glu_set_source(self.h, self.rows.size, self.ptr(self.ap), self.ptr(self.rows),
                                                self.ptr(slots), None))
        ax = np.stack([np.ascontiguousarray(A.T[self.cols, self.rows], np.float64) for A in mats])
        self.capi.check(self.eng.glu_load_source_values(self.h, 0, len(mats), self.ptr(ax), self.capi.GLU_HOST, None))

    def factor(self, first=0, count=1, perturb=0):
        return self.eng.glu_factor(self.h, first, count, perturb, None)

    def factors(self, z):
        """L + U - I of value set z as a dense FP32 matrix."""
        nnz = self.stats().nnz_lu
        val, cp, ri = np.empty(nnz, np.float32), np.empty(self.n + 1, np.uint32), np.empty(nnz, np.uint32)
        self.eng.glu_symbolic_export(self.sym, self.ptr(cp), self.ptr(ri), None, None, None, None)
        self.capi.check(self.eng.glu_store_lu_values(self.h, z, 1, self.ptr(val), self.capi.GLU_HOST, None))
        F = np.zeros((self.n, self.n), np.float32)
        F[ri, np.repeat(np.arange(self.n), np.diff(cp.astype(np.int64)))] = val
        return F

    def solve(self, z, b, transposed=False):
        """FP32 solution(s) of value set z for the rows of b."""
        b = np.ascontiguousarray(b, np.float32)
        x = np.empty_like(b)
        call = self.eng.glu_solve_transposed if transposed else self.eng.glu_solve
        self.capi.check(call(self.h, z, b.size // self.n, self.ptr(b), self.ptr(x), self.capi.GLU_HOST, None))
        return x

    def solve_refined(self, z, b, tol, steps):
        """FP64 solution of value set z, at most ``steps`` refinements."""
        b = np.ascontiguousarray(b, np.float64)
        x, st = np.empty_like(b), self.capi.RefineStats()
        r = self.eng.glu_solve_refined(self.h, z, 1, b.size // self.n, self.ptr(b), self.ptr(x), tol, steps, 0,
                                       self.capi.GLU_HOST, C.byref(st), None)
        assert r in (self.capi.GLU_OK, self.capi.GLU_ERR_NOT_CONVERGED)
        return x, st


@contextlib.contextmanager
def handle(A, sets=1, dense=True):
    """A handle with A's pattern; dense=False: without a dense trailing block."""
    H = Handle(A, sets, dense)
    try:
        yield H
    finally:
        H.eng.glu_destroy(H.h)
        H.eng.glu_symbolic_destroy(H.sym)


def blocks(width, count, seed):
    """Block tridiagonal n x n matrix of filled width x width blocks, diagonally dominant by a factor of two."""
    rng = np.random.default_rng(seed)
    n = width * count
    at = np.arange(n) // width
    A = np.where(np.abs(at[:, None] - at[None, :]) <= 1, rng.uniform(-1.0, 1.0, (n, n)), 0.0)
    np.fill_diagonal(A, 0.0)
    np.fill_diagonal(A, 2.0 * np.maximum(np.abs(A).sum(0), np.abs(A).sum(1)) + 1.0)
    return A
