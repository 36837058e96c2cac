"""The choice between the exact slab and a screen for small searches counts the
columns, the rows and the copies a screen would first make of matrices that have
none: shapes where the slab was measured faster keep it (and add nothing to the
matrices' device memory), a matrix searched before is screened sooner than a fresh
one, and either choice gives the exact engine's results bit for bit."""
import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu
CODES = {"binary": 0, "cosine": 1, "euclidean": 2, "manhattan": 3, "pearson": 4, "js": 5, "covariance": 6}


def matrix(ctx, nrow, ncol, density, seed):
    from sparsedist_gb300 import _lib
    rng = np.random.default_rng(seed)
    m = max(1, int(density * nrow))                       # entries per column, rows drawn from as many strata
    at = (np.arange(m) * nrow) // m
    rows = at[None, :] + rng.integers(0, max(1, nrow // m), (ncol, m))
    vals = np.abs(rng.standard_normal(rows.shape)) + 1e-3
    M = sp.csc_matrix((vals.ravel(), rows.ravel().astype(np.int32), np.arange(0, ncol * m + 1, m)), shape=(nrow, ncol))
    return _lib.Resident(ctx, nrow, ncol, M.indptr, M.indices, M.data)


def search(ctx, X, Y, method, k, engine):
    from sparsedist_gb300 import _lib
    nq = X.ncol
    idx, dst = np.empty((k, nq), np.int32), np.empty((k, nq), np.float64)
    ke, fl = C.c_int(), C.c_int()
    ctx.set_engine(engine)
    _lib.check(ctx.lib.sdg_knn_block(ctx.handle, X.handle, Y.handle, 0, nq, CODES[method], 1, k, 0, 1, idx.ctypes.data,
                                     dst.ctypes.data, 0, C.byref(ke), C.byref(fl)))
    return idx.tobytes() + dst.tobytes(), ctx.stats()["pairs_screened"] > 0


@pytest.mark.parametrize("method,nrow,nr,nq,density,screened", [
    ("pearson", 2000, 60000, 8, 0.1, False), ("pearson", 12000, 12000, 60, 0.01, False),
    ("covariance", 2000, 60000, 8, 0.1, False), ("binary", 2000, 300, 2000, 0.1, False),
    ("binary", 30000, 300, 256, 0.05, False), ("manhattan", 2000, 3000, 400, 0.1, True),
    ("manhattan", 8000, 2000, 20, 0.05, True), ("cosine", 3000, 2500, 800, 0.04, True),
    ("euclidean", 3000, 2000, 300, 0.05, True), ("js", 3000, 2000, 300, 0.05, True)])
def test_fresh_matrices(method, nrow, nr, nq, density, screened):
    from sparsedist_gb300 import _lib
    ctx = _lib.Context()
    X, Y = matrix(ctx, nrow, nq, density, 1), matrix(ctx, nrow, nr, density, 2)
    got, took = search(ctx, X, Y, method, 10, 0)
    assert took == screened
    assert got == search(ctx, X, Y, method, 10, 1)[0]


def test_copies_made_before_count():
    from sparsedist_gb300 import _lib
    ctx = _lib.Context()
    X, Y = matrix(ctx, 3000, 500, 0.05, 1), matrix(ctx, 3000, 2000, 0.05, 2)
    want = search(ctx, X, Y, "binary", 10, 1)[0]
    assert search(ctx, X, Y, "binary", 10, 0) == (want, False)
    assert search(ctx, X, Y, "binary", 10, 2) == (want, True)
    assert search(ctx, X, Y, "binary", 10, 0) == (want, True)
