"""Queries that a screen could not bound (tied sets above its table), scattered
among others, finished together by the exact engine: every screen, self-search
with and without the query itself, an empty column, one leftover and more than
one slab of them.  Bit for bit against the exact engine."""
import numpy as np
import pytest
import scipy.sparse as sp

from backends import same_bits

pytestmark = pytest.mark.gpu


def tied(nrow, n, every, seed):
    """Random columns; each column with index % every == 0 is one of two fixed patterns, column 7 is empty."""
    rng = np.random.default_rng(seed)
    M = (rng.random((nrow, n)) < 0.3) * rng.integers(1, 4, (nrow, n)).astype(float)
    pat = (rng.random((nrow, 2)) < 0.3) * rng.integers(1, 4, (nrow, 2)).astype(float)
    at = np.arange(0, n, every)
    M[:, at] = pat[:, (at // every) % 2]
    M[:, 7] = 0.0
    return sp.csc_matrix(M)


@pytest.mark.parametrize("method,engine", [("binary", 2), ("binary", 3), ("cosine", 3), ("manhattan", 2), ("js", 2),
                                           ("covariance", 2)])
@pytest.mark.parametrize("n,every,k", [(9000, 3, 5), (9000, 4, 40)])
def test_scattered_leftovers(method, engine, n, every, k):
    import sparsedist_gb300 as sdg
    from sparsedist_gb300 import _lib
    X = tied(60, n, every, seed=n + every)
    for include_self in (False, True):
        out = []
        for e in (engine, 1):
            ctx = _lib.Context()
            ctx.set_engine(e)
            out.append(sdg.sparseKNN(X, k=k, method=method, include_self=include_self, verbose=False, ctx=ctx))
            if e != 1 and k == 5:                    # a table of 64 k candidates holds the tied sets of k = 40
                assert ctx.stats()["overflow_queries"] > 1
        assert same_bits(out[0].idx, out[1].idx) and same_bits(out[0].dist, out[1].dist)


def test_one_leftover_and_several_slabs():
    import sparsedist_gb300 as sdg
    from sparsedist_gb300 import _lib
    Y = tied(50, 20000, 2, seed=9)
    for pick in (np.array([3, 11, 4, 21]), np.r_[np.arange(0, 8000, 2), 1, 3]):   # 4,000 x 20,000 doubles: 3 slabs
        out = []
        for e in (2, 1):
            ctx = _lib.Context()
            ctx.set_engine(e)
            out.append(sdg.sparseKNN(Y[:, pick], Y, k=6, method="binary", verbose=False, ctx=ctx))
        assert same_bits(out[0].idx, out[1].idx) and same_bits(out[0].dist, out[1].dist)
