"""A self-search that keeps the query itself (include_self) on data with exact
copies of columns: the restored self value ties with the copies' values and the
lower index comes first, also where only one neighbour is asked for.  Every
engine, bit for bit against the exact engine, and the small case against the
oracle."""
import numpy as np
import pytest
import scipy.sparse as sp

from backends import OracleBackend, same_bits

pytestmark = pytest.mark.gpu


def copies(nrow, ncol, density, seed):
    """Columns ncol / 2 .. are copies of columns 0 .. ncol / 2."""
    rng = np.random.default_rng(seed)
    H = sp.random(nrow, ncol // 2, density=density, format="csc", random_state=rng,
                  data_rvs=lambda n: np.abs(rng.standard_normal(n)) + 1e-3)
    M = sp.hstack([H, H], format="csc")
    M.sort_indices()
    return M


def search(X, k, method, dist, engine):
    import sparsedist_gb300 as sdg
    from sparsedist_gb300 import _lib
    ctx = _lib.Context()
    ctx.set_engine(engine)
    r = sdg.sparseKNN(X, k=k, method=method, dist=dist, include_self=True, verbose=False, ctx=ctx)
    return r.idx, r.dist, ctx.stats()["pairs_screened"] > 0


@pytest.mark.parametrize("method,dist,engine", [
    ("binary", True, 0), ("binary", True, 2), ("binary", False, 3), ("cosine", True, 0), ("cosine", True, 2),
    ("cosine", False, 3), ("euclidean", True, 0), ("euclidean", True, 2), ("euclidean", True, 3),
    ("manhattan", True, 0), ("manhattan", True, 2), ("pearson", True, 2), ("pearson", False, 2), ("js", True, 0),
    ("js", True, 2), ("covariance", True, 2)])
@pytest.mark.parametrize("k", [1, 2])
def test_copies_tie_with_the_query_itself(method, dist, engine, k):
    X = copies(2000, 1200, 0.05, 11)
    idx, dst, screened = search(X, k, method, dist, engine)
    assert screened or engine == 0
    want = search(X, k, method, dist, 1)
    assert same_bits(idx, want[0]) and same_bits(dst, want[1])


@pytest.mark.parametrize("method,engine", [("binary", 2), ("binary", 3), ("cosine", 2), ("cosine", 3),
                                           ("euclidean", 2), ("euclidean", 3), ("manhattan", 2), ("js", 2)])
def test_copies_against_the_oracle(method, engine):
    X = copies(300, 160, 0.1, 5)
    idx, dst, screened = search(X, 1, method, True, engine)
    assert screened
    oi, od, _ = OracleBackend().knn(X, k=1, method=method, dist=True, include_self=True)
    assert same_bits(np.asarray(idx), oi) and same_bits(np.asarray(dst), od)
