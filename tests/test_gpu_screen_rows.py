"""The FP32 screen over row-ordered reference entries (engine 2) at the edges of
its layout: columns around the sub-ranges and parts, query columns around the
stretch length (1,024 stored entries), cells full of entries (bank order),
hardly any entries, the select's narrow and wide blocks, short rows against
long lists and massive ties.  Bit for bit against the exact engine on the same
matrices (which the oracle tests pin)."""
import numpy as np
import pytest
import scipy.sparse as sp

from backends import same_bits

pytestmark = pytest.mark.gpu

METHODS = ["binary", "cosine", "euclidean", "manhattan", "pearson", "js", "covariance"]


def matrix(nrow, ncol, density, seed, ties=False):
    rng = np.random.default_rng(seed)
    M = sp.random(nrow, ncol, density=density, format="csc", random_state=rng,
                  data_rvs=(lambda n: rng.integers(1, 3, n).astype(float)) if ties
                  else (lambda n: np.abs(rng.standard_normal(n)) + 1e-3))
    M.sort_indices()
    return M


def check(X, Y, method, k):
    import sparsedist_gb300 as sdg
    from sparsedist_gb300 import _lib
    out = []
    for engine in (2, 1):
        ctx = _lib.Context()
        ctx.set_engine(engine)
        out.append(sdg.sparseKNN(X, Y, k=k, method=method, verbose=False, ctx=ctx))
        if engine == 2:
            assert ctx.stats()["pairs_screened"] > 0
    assert same_bits(out[0].idx, out[1].idx)
    assert same_bits(out[0].dist, out[1].dist)


@pytest.mark.parametrize("method", METHODS)
@pytest.mark.parametrize("nrow,nr,nq,density,k", [
    (60, 511, 40, 0.6, 7), (60, 513, 310, 0.9, 10), (300, 1025, 33, 0.3, 20), (3000, 2047, 5, 0.7, 3),
    (5000, 4097, 50, 0.002, 5), (2500, 1500, 1, 0.5, 1), (700, 1300, 64, 0.1, 300), (900, 1100, 20, 0.2, 1024)])
def test_layout_edges_equal_the_exact_engine(method, nrow, nr, nq, density, k):
    check(matrix(nrow, nq, density, 1), matrix(nrow, nr, density, 2), method, k)


@pytest.mark.parametrize("stored", [1023, 1024, 1025, 2048, 2500])
@pytest.mark.parametrize("method", ["manhattan", "cosine", "js"])
def test_stretches_of_long_queries(method, stored):
    rng = np.random.default_rng(stored)
    rows = np.concatenate([np.sort(rng.permutation(2600)[:stored]), [3]]).astype(np.int32)
    X = sp.csc_matrix((np.abs(rng.standard_normal(stored + 1)) + 0.01, rows, [0, stored, stored + 1]), shape=(2600, 2))
    check(X, matrix(2600, 900, 0.3, 5), method, 12)


@pytest.mark.parametrize("method", ["binary", "manhattan", "euclidean"])
def test_massive_ties_overflow_to_the_exact_engine(method):
    check(matrix(12, 60, 0.3, 3, ties=True), matrix(12, 6000, 0.3, 4, ties=True), method, 9)
