"""The exact values of the screens' candidates (k_rerank) at the edges of its
lists: columns of 0, 1, 31 .. 129 stored entries, identical and disjoint columns,
the self pair restored, more than 32 candidates, degenerate columns kept.  Bit
for bit against the oracle (pearson / js / covariance: against the exact engine,
whose values the oracle tests bound)."""
import numpy as np
import pytest
import scipy.sparse as sp

from backends import OracleBackend, same_bits

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 2, 31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 128, 129, 200]


def columns(nrow, ncol, seed):
    rng = np.random.default_rng(seed)
    rows, vals, p = [], [], [0]
    for j in range(ncol):
        m = LENGTHS[j % len(LENGTHS)]
        if j % 7 == 3:                         # a run at the end of the rows: shares nothing with the next ones
            r = np.arange(nrow - m, nrow)
        elif j % 7 == 5:
            r = np.arange(m)
        else:
            r = np.sort(rng.permutation(nrow)[:m])
        rows.append(r)
        vals.append(np.abs(rng.standard_normal(m)) + 0.01)
        p.append(p[-1] + m)
    M = sp.csc_matrix((np.concatenate(vals), np.concatenate(rows).astype(np.int32), np.array(p, np.int32)),
                      shape=(nrow, ncol))
    return sp.hstack([M, M[:, : ncol // 4]], format="csc")       # identical columns


@pytest.mark.parametrize("include_self,k", [(False, 1), (False, 33), (False, 70), (True, 12), (True, 33)])
@pytest.mark.parametrize("drop", [True, False])
@pytest.mark.parametrize("method", ["binary", "cosine", "euclidean", "manhattan", "pearson", "js", "covariance"])
def test_list_edges(method, drop, include_self, k):
    import sparsedist_gb300 as sdg
    from sparsedist_gb300 import _lib
    X = columns(430, 160, 21)
    ctx = _lib.Context()
    ctx.set_engine(2)
    got = sdg.sparseKNN(X, k=k, method=method, include_self=include_self, drop_degenerate=drop, verbose=False, ctx=ctx)
    if method in ("pearson", "js", "covariance"):
        ctx.set_engine(1)
        want = sdg.sparseKNN(X, k=k, method=method, include_self=include_self, drop_degenerate=drop, verbose=False,
                             ctx=ctx)
        idx, dist = want.idx, want.dist
    else:
        idx, dist, *_ = OracleBackend().knn(X, k=k, method=method, include_self=include_self, drop_degenerate=drop)
    assert same_bits(got.idx, idx) and same_bits(got.dist, dist)
