"""The exact values of the screens' candidates on short columns (a thread per
candidate) around the lengths where the choice lies, with empty columns, copies,
one long column among short ones and more candidates than a block has threads.
Bit for bit against the exact engine."""
import numpy as np
import pytest
import scipy.sparse as sp

from backends import same_bits

pytestmark = pytest.mark.gpu


def columns(nrow, ncol, stored, seed):
    rng = np.random.default_rng(seed)
    rows = [np.sort(rng.permutation(nrow)[:stored + (j % 3) - 1]) for j in range(ncol)]
    rows[5] = np.array([], int)
    rows[7] = np.arange(nrow)                              # a long one
    p = np.cumsum([0] + [len(r) for r in rows])
    x = rng.integers(1, 4, p[-1]).astype(float)
    M = sp.csc_matrix((x, np.concatenate(rows).astype(np.int32), p.astype(np.int32)), shape=(nrow, ncol))
    return sp.hstack([M, M[:, : ncol // 5]], format="csc")


@pytest.mark.parametrize("method", ["manhattan", "euclidean", "js", "covariance", "binary", "cosine", "pearson"])
@pytest.mark.parametrize("stored,k,include_self", [(2, 40, False), (20, 9, True), (23, 5, False), (25, 5, True),
                                                   (62, 12, False), (66, 12, True)])
def test_short_columns(method, stored, k, include_self):
    import sparsedist_gb300 as sdg
    from sparsedist_gb300 import _lib
    X = columns(400, 900, stored, stored)
    out = []
    for engine in (2, 1):
        ctx = _lib.Context()
        ctx.set_engine(engine)
        for kw in ({"include_self": include_self}, {"Y": X[:, 100:800]}):
            out.append(sdg.sparseKNN(X, k=k, method=method, drop_degenerate=stored != 20, verbose=False, ctx=ctx, **kw))
        if engine == 2:
            assert ctx.stats()["pairs_screened"] > 0
    for a, b in zip(out[:2], out[2:]):
        assert same_bits(a.idx, b.idx) and same_bits(a.dist, b.dist)


def test_many_candidates_of_long_columns():
    """Manhattan, k nq above the walk's limit on columns longer than its other one."""
    import sparsedist_gb300 as sdg
    from sparsedist_gb300 import _lib
    X = columns(900, 2700, 100, 3)
    out = []
    for engine in (2, 1):
        ctx = _lib.Context()
        ctx.set_engine(engine)
        out.append(sdg.sparseKNN(X, k=90, method="manhattan", include_self=True, verbose=False, ctx=ctx))
        if engine == 2:
            assert ctx.stats()["pairs_screened"] > 0
    assert same_bits(out[0].idx, out[1].idx) and same_bits(out[0].dist, out[1].dist)
