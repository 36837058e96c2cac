"""The exact re-rank of a few queries with many candidates: a query's candidates
over several CTAs, at counts around the groups of 32.  Bit for bit against the
exact engine."""
import numpy as np
import pytest
import scipy.sparse as sp

from backends import same_bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", ["binary", "cosine", "euclidean", "manhattan", "pearson", "js", "covariance"])
@pytest.mark.parametrize("nq,k", [(1, 31), (1, 33), (2, 300), (3, 64), (40, 97), (700, 33)])
def test_few_queries(method, nq, k):
    import sparsedist_gb300 as sdg
    from sparsedist_gb300 import _lib
    rng = np.random.default_rng(nq)
    M = sp.random(3000, nq + 1500, density=0.1, format="csc", random_state=rng,
                  data_rvs=lambda n: np.abs(rng.standard_normal(n)) + 1e-3)
    M.sort_indices()
    out = []
    for engine in (2, 1):
        ctx = _lib.Context()
        ctx.set_engine(engine)
        out.append(sdg.sparseKNN(M[:, :nq], M[:, nq:], k=k, method=method, verbose=False, ctx=ctx))
        if engine == 2:
            assert ctx.stats()["pairs_screened"] > 0
    assert same_bits(out[0].idx, out[1].idx) and same_bits(out[0].dist, out[1].dist)
