"""The dense screen's merge (one, eight or thirty-two warps per query by the
block's size) and the FP32 cut at the edges of their rules: a single query
over every CTA's lists, the block sizes around both borders, the longest
lists.  idx and distances bit for bit against the oracle's search."""
import numpy as np
import pytest

from backends import OracleBackend, same_bits
from test_gpu_dense import as_csc, dense_knn, dense_query

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method,code", [("cosine", 1), ("euclidean", 2)])
@pytest.mark.parametrize("nq,n,k", [(1, 70001, 64), (1, 40000, 1), (304, 20000, 10), (305, 20000, 64)])
def test_queries_over_many_lists(method, code, nq, n, k):
    import ctypes as C
    from sparsedist_gb300 import _lib, synth
    X = synth.dense_embeddings(d=24, n=n + nq, centres=40, seed=11)
    ctx = _lib.Context()
    h = C.c_void_p()
    R = X[:n].contiguous()
    _lib.check(ctx.lib.sdg_dense_upload(ctx.handle, R.data_ptr(), 24, n, C.byref(h)))
    Q = np.ascontiguousarray(X[n:].cpu().numpy())
    got = dense_query(ctx, h, Q, code, k, 0)
    ctx.lib.sdg_dense_free(h)
    wi, wd, _ = OracleBackend().knn(as_csc(X[n:]), as_csc(R), k=k, method=method)
    assert same_bits(got[0], wi) and same_bits(got[1], wd)


@pytest.mark.parametrize("nq", [2431, 2432, 5000])
def test_blocks_around_the_warp_per_query_rule(nq):
    import ctypes as C
    from sparsedist_gb300 import _lib, synth
    X = synth.dense_embeddings(d=16, n=5000, centres=20, seed=12)
    ctx = _lib.Context()
    h = C.c_void_p()
    _lib.check(ctx.lib.sdg_dense_upload(ctx.handle, X.data_ptr(), 16, 5000, C.byref(h)))
    got = dense_knn(ctx, h, 0, nq, 1, 64, 0)
    ctx.lib.sdg_dense_free(h)
    wi, wd, _ = OracleBackend().knn(as_csc(X), k=64, method="cosine")
    assert same_bits(got[0], wi[:nq]) and same_bits(got[1], wd[:nq])
