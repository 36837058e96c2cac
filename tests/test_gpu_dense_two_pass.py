"""The dense screen in two passes (maxima, threshold, appended references) on
both sides of its rule: ragged d and n, few and many maxima per query, degenerate
references and queries (no key of theirs may raise a threshold), all-negative
similarities, near duplicates, self-search.  Bit for bit against the oracle."""
import numpy as np
import pytest

from backends import OracleBackend, same_bits
from test_gpu_dense import as_csc, dense_knn, dense_query

pytestmark = pytest.mark.gpu


def upload(ctx, X):
    import ctypes as C
    from sparsedist_gb300 import _lib
    h = C.c_void_p()
    _lib.check(ctx.lib.sdg_dense_upload(ctx.handle, X.data_ptr(), X.shape[1], X.shape[0], C.byref(h)))
    return h


@pytest.mark.parametrize("method,code", [("cosine", 1), ("euclidean", 2)])
@pytest.mark.parametrize("d,n,nq,k", [(20, 1000, 63, 5), (20, 1000, 64, 5), (33, 1025, 100, 8), (64, 4096, 129, 1),
                                      (130, 9001, 200, 17), (256, 3000, 256, 64), (100, 20000, 77, 50)])
def test_queries(method, code, d, n, nq, k):
    from sparsedist_gb300 import _lib, synth
    X = synth.dense_embeddings(d=d, n=n + nq, centres=9, dup_frac=0.05, seed=31)
    X[5] = 0.0
    X[n - 1] = 0.0
    X[n + 3] = 0.0                                   # a degenerate query: all NA
    ctx = _lib.Context()
    R = X[:n].contiguous()
    h = upload(ctx, R)
    got = dense_query(ctx, h, np.ascontiguousarray(X[n:].cpu().numpy()), code, k, 0)
    ctx.lib.sdg_dense_free(h)
    wi, wd, _ = OracleBackend().knn(as_csc(X[n:]), as_csc(R), k=k, method=method)
    assert same_bits(got[0], wi) and same_bits(got[1], wd)


@pytest.mark.parametrize("method,code", [("cosine", 1), ("euclidean", 2)])
def test_negative_similarities_and_zero_columns(method, code):
    """Every true similarity is below 0, so a degenerate or padding reference's 0 would be the largest."""
    import torch
    from sparsedist_gb300 import _lib
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    R = -(torch.rand(777, 24, generator=g, device="cuda") + 0.1)
    R[10:40] = 0.0
    Q = torch.rand(130, 24, generator=g, device="cuda") + 0.1
    ctx = _lib.Context()
    h = upload(ctx, R)
    got = dense_query(ctx, h, np.ascontiguousarray(Q.cpu().numpy()), code, 6, 0)
    ctx.lib.sdg_dense_free(h)
    wi, wd, _ = OracleBackend().knn(as_csc(Q), as_csc(R), k=6, method=method)
    assert same_bits(got[0], wi) and same_bits(got[1], wd)


@pytest.mark.parametrize("method,code", [("cosine", 1), ("euclidean", 2)])
@pytest.mark.parametrize("n,k", [(700, 3), (5000, 40)])
def test_self_search(method, code, n, k):
    from sparsedist_gb300 import _lib, synth
    X = synth.dense_embeddings(d=48, n=n, centres=5, dup_frac=0.2, seed=32)
    X[123] = 0.0
    ctx = _lib.Context()
    h = upload(ctx, X)
    got = dense_knn(ctx, h, 100, 500, code, k, 0)
    ctx.lib.sdg_dense_free(h)
    wi, wd, _ = OracleBackend().knn(as_csc(X), k=k, method=method)
    assert same_bits(got[0], wi[100:600]) and same_bits(got[1], wd[100:600])
