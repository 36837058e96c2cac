"""The dense screen's thresholds from a strided sample: strides 1 to 8 and the
sizes where they change, a remainder that no whole run of the stride holds,
references stored in turn by class (the sample has to see every class), one query
and CTA pairs (d > 128, an even number of 128-query groups), self-search with the
query inside and outside its sample.  Bit for bit against the oracle."""
import numpy as np
import pytest

from backends import OracleBackend, same_bits
from test_gpu_dense import as_csc, dense_knn, dense_query
from test_gpu_dense_two_pass import upload

pytestmark = pytest.mark.gpu


def check(X, n, code, method, k, mode=0):
    from sparsedist_gb300 import _lib
    ctx = _lib.Context()
    R = X[:n].contiguous()
    h = upload(ctx, R)
    got = dense_query(ctx, h, np.ascontiguousarray(X[n:].cpu().numpy()), code, k, mode)
    ctx.lib.sdg_dense_free(h)
    wi, wd, _ = OracleBackend().knn(as_csc(X[n:]), as_csc(R), k=k, method=method)
    assert same_bits(got[0], wi) and same_bits(got[1], wd)


# k = 2: a stride of s needs n / s > 256 * 3 (32 maxima of 32 columns: 4 tiles)
@pytest.mark.parametrize("method,code", [("cosine", 1), ("euclidean", 2)])
@pytest.mark.parametrize("d,n,nq,k", [(40, 128, 3, 4), (40, 129, 3, 4), (64, 769 * 2 - 1, 5, 2), (64, 769 * 2, 5, 2),
                                      (64, 769 * 8 - 1, 5, 2), (64, 769 * 8, 1, 2), (70, 16 * 1024 + 7, 40, 9),
                                      (130, 9001, 256, 3), (256, 12007, 300, 6), (192, 7001, 512, 1)])
def test_strides(method, code, d, n, nq, k):
    from sparsedist_gb300 import synth
    X = synth.dense_embeddings(d=d, n=n + nq, centres=7, dup_frac=0.05, seed=41)
    X[8] = 0.0
    X[n - 1] = 0.0
    check(X, n, code, method, k)
    if nq > 128:
        check(X, n, code, method, k, mode=3)


@pytest.mark.parametrize("method,code", [("cosine", 1), ("euclidean", 2)])
@pytest.mark.parametrize("period", [5, 7, 8])
def test_references_in_turn_by_class(method, code, period):
    """Reference r belongs to class r mod period; a query's neighbours are one class's."""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(period)
    d, n, nq, k = 48, 20000, 65, 5
    centres = torch.randn(period, d, generator=g, device="cuda") * 3
    label = torch.arange(n + nq, device="cuda") % period
    X = (centres[label] + 0.3 * torch.randn(n + nq, d, generator=g, device="cuda")).contiguous()
    check(X, n, code, method, k)


@pytest.mark.parametrize("method,code", [("cosine", 1), ("euclidean", 2)])
@pytest.mark.parametrize("d,n,nq,k", [(48, 14001, 300, 4), (144, 9000, 256, 2)])
def test_self_search(method, code, d, n, nq, k):
    from sparsedist_gb300 import _lib, synth
    X = synth.dense_embeddings(d=d, n=n, centres=5, dup_frac=0.2, seed=42)
    X[1003] = 0.0
    ctx = _lib.Context()
    h = upload(ctx, X)
    got = dense_knn(ctx, h, 1000, nq, code, k, 0)
    ctx.lib.sdg_dense_free(h)
    wi, wd, _ = OracleBackend().knn(as_csc(X), k=k, method=method)
    assert same_bits(got[0], wi[1000:1000 + nq]) and same_bits(got[1], wd[1000:1000 + nq])


@pytest.mark.parametrize("method,code", [("cosine", 1), ("euclidean", 2)])
@pytest.mark.parametrize("d,nq,k", [(32, 70, 5), (200, 256, 3)])
def test_clusters_that_overflow_the_lists(method, code, d, nq, k):
    """Contiguous clusters of 4,000 within the bound of one another: the lists of
    what passes the thresholds overflow and the block repeats with running lists."""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(d)
    centres = torch.randn(5, d, generator=g, device="cuda")
    label = torch.cat([torch.arange(5, device="cuda").repeat_interleave(4000), torch.arange(nq, device="cuda") % 5])
    X = (centres[label] + 0.05 * torch.randn(20000 + nq, d, generator=g, device="cuda")).contiguous()
    check(X, 20000, code, method, k)
