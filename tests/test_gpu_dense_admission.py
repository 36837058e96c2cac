"""The dense server's admission estimate of a request is no less than the device
memory its search takes from the pool at most (the search run alone), and not more
than one and a half times as much."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_dense import dense_query
from test_gpu_dense_two_pass import upload

pytestmark = pytest.mark.gpu
USED_CURRENT, USED_HIGH = 7, 8               # CUmemPool_attribute


class Pool:
    def __init__(self):
        self.lib = C.CDLL("libcuda.so.1")
        dev, self.pool = C.c_int(), C.c_void_p()
        assert self.lib.cuDeviceGet(C.byref(dev), 0) == 0
        assert self.lib.cuDeviceGetDefaultMemPool(C.byref(self.pool), dev) == 0

    def get(self, attr):
        v = C.c_uint64()
        assert self.lib.cuMemPoolGetAttribute(self.pool, attr, C.byref(v)) == 0
        return v.value

    def peak_of(self, call):
        import torch
        call()
        torch.cuda.synchronize()
        zero = C.c_uint64(0)
        assert self.lib.cuMemPoolSetAttribute(self.pool, USED_HIGH, C.byref(zero)) == 0
        before = self.get(USED_CURRENT)
        call()
        torch.cuda.synchronize()
        return self.get(USED_HIGH) - before


def estimate(ctx, h, Q, method, k):
    """bytes_admitted by one request, behind one that keeps the only worker busy (every pair valued exactly)."""
    from sparsedist_gb300 import _lib
    srv = _lib.Server(ctx, h, workers=1, max_slots=4, mem_budget=1 << 40, dense=True)
    first = srv.submit_dense(np.random.default_rng(1).standard_normal((48, Q.shape[1])).astype(np.float32), 1, 1100)
    one = srv.stats()["bytes_admitted"]
    second = srv.submit_dense(Q, method, k)
    two = srv.stats()
    assert two["completed"] == 0
    for r in (first, second):
        srv.wait(r)
        srv.result(r)
    srv.close()
    return two["bytes_admitted"] - one


@pytest.mark.parametrize("d,n,nq,method,k", [(64, 300000, 128, 1, 10), (256, 200000, 1, 1, 20), (100, 250000, 777, 2, 15),
                                             (200, 200000, 2048, 1, 50), (64, 150000, 60, 2, 64), (64, 200000, 40, 1, 100),
                                             (300, 200000, 64, 2, 10)])
def test_estimate_covers_the_search(d, n, nq, method, k):
    from sparsedist_gb300 import _lib, synth
    ctx = _lib.Context()
    X = synth.dense_embeddings(d=d, n=n + nq, centres=50, seed=3)
    h = upload(ctx, X[:n].contiguous())
    Q = np.ascontiguousarray(X[n:].cpu().numpy())
    peak = Pool().peak_of(lambda: dense_query(ctx, h, Q, method, k, 0))
    got = estimate(ctx, h, Q, method, k)
    ctx.lib.sdg_dense_free(h)
    assert peak <= got <= 1.5 * peak + (4 << 20)
