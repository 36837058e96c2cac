"""A small search of resident matrices, searched once before, captured into a CUDA
graph: the replay writes the values of the eager call, whose automatic choice may
be a screen (which reads counts back and could not be captured)."""
import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def matrix(nrow, ncol, seed):
    rng = np.random.default_rng(seed)
    M = sp.random(nrow, ncol, density=0.08, format="csc", random_state=rng,
                  data_rvs=lambda n: np.abs(rng.standard_normal(n)) + 1e-3)
    M.sort_indices()
    return M


@pytest.mark.parametrize("method", [0, 1, 2, 3, 4, 5, 6])
@pytest.mark.parametrize("block", [False, True])
def test_replay_equals_the_eager_call(method, block):
    import torch
    from sparsedist_gb300 import _lib
    ctx = _lib.Context()
    X, Y = ((lambda M: _lib.Resident(ctx, *M.shape, M.indptr, M.indices, M.data))(matrix(5000, n, n))
            for n in (200, 3000))
    k, nq = 9, 120 if block else 200
    idx = torch.zeros(k, nq, dtype=torch.int32, device="cuda")
    dst = torch.zeros(k, nq, dtype=torch.float64, device="cuda")
    ke, fl = C.c_int(), C.c_int()

    def search():
        if block:
            return ctx.lib.sdg_knn_block(ctx.handle, X.handle, Y.handle, 40, nq, method, 1, k, 0, 1, idx.data_ptr(),
                                         dst.data_ptr(), 1, C.byref(ke), C.byref(fl))
        return ctx.lib.sdg_knn_resident_device(ctx.handle, X.handle, Y.handle, method, 1, k, 0, 1, idx.data_ptr(),
                                               dst.data_ptr(), C.byref(ke), C.byref(fl))

    _lib.check(search())
    torch.cuda.synchronize()
    want = idx.clone(), dst.clone()
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    ctx.set_stream(stream.cuda_stream)
    try:
        with torch.cuda.graph(graph, stream=stream):
            rc = search()
        _lib.check(rc)
        for _ in range(2):
            idx.zero_()
            dst.zero_()
            torch.cuda.synchronize()
            graph.replay()
            torch.cuda.synchronize()
            assert torch.equal(idx, want[0]) and torch.equal(dst, want[1])
    finally:
        torch.cuda.synchronize()
        ctx.set_stream(None)
    _lib.check(search())                     # the context searches on as before
    torch.cuda.synchronize()
    assert torch.equal(idx, want[0]) and torch.equal(dst, want[1])
