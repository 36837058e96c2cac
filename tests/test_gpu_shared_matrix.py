"""Small searches of several threads, each with its own context and stream, against
one fresh resident matrix (as reference, and as the query matrix of blocks): the
matrix's screening data is built once and complete before any of them reads it, so
every result is the exact engine's.  And a search that is cancelled returns its
device buffers."""
import ctypes as C
import threading

import numpy as np
import pytest
import scipy.sparse as sp

from test_gpu_dense_admission import USED_CURRENT, Pool

pytestmark = pytest.mark.gpu
CODES = {"binary": 0, "euclidean": 2, "manhattan": 3}


def resident(ctx, nrow, ncol, seed):
    from sparsedist_gb300 import _lib
    rng = np.random.default_rng(seed)
    M = sp.random(nrow, ncol, density=0.06, format="csc", random_state=rng,
                  data_rvs=lambda n: np.abs(rng.standard_normal(n)) + 1e-3)
    M.sort_indices()
    return _lib.Resident(ctx, nrow, ncol, M.indptr, M.indices, M.data)


def block(ctx, X, Y, q0, nq, method, k=8):
    from sparsedist_gb300 import _lib
    idx, dst = np.empty((k, nq), np.int32), np.empty((k, nq), np.float64)
    ke, fl = C.c_int(), C.c_int()
    _lib.check(ctx.lib.sdg_knn_block(ctx.handle, X.handle, Y.handle if Y else None, q0, nq, CODES[method], 1, k, 0, 1,
                                     idx.ctypes.data, dst.ctypes.data, 0, C.byref(ke), C.byref(fl)))
    return idx.tobytes() + dst.tobytes()


@pytest.mark.parametrize("method", ["binary", "euclidean", "manhattan"])
def test_threads_share_a_fresh_matrix(method):
    from sparsedist_gb300 import _lib
    main = _lib.Context()
    ctxs = [_lib.Context() for _ in range(6)]
    for round_ in range(5):
        Y, X = resident(main, 3000, 2500, 10 + round_), resident(main, 3000, 900, 50 + round_)
        main.set_engine(1)
        # threads 0 .. 2: blocks of X against Y; 3 .. 5: blocks of Y's own columns
        args = [(X, Y, 300 * t, 300) if t < 3 else (Y, None, 400 * t, 400) for t in range(6)]
        want = [block(main, *a, method) for a in args]
        got, go = [None] * 6, threading.Barrier(6)

        def work(t):
            go.wait()
            got[t] = block(ctxs[t], *args[t], method)

        threads = [threading.Thread(target=work, args=(t,)) for t in range(6)]
        for th in threads:
            th.start()
        for th in threads:
            th.join()
        assert got == want
        assert any(c.stats()["pairs_screened"] for c in ctxs)


def test_a_cancelled_search_returns_its_buffers():
    from sparsedist_gb300 import _lib
    ctx, pool = _lib.Context(), Pool()
    Y, X = resident(ctx, 3000, 2500, 1), resident(ctx, 3000, 900, 2)
    for engine in (2, 3):
        ctx.set_engine(engine)
        want = block(ctx, X, Y, 0, 900, "euclidean")
        used = pool.get(USED_CURRENT)
        ctx.cancel()
        with pytest.raises(_lib.SdgError):
            block(ctx, X, Y, 0, 900, "euclidean")
        ctx.reset_cancel()
        assert pool.get(USED_CURRENT) <= used
        assert block(ctx, X, Y, 0, 900, "euclidean") == want
