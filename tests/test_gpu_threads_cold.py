"""Cold searches from several threads, each with its own context and matrices (the
FP32 screen builds its row-ordered copy in every one), at the same time: each
thread's results are the single-threaded ones, bit for bit."""
import threading

import numpy as np
import pytest
import scipy.sparse as sp

from backends import same_bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", ["manhattan", "js", "cosine"])
def test_threads_search_their_own_matrices(method):
    import sparsedist_gb300 as sdg
    from sparsedist_gb300 import _lib

    def matrix(seed):
        rng = np.random.default_rng(seed)
        M = sp.random(2000, 1800 + 37 * seed, density=0.05, format="csc", random_state=rng,
                      data_rvs=lambda n: np.abs(rng.standard_normal(n)) + 1e-3)
        M.sort_indices()
        return M

    def search(M):
        ctx = _lib.Context()
        ctx.set_engine(2)
        return sdg.sparseKNN(M, k=12, method=method, verbose=False, ctx=ctx)

    mats = [matrix(t) for t in range(6)]
    want = [search(M) for M in mats]
    bad = []

    def work(t):
        try:
            for _ in range(4):
                got = search(mats[t])
                if not (same_bits(got.idx, want[t].idx) and same_bits(got.dist, want[t].dist)):
                    bad.append(t)
        except Exception as e:              # noqa: BLE001 - reported by the main thread
            bad.append((t, e))

    threads = [threading.Thread(target=work, args=(t,)) for t in range(6)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not bad
