"""Searches of at most 2^22 pairs take the exact slab or a screen by predicted
cost: the automatic choice equals the exact engine bit for bit on both sides of
the rule, for every method and option (similarities, the self column kept,
degenerate columns kept, stored zeros, empty columns, signed values)."""
import numpy as np
import pytest
import scipy.sparse as sp

from backends import same_bits

pytestmark = pytest.mark.gpu


def matrix(nrow, ncol, density, seed, signed=False, zeros=True):
    rng = np.random.default_rng(seed)
    M = sp.random(nrow, ncol, density=density, format="csc", random_state=rng,
                  data_rvs=lambda n: rng.standard_normal(n) if signed else np.abs(rng.standard_normal(n)) + 1e-3)
    M.sort_indices()
    if zeros:
        M.data[:: 17] = 0.0                                  # stored zeros
        M.data[M.indptr[3]:M.indptr[4]] = 0.0                # a column of them
    return M


def both(ctx, *a, **kw):
    import sparsedist_gb300 as sdg
    out = []
    for engine in (0, 1):
        ctx.set_engine(engine)
        out.append(sdg.sparseKNN(*a, verbose=False, ctx=ctx, **kw))
        if engine == 0:
            screened = ctx.stats()["pairs_screened"] > 0
    assert same_bits(out[0].idx, out[1].idx)
    assert same_bits(out[0].dist, out[1].dist)
    return screened


@pytest.mark.parametrize("method,dist", [("binary", True), ("binary", False), ("cosine", True), ("cosine", False),
                                         ("euclidean", True), ("manhattan", True), ("pearson", True),
                                         ("pearson", False), ("js", True), ("covariance", True)])
def test_automatic_choice_equals_the_exact_engine(method, dist):
    from sparsedist_gb300 import _lib
    ctx = _lib.Context()
    signed = method in ("cosine", "euclidean", "manhattan", "pearson", "covariance")
    taken = set()
    # few steps; many steps; many steps of columns that share almost nothing
    for nrow, nx, ny, density in ((300, 150, 180, 0.03), (4000, 300, 2500, 0.06), (30000, 90, 4000, 0.004)):
        X, Y = matrix(nrow, nx, density, 1, signed), matrix(nrow, ny, density, 2, signed)
        for drop in (True, False):
            taken.add(both(ctx, X, Y, k=9, method=method, dist=dist, drop_degenerate=drop))
    X = matrix(3000, 900, 0.08, 3, signed)
    for include_self in (True, False):
        taken.add(both(ctx, X, k=11, method=method, dist=dist, include_self=include_self))
    assert taken == {True, False}
