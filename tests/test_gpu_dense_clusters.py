"""The dense screen on clustered references: stored cluster by cluster or in turn,
the sample's thresholds leave the lists room (no block repeats); queries with more
candidates within the uniform bound than the table holds are cut by the per-pair
bound; a tight cluster that overflows the lists repeats the block with running
lists, for every list length and on CTA pairs.  Bit for bit against the slab
screen (mode 2)."""
import numpy as np
import pytest

from backends import same_bits
from test_gpu_dense import dense_knn, dense_query
from test_gpu_dense_two_pass import upload

pytestmark = pytest.mark.gpu


def clusters(n, nq, d, classes, sigma, seed, order):
    """n references of `classes` clusters (in order, in turn or shuffled) and nq queries from them."""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    centres = torch.randn(classes, d, generator=g, device="cuda")
    label = torch.randint(0, classes, (n,), generator=g, device="cuda")
    if order == "in order":
        label = label.sort().values
    elif order == "in turn":
        label = torch.arange(n, device="cuda") % classes
    of = torch.cat([label, torch.randint(0, classes, (nq,), generator=g, device="cuda")])
    X = centres[of] + sigma * torch.randn(n + nq, d, generator=g, device="cuda")
    return X[:n].contiguous(), X[n:].contiguous()


def check(R, Q, code, k, mode):
    from sparsedist_gb300 import _lib
    ctx = _lib.Context()
    h = upload(ctx, R)
    q = np.ascontiguousarray(Q.cpu().numpy())
    got = dense_query(ctx, h, q, code, k, mode)
    stats = ctx.stats()
    want = dense_query(ctx, h, q, code, k, 2)
    ctx.lib.sdg_dense_free(h)
    assert same_bits(got[0], want[0]) and same_bits(got[1], want[1])
    return stats


@pytest.mark.parametrize("code", [1, 2])
@pytest.mark.parametrize("order", ["in order", "in turn", "shuffled"])
@pytest.mark.parametrize("n,d,nq,classes,k", [(150000, 64, 700, 30, 10), (120000, 160, 256, 100, 15),
                                              (100003, 100, 300, 7, 3)])
def test_no_block_repeats(code, order, n, d, nq, classes, k):
    R, Q = clusters(n, nq, d, classes, 0.3, d, order)
    stats = check(R, Q, code, k, 0)
    assert stats["repeated_blocks"] == 0 and stats["overflow_queries"] == 0


def beyond_the_table(R, Q, code, k):
    """Queries with more than 64 k + 256 references within the per-pair bound (its rounding allowances taken 5 % wider)."""
    import torch
    norm = (lambda M: torch.nn.functional.normalize(M.double(), dim=1)) if code == 1 else (lambda M: M.double())
    r, q = norm(R), norm(Q)
    rb, qb = (M.float().bfloat16().double() for M in (r, q))
    er, eq, nr, nq = (r - rb).norm(dim=1), (q - qb).norm(dim=1), rb.norm(dim=1), qb.norm(dim=1)
    acc = (R.shape[1] + 64) * 2.0 ** -21
    beyond = 0
    for a in range(0, len(Q), 256):
        b = slice(a, a + 256)
        s = qb[b] @ rb.T
        E = 1.06 * (eq[b, None] * r.norm(dim=1) + nq[b, None] * (er + acc * nr)) + 1e-6 * s.abs()
        if code == 2:
            N = (q[b] ** 2).sum(1)[:, None] + (r ** 2).sum(1)
            s, E = 2 * s - N, 2 * E + 1e-6 * N
        T = (s - E).topk(k, dim=1).values[:, -1:]
        beyond += int((((s + E) >= T).sum(1) > 64 * k + 256).sum())
    return beyond


@pytest.mark.parametrize("code", [1, 2])
@pytest.mark.parametrize("nq", [40, 900, 3000])                # 32, 8 and 1 warps a query
def test_more_candidates_than_the_table(code, nq):
    R, Q = clusters(200000, nq, 256, 10, 0.3, 3, "shuffled")
    stats = check(R, Q, code, 5, 0)
    assert stats["repeated_blocks"] == 0 and stats["overflow_queries"] <= beyond_the_table(R, Q, code, 5)


@pytest.mark.parametrize("code", [1, 2])
@pytest.mark.parametrize("d,mode", [(100, 0), (144, 0), (100, 3)])
@pytest.mark.parametrize("k", [1, 16, 17, 25, 33, 64])
def test_blocks_repeat(code, d, mode, k):
    """Three quarters of the references in one tight cluster, 60 queries from it."""
    import torch
    R, Q = clusters(30000, 2048, d, 1, 0.01, 11, "shuffled")
    g = torch.Generator(device="cuda")
    g.manual_seed(k)
    R[::4] = torch.randn(7500, d, generator=g, device="cuda")
    Q[60:] = torch.randn(1988, d, generator=g, device="cuda")
    R[5] = 0.0
    stats = check(R, Q, code, k, mode)
    assert stats["repeated_blocks"] == 1


def test_self_search_own_column():
    """The query's own column in and out of the sample, at the ends of runs."""
    from sparsedist_gb300 import _lib
    R, _ = clusters(20011, 1, 48, 9, 0.3, 5, "in order")
    ctx = _lib.Context()
    h = upload(ctx, R)
    for q0, nq in ((0, 700), (9000, 300), (19900, 111)):
        got, want = (dense_knn(ctx, h, q0, nq, 1, 4, mode) for mode in (0, 2))
        assert same_bits(got[0], want[0]) and same_bits(got[1], want[1])
    ctx.lib.sdg_dense_free(h)
