"""Chosen queries: few of them (the tile kernel) and enough for the filter give
the rows of the search over all points, and searches of several query batches
those of one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

umapcu = pytest.importorskip("umapcu")
from oracle import oracle as O

torch = pytest.importorskip("torch")


def _chosen(X, q, k, metric):
    x = torch.from_numpy(X).cuda()
    qd = torch.from_numpy(q.astype(np.int32)).cuda()
    idx = torch.empty(q.size, k, dtype=torch.int32, device="cuda")
    dist = torch.empty(q.size, k, device="cuda")
    torch.cuda.synchronize()
    umapcu._check(umapcu._lib.umapcu_knn_exact_dev(x.data_ptr(), X.shape[0], X.shape[1], qd.data_ptr(), q.size, k,
                                                   umapcu._metric(metric), idx.data_ptr(), dist.data_ptr(), None))
    torch.cuda.synchronize()
    return idx.cpu().numpy(), dist.cpu().numpy()


# the line between the two: 6000 x 10, k = 3: 600 (below it 4M pairs: 700);
# 6000 x 190, k = 15: 1074; 50k x 20, k = 3: 343; 300k x 4, k = 32: 72; 6000 x 10,
# k = 1: 2700 (12M pairs: 2098), k = 2: 1399 (8M); 20k x 4, k = 1: 2045
@pytest.mark.parametrize("n,dim,k,metric,counts", [(6000, 10, 3, "euclidean", (1, 64, 65, 699, 700, 2000)),
                                                   (6000, 190, 15, "cosine", (129, 1073, 1075)),
                                                   (50_000, 20, 3, "euclidean", (5, 342, 344, 513)),
                                                   (300_000, 4, 32, "euclidean", (63, 71, 73, 200)),
                                                   (6000, 10, 1, "euclidean", (2699, 2700)), (6000, 10, 2, "cosine", (1398, 1399)),
                                                   (20_000, 4, 1, "euclidean", (2044, 2046))])
def test_chosen_queries(n, dim, k, metric, counts):
    rng = np.random.default_rng(n + dim)
    X = (rng.normal(size=(n, dim)) * rng.uniform(0.3, 2, (n, 1))).astype(np.float32)
    allq = rng.permutation(n)[: max(counts)]
    ai, ad = umapcu.knn_exact(X, k, metric)
    for c in counts:
        q = allq[:c]
        gi, gd = _chosen(X, q, k, metric)
        assert np.array_equal(gi, ai[q]) and np.array_equal(gd, ad[q])


def test_several_batches_of_queries():
    """80k queries are more than two waves of 256-query blocks: the first and
    last rows of both batches against the tile kernel's."""
    n, k = 80_000, 10
    X = np.random.default_rng(3).normal(size=(n, 5)).astype(np.float32)
    ai, ad = umapcu.knn_exact(X, k)
    edge = 2 * 148 * 256
    q = np.concatenate([np.arange(40), np.arange(edge - 40, edge + 40), np.arange(n - 40, n)])
    gi, gd = _chosen(X, q, k, "euclidean")  # 200 queries: the tile kernel
    assert np.array_equal(gi, ai[q]) and np.array_equal(gd, ad[q])


def test_ranks_of_several_batches_of_queries():
    """16 384 queries are a batch of the rank filter: over 20 000 the mean of two
    halves of one batch each."""
    n, k = 20_000, 12
    rng = np.random.default_rng(4)
    X = rng.normal(size=(n, 6)).astype(np.float32)
    Y = X[:, :2] + 0.5 * rng.normal(size=(n, 2)).astype(np.float32)
    t = [umapcu.embedding_quality(X, Y, None, k, queries=q)["trust"]
         for q in (np.arange(n), np.arange(n // 2), np.arange(n // 2, n))]
    # sums of whole numbers below 2^53 times one factor: a few roundings
    assert abs(t[0] - 0.5 * (t[1] + t[2])) < 1e-14
    sub = rng.choice(n, 60, replace=False)
    got = umapcu.embedding_quality(X, Y, None, k, queries=sub)["trust"]
    assert got == O.trustworthiness(X, Y, k, queries=sub.astype(np.uint32))


# queries the filter cannot settle (their equal rows overflow a candidate list),
# among others it settles: one, just below, at and above a group of 64, and
# nearly all; few of them split the points, many do not
@pytest.mark.parametrize("metric,members", [("euclidean", (1, 63, 64, 65, 390)), ("cosine", (2, 300))])
def test_queries_left_by_the_filter(metric, members):
    n, dim, k = 50_000, 20, 3
    rng = np.random.default_rng(8)
    X = rng.normal(size=(n, dim)).astype(np.float32)
    X[20_000:20_600] = X[20_000]  # more equal rows in a tile than a part's list holds
    others = np.concatenate([np.arange(0, 20_000, 37), np.arange(21_000, n, 37)])
    for m in members:
        inside = 20_000 + rng.permutation(600)[:m]
        q = rng.permutation(np.concatenate([inside, others[: 400 - m]]))
        gi, gd = _chosen(X, q, k, metric)
        for part in np.array_split(np.arange(q.size), 4):  # 100 queries: the tile kernel
            ti, td = _chosen(X, q[part], k, metric)
            assert np.array_equal(gi[part], ti) and np.array_equal(gd[part], td)


def test_all_queries_left_by_the_filters():
    """Tight clusters far apart: every list overflows, and all queries make more
    groups than blocks."""
    n, k = 40_000, 5
    rng = np.random.default_rng(9)
    X = (10 * rng.normal(size=(4, 8))[rng.integers(0, 4, n)] + 1e-3 * rng.normal(size=(n, 8))).astype(np.float32)
    gi, gd = umapcu.knn_exact(X, k)
    q = rng.permutation(n)[:200]
    ti, td = _chosen(X, q, k, "euclidean")
    assert np.array_equal(gi[q], ti) and np.array_equal(gd[q], td)
    Y = X[:, :2].copy()
    sub = rng.permutation(n)[:1000].astype(np.uint32)
    t = [umapcu.embedding_quality(X, Y, None, k, queries=s)["trust"] for s in [sub] + list(sub.reshape(10, 100))]
    assert abs(t[0] - np.mean(t[1:])) < 1e-13
