"""Exact kNN through the tensor-core filter: bit for bit the oracle's lists at
the filter's edges -- partial tiles and query blocks, the dims where its
operands change form, the smallest and largest k, and data its bounds cannot
settle (ties beyond the candidate lists, wide ranges, non-finite rows)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

umapcu = pytest.importorskip("umapcu")
from oracle import oracle as O


def _same(X, k, metric="euclidean"):
    gi, gd = umapcu.knn_exact(X, k, metric)
    oi, od = O.knn_exact(X, k, metric=umapcu._metric(metric))
    assert np.array_equal(gi.astype(np.uint32), oi)
    assert np.array_equal(gd, od)


# 2048 points: the smallest search; 255 / 257 rows past a tile; dims 10 / 11
# (six and three products), 20 / 21, 41 / 42, 62 / 63 (chunks of 64 columns;
# two query blocks a block up to 63), 191 (the widest)
@pytest.mark.parametrize("n,dim,k,metric", [(2048, 2, 15, "euclidean"), (2303, 10, 1, "euclidean"),
                                            (2561, 11, 32, "euclidean"), (4097, 20, 15, "cosine"),
                                            (4096, 21, 15, "euclidean"), (3000, 41, 7, "euclidean"),
                                            (3000, 42, 30, "cosine"), (5003, 62, 15, "euclidean"),
                                            (2500, 63, 15, "euclidean"), (2100, 191, 5, "euclidean"),
                                            (2100, 192, 5, "euclidean"), (20_001, 1, 15, "euclidean")])
def test_filter_bit_exact(n, dim, k, metric):
    rng = np.random.default_rng(n + dim)
    c = rng.normal(0, 5, (8, dim))
    X = (c[rng.integers(0, 8, n)] + rng.normal(size=(n, dim)) * rng.uniform(0.3, 2, (n, 1))).astype(np.float32)
    _same(X, k, metric)


@pytest.mark.parametrize("kind", ["duplicates", "few_values", "offset", "outliers", "tiny", "zero_rows", "sorted"])
def test_filter_hard_data(kind):
    rng = np.random.default_rng(5)
    n, dim = 3000, 12
    X = rng.normal(size=(n, dim)).astype(np.float32)
    metric = "euclidean"
    if kind == "duplicates":  # more equal points than a candidate list holds
        X[:1500] = X[0]
    elif kind == "few_values":
        X = np.round(X[:, :3]).astype(np.float32)
    elif kind == "offset":  # distances small beside the coordinates
        X = (X * 1e-2 + 1000.0).astype(np.float32)
    elif kind == "outliers":
        X[::100] *= 1e6
    elif kind == "tiny":
        X = (X * 1e-25).astype(np.float32)
    elif kind == "zero_rows":
        X[::7] = 0.0
        metric = "cosine"
    else:  # neighbours share a place modulo the groups
        X = X[np.argsort(X[:, 0])]
        X = np.ascontiguousarray(X.reshape(24, 125, dim).transpose(1, 0, 2).reshape(n, dim))
    _same(X, 15, metric)


@pytest.mark.parametrize("value", [np.inf, 1e20])
def test_filter_data_beyond_its_bound(value):
    """Rows whose norms the bound cannot hold send the whole search to the
    tile kernel: finite rows keep the oracle's lists."""
    X = np.random.default_rng(6).normal(size=(2500, 8)).astype(np.float32)
    X[17, 3] = value
    gi, gd = umapcu.knn_exact(X, 10)
    oi, od = O.knn_exact(X, 10)
    ok = np.arange(2500) != 17
    assert np.array_equal(gi.astype(np.uint32)[ok], oi[ok]) and np.array_equal(gd[ok], od[ok])


def test_filter_query_subset():
    """The metrics' query rows (any order) through the filter."""
    rng = np.random.default_rng(7)
    X = rng.normal(size=(9000, 6)).astype(np.float32)
    Y = X[:, :2].copy()
    sub = rng.choice(9000, 777, replace=False).astype(np.uint32)
    ki, _ = O.knn_exact(X, 15)
    q = umapcu.embedding_quality(X, Y, ki.astype(np.int32), 15, queries=sub)
    assert q["trust"] == O.trustworthiness(X, Y, 15, queries=sub)
    assert q["knn_preservation"] == pytest.approx(O.knn_preservation(ki, Y, 15, queries=sub), abs=1e-12)


# 15 / 16 neighbours: four and five steps of the search; 31: the most, 32: the
# tile kernel; dims 63 / 64: chunks; 191: too wide beside the rank tables; Y
# unrelated to X: thresholds all over the distances
@pytest.mark.parametrize("n,dim,k,metric,kind", [(2048, 3, 15, "euclidean", "plain"), (3001, 50, 16, "euclidean", "plain"),
                                                 (2500, 63, 31, "euclidean", "plain"), (2500, 64, 32, "euclidean", "plain"),
                                                 (2600, 100, 15, "cosine", "plain"), (2100, 191, 15, "euclidean", "plain"),
                                                 (3000, 10, 15, "euclidean", "ties"), (3000, 8, 1, "cosine", "ties"),
                                                 (4000, 12, 15, "euclidean", "offset"), (3000, 12, 15, "euclidean", "duplicates"),
                                                 (2500, 6, 15, "euclidean", "infinite")])
def test_rank_filter_counts(n, dim, k, metric, kind):
    rng = np.random.default_rng(n + dim + k)
    X = rng.normal(size=(n, dim)).astype(np.float32)
    if kind == "ties":
        X = np.round(X).astype(np.float32) + 1.0
    elif kind == "offset":  # every point within the bound of every threshold: lists overflow
        X = (X * 1e-3 + 1000.0 * np.sign(X[:, :1])).astype(np.float32)
    elif kind == "duplicates":
        X[: n // 2] = X[0]
    elif kind == "infinite":
        X[5, 1] = 1e20
    Y = rng.normal(size=(n, 2)).astype(np.float32)
    q = rng.choice(n, 700, replace=False).astype(np.uint32)
    got = umapcu.embedding_quality(X, Y, None, k, queries=q, dist_metric=metric)
    assert got["trust"] == O.trustworthiness(X, Y, k, queries=q, metric=umapcu._metric(metric))
