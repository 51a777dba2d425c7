"""Calls of different widths side by side in several threads: what one thread
asks of a kernel's attributes holds for the others too."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

umapcu = pytest.importorskip("umapcu")


def _rings(n, parts, seed):
    """Separate rings of n points each with chords: a graph of that many components."""
    rng = np.random.default_rng(seed)
    i = np.arange(n * parts)
    j = i // n * n + (i + 1) % n
    c = i // n * n + rng.integers(0, n, i.size)
    a, b = np.concatenate([i, i]), np.concatenate([j, c])
    a, b = a[a != b], b[a != b]
    key = np.unique(np.minimum(a, b) * (n * parts) + np.maximum(a, b))
    a, b = key // (n * parts), key % (n * parts)
    row, col = np.concatenate([a, b]), np.concatenate([b, a])
    o = np.lexsort((col, row))
    return umapcu.CoordinateList(row[o].astype(np.uint32), col[o].astype(np.uint32), np.ones(row.size, np.float32), n * parts)


def test_searches_and_spectral_starts_of_different_widths():
    rng = np.random.default_rng(0)
    # 20 and 50 dims: two blocks of queries a block in 193 and 225 KB of shared
    # memory, 100 and 150: one block in 209 and 225 KB; k = 10 and 31: tables of
    # different length
    data = [rng.normal(size=(3000, dim)).astype(np.float32) for dim in (20, 50, 100, 150)]
    q = rng.choice(3000, 1500, replace=False).astype(np.uint32)
    graph = _rings(60, 8, 1)
    calls = [lambda x=x: umapcu.knn_exact(x, 10)[0] for x in data]
    calls += [lambda x=x, k=k: np.float64(umapcu.embedding_quality(x, x[:, :2], None, k, q)["trust"])
              for x, k in ((data[0], 10), (data[1], 31))]
    calls += [lambda d=d: umapcu.spectral_layout(graph, d, 1) for d in (2, 3, 10)]
    want = [f() for f in calls]
    repeats = [120, 120, 60, 60, 60, 60, 10, 10, 10]
    wrong = []

    def work(i):
        try:
            for _ in range(repeats[i]):
                if not np.array_equal(calls[i](), want[i]):
                    wrong.append(i)
        except Exception as e:  # noqa: BLE001
            wrong.append((i, repr(e)))

    threads = [threading.Thread(target=work, args=(i,)) for i in [0, 1, 0, 1] + list(range(len(calls)))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
