"""Large copies of pageable host arrays (several threads through page-locked
slots) against the runtime's copies of smaller ones: whole chunks, remainders
and several callers at once give the same bytes."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

umapcu = pytest.importorskip("umapcu")


def _rows(n, k, seed):
    d = np.sort(np.random.default_rng(seed).exponential(size=(n, k)), axis=1)
    return np.ascontiguousarray(d, np.float32)


def _by_parts(d):
    parts = [umapcu.smooth_knn_dist(d[i:i + 200_000]) for i in range(0, d.shape[0], 200_000)]
    return [np.concatenate([p[t] for p in parts]) for t in range(2)]


# 8 MiB up and 16 MiB down are the least such copies, a chunk 1 MiB: rows of 4 k
# bytes up and 4 bytes a row down, at the least sizes, one short of them, and
# with odd remainders
@pytest.mark.parametrize("n,k", [(524_287, 4), (524_288, 4), (524_289, 4), (4_194_303, 1), (4_194_304, 1), (4_500_007, 1)])
def test_large_copies_equal_small_ones(n, k):
    d = _rows(n, k, n)
    sigma, rho = umapcu.smooth_knn_dist(d)
    want = _by_parts(d)
    assert np.array_equal(sigma, want[0]) and np.array_equal(rho, want[1])


def test_large_copies_from_several_threads():
    data = [_rows(4_300_000 + i, 1, i) for i in range(4)]
    got = [None] * 4

    def work(i):
        got[i] = umapcu.smooth_knn_dist(data[i])

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for i in range(4):
        want = _by_parts(data[i])
        assert np.array_equal(got[i][0], want[0]) and np.array_equal(got[i][1], want[1])
    umapcu.release_cached()  # the block is given back, and allocated again by the next
    again = umapcu.smooth_knn_dist(data[0])
    assert np.array_equal(again[0], got[0][0])
