"""Index checks of short arrays, on the host, and of arrays just past the line, on
the device: the same calls are refused and the same pass."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

umapcu = pytest.importorskip("umapcu")
K = 4


def _ring(n):
    """n points in a ring with K neighbours each, rows ascending: n K entries."""
    i = np.repeat(np.arange(n), K)
    j = (i + np.tile([1, n - 1, 2, n - 2], n)) % n
    d = np.tile(np.array([1, 1, 2, 2], np.float32), n) * (1.0 + 0.5 * np.sin(i.astype(np.float32)))
    return i.astype(np.uint32), j.astype(np.uint32), np.sort(d.reshape(n, K), axis=1)


def _refused(call):
    with pytest.raises(umapcu.ManifoldsError) as e:
        call()
    assert e.value.status == umapcu.BAD_ARG


# 32 768 entries in all: 4096 points have 2 x 16 384 in the cross-entropy and the
# spectral start, 2730 3 x 10 920 with the neighbours in the density state
@pytest.mark.parametrize("n", [5, 2730, 2731, 4096, 4097])
@pytest.mark.parametrize("array,place,value", [("row", 0, -1), ("col", -1, None), ("col", 7, 2 ** 31), ("nbr", -1, None),
                                               ("nbr", 3, -1), ("order", 9, 0), (None, 0, 0)])
def test_short_and_long_arrays(n, array, place, value):
    row, col, dist = _ring(n)
    nbr = col.astype(np.int64)
    value = n if value is None else value
    if array == "row":
        row[place] = np.uint32(value & 0xFFFFFFFF)
    elif array == "col":
        col[place] = np.uint32(value)
    elif array == "nbr":
        nbr[place] = value
    elif array == "order":
        row[place] = value
    g = umapcu.CoordinateList(row, col, np.linspace(0.2, 1.0, row.size).astype(np.float32), n)
    idx = nbr.astype(np.int32).reshape(n, K)
    y = np.random.default_rng(n).normal(size=(n, 2)).astype(np.float32)
    dens = lambda: umapcu.DensState.new(umapcu.DensParams(), g, idx, dist)  # noqa: E731
    ce = lambda: umapcu.fuzzy_cross_entropy(g, y, 1.5, 0.9)  # noqa: E731
    spec = lambda: umapcu.spectral_layout(g, 2, 1)  # noqa: E731
    if array is None:
        assert np.isfinite(dens().r).all() and np.isfinite(ce()) and np.isfinite(spec()).all()
        return
    _refused(dens)
    if array in ("row", "col"):
        _refused(ce)
        _refused(spec)
    else:
        assert np.isfinite(ce())
