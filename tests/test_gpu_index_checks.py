"""Indices out of range in the callers' arrays are refused (the checks run on the
device, before anything reads at the indices' places), at the first, the last
and an inner entry, and a valid call afterwards gives what it gave before."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

umapcu = pytest.importorskip("umapcu")
from tests._problems import oracle_graph

N = 2500


@pytest.fixture(scope="module")
def prob():
    return oracle_graph(n=N, dim=30, k=15, n_epochs=60)


def _refused(call):
    with pytest.raises(umapcu.ManifoldsError) as e:
        call()
    assert e.value.status == umapcu.BAD_ARG


@pytest.mark.parametrize("value", [-1, N, 2 ** 31 - 1])
@pytest.mark.parametrize("place", [0, 12_345, N * 15 - 1])
def test_neighbours_out_of_range(prob, place, value):
    idx = np.array(prob["idx"], np.int32)
    good = umapcu.construct_umap_graph(idx, prob["dist"], None, 60)
    bad = idx.copy()
    bad.reshape(-1)[place] = value
    _refused(lambda: umapcu.construct_umap_graph(bad, prob["dist"], None, 60))
    _refused(lambda: umapcu.DensState.new(umapcu.DensParams(), good, bad, prob["dist"]))
    again = umapcu.construct_umap_graph(idx, prob["dist"], None, 60)
    assert np.array_equal(good.values, again.values) and np.array_equal(good.col_indices, again.col_indices)


@pytest.mark.parametrize("place", ["first", "inner", "last"])
@pytest.mark.parametrize("array,value", [("row", N), ("row", 2 ** 32 - 1), ("col", N), ("col", 2 ** 32 - 1), ("order", 0)])
def test_graph_entries_out_of_range(prob, place, array, value):
    row, col = np.array(prob["row"], np.uint32), np.array(prob["col"], np.uint32)
    at = {"first": 0, "inner": row.size // 3, "last": row.size - 1}[place]
    if array == "order":  # rows that go back: refused where the rows must be grouped
        if place == "first":
            pytest.skip("nothing before the first entry")
        row[at] = 0
    else:
        (row if array == "row" else col)[at] = value
    g = umapcu.CoordinateList(row, col, prob["val"], N)
    _refused(lambda: umapcu.DensState.new(umapcu.DensParams(), g, prob["idx"], prob["dist"]))
    if array != "order":
        _refused(lambda: umapcu.spectral_layout(g, 2, 1))
        _refused(lambda: umapcu.fuzzy_cross_entropy(g, np.zeros((N, 2), np.float32), 1.5, 0.9))
    ok = umapcu.CoordinateList(prob["row"], prob["col"], prob["val"], N)
    assert np.isfinite(umapcu.DensState.new(umapcu.DensParams(), ok, prob["idx"], prob["dist"]).r).all()
