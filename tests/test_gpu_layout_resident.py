"""Small one-shot layouts (all epochs in one cooperative launch) against the
same epochs launched one by one from a resident state: the same batches and
sums, so bit for bit equal, at the edges of the launch's forms."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

umapcu = pytest.importorskip("umapcu")


def _graph(n, degree, seed, hub=False):
    """A random symmetric weighted adjacency, rows and columns ascending."""
    rng = np.random.default_rng(seed)
    i = rng.integers(0, n, n * degree // 2)
    j = rng.integers(0, n, n * degree // 2)
    if hub:
        i = np.concatenate([i, np.zeros(n - 1, np.int64)])
        j = np.concatenate([j, np.arange(1, n)])
    i, j = i[i != j], j[i != j]
    key = np.unique(np.minimum(i, j) * n + np.maximum(i, j))
    a, b = key // n, key % n
    w = np.exp(rng.uniform(np.log(0.01), 0, key.size)).astype(np.float32)
    row, col, val = np.concatenate([a, b]), np.concatenate([b, a]), np.concatenate([w, w])
    order = np.lexsort((col, row))
    ptr = np.zeros(n + 1, np.uint64)
    ptr[1:] = np.cumsum(np.bincount(row, minlength=n))
    return umapcu.Adjacency(ptr, col[order].astype(np.uint32), val[order])


# 33 points: a segment of one node; 148 / 296 / 444 / 592 segments (4 736,
# 9 472, 14 208, 18 944 points) are the most of each form, one point more goes
# to the next (past the last: a launch per epoch); degree 60: several rounds of
# batches a segment; the hub's segment is too long for a block
@pytest.mark.parametrize("n,degree,n_dim,epochs,sgd,hub", [(33, 4, 2, 30, False, False), (1000, 20, 3, 41, False, False),
                                                           (2048, 60, 2, 40, True, False), (18_944, 12, 2, 12, False, False),
                                                           (18_945, 12, 3, 12, False, False), (4_737, 10, 2, 19, True, False),
                                                           (9_473, 40, 2, 18, False, False), (14_209, 10, 3, 12, False, False),
                                                           (4_736, 70, 3, 21, False, False), (9_500, 8, 2, 16, False, True),
                                                           (700, 10, 2, 3, False, False), (500, 10, 1, 12, False, False)])
def test_one_launch_equals_launch_per_epoch(n, degree, n_dim, epochs, sgd, hub):
    adj = _graph(n, degree, n + degree, hub)
    y0 = np.random.default_rng(n).uniform(-10, 10, (n, n_dim)).astype(np.float32)
    p = umapcu.UmapOptimParams(n_epochs=epochs)
    opt = umapcu.OPT_SGD if sgd else umapcu.OPT_ADAM
    y = y0.copy()
    umapcu.optimise_embedding_adam_gpu(y, adj, p, None, 11, optimiser=opt)
    st = umapcu.UmapGpuState(y0, adj, p, None, 11)
    st.run(0, epochs, opt)
    assert np.array_equal(y, st.read()[0])
    st.close()


def test_one_launch_then_density_epochs_and_log_lines(capfd):
    """densMAP: the epochs before the density term in one launch, the others
    one by one; printed gradient norms (verbose) do not change the result."""
    n = 1500
    adj = _graph(n, 16, 3)
    rng = np.random.default_rng(4)
    r = rng.normal(size=n).astype(np.float32)
    dens = umapcu.DensState(umapcu.DensParams(), r, np.ones(n, np.float32), float(n))
    y0 = rng.uniform(-10, 10, (n, 2)).astype(np.float32)
    p = umapcu.UmapOptimParams(n_epochs=230)
    y = y0.copy()
    umapcu.optimise_embedding_adam_gpu(y, adj, p, dens, 5, verbose=1)
    assert capfd.readouterr().out.count("grad norm") == 3  # epochs 100, 200, 230
    st = umapcu.UmapGpuState(y0, adj, p, dens, 5)
    st.run(0, 230)
    assert np.array_equal(y, st.read()[0])
    st.close()
