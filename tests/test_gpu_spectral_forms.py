"""Where the components' tridiagonal problems move from the host to the device:
two components of 82 (host) and 86 rows, three of any -- each component's leading
coordinates against the oracle's Lanczos of it alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

umapcu = pytest.importorskip("umapcu")
from oracle import oracle as O
from tests.test_gpu_spectral import _neg_norm_adjacency, _strip_graph


@pytest.mark.parametrize("n_comp,sizes", [(2, (300, 450)), (12, (250, 300)), (13, (250, 300)), (2, (200, 300, 90))])
def test_two_and_three_components(n_comp, sizes):
    parts, off = [], 0
    for i, m in enumerate(sizes):
        g = _strip_graph(m, seed=51 + i)
        parts.append((g["row"] + off, g["col"] + off, g["val"]))
        off += m
    r, c, v = (np.concatenate([p[k] for p in parts]) for k in range(3))
    y = umapcu.spectral_layout(umapcu.CoordinateList(r.astype(np.uint32), c.astype(np.uint32), v.astype(np.float32), off),
                               n_comp, seed=9)
    assert y.shape == (off, n_comp) and np.isfinite(y).all()
    off = 0
    for label, m in enumerate(sizes):
        sub = dict(row=parts[label][0] - off, col=parts[label][1] - off, val=parts[label][2])
        _, V = O.lanczos_smallest(_neg_norm_adjacency(sub, m), n_comp + 1, O.splitmix_start(m, 9 + label))
        for d in range(2):  # the modes along the strip, well separated
            assert abs(np.corrcoef(V[:, 1 + d], y[off:off + m, d])[0, 1]) > 0.9999, (label, d)
        off += m
