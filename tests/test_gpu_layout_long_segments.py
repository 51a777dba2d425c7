"""Small one-shot layouts with a segment too long for the launch of all epochs:
every epoch runs once from the start, and each printed line is that of the
launches per epoch."""
import re

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

umapcu = pytest.importorskip("umapcu")
from tests.test_gpu_layout_resident import _graph


def _run(capfd, adj, y0, p, dens, n_dim):
    y = y0.copy()
    umapcu.optimise_embedding_adam_gpu(y, adj, p, dens, 5, verbose=1)
    out = capfd.readouterr().out
    return y, re.findall(r"Epoch (\d+) / \d+: grad norm ([^\s]+)", out)


# odd and even numbers of epochs before the first line; with the density term
# (half of the epochs)
@pytest.mark.parametrize("n_dim,epochs,with_dens", [(2, 230, False), (3, 101, False), (2, 7, False), (2, 120, True)])
def test_long_segment_with_log_lines(capfd, monkeypatch, n_dim, epochs, with_dens):
    n = 9_500
    adj = _graph(n, 8, 17, hub=True)
    rng = np.random.default_rng(epochs)
    y0 = rng.uniform(-10, 10, (n, n_dim)).astype(np.float32)
    dens = None
    if with_dens:
        dens = umapcu.DensState(umapcu.DensParams(frac=0.5), rng.normal(size=n).astype(np.float32), np.ones(n, np.float32),
                                float(n))
    p = umapcu.UmapOptimParams(n_epochs=epochs)
    got, lines = _run(capfd, adj, y0, p, dens, n_dim)
    want_epochs = [e for e in range(1, epochs + 1) if e % 100 == 0 or e == epochs]
    assert [int(e) for e, _ in lines] == want_epochs
    monkeypatch.setenv("UMAPCU_NO_SCHEDULE_LISTS", "1")  # no precomputed schedule: an epoch per launch
    want, per_launch = _run(capfd, adj, y0, p, dens, n_dim)
    assert np.array_equal(got, want)
    assert lines == per_launch
