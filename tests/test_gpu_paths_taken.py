"""The fast paths are the ones taken on ordinary data: results alone cannot tell,
as every one of them has an exact fallback. Kernels and copies are listed by the
profiler, in a process of its own."""
import json
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

pytest.importorskip("umapcu")

CHILD = r"""
import json
import sys
sys.path[:0] = sys.argv[1:]
import numpy as np
import torch
import umapcu
from torch.profiler import ProfilerActivity, profile
from tests.test_gpu_layout_resident import _graph


def events(f):
    f()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        f()
    return [(e.name, e.time_range.end - e.time_range.start) for e in p.events() if e.device_type.name == "CUDA"]


rng = np.random.default_rng(0)
out = {}
n = 4000
adj, y0 = _graph(n, 10, 1), rng.uniform(-10, 10, (n, 2)).astype(np.float32)
ev = events(lambda: umapcu.optimise_embedding_adam_gpu(y0.copy(), adj, umapcu.UmapOptimParams(n_epochs=60), None, 3))
out["resident"] = sum("k_layout_resident" in name for name, _ in ev)
out["epochs"] = sum("k_epoch" in name for name, _ in ev)
d = np.sort(rng.exponential(size=(4_500_000, 1)), axis=1).astype(np.float32)  # 18 MB up, 2 x 18 MB down
ev = events(lambda: umapcu.smooth_knn_dist(d))
out["staged_up"] = sum("HtoD" in name and "Pinned" in name for name, _ in ev)
out["staged_down"] = sum("DtoH" in name and "Pinned" in name for name, _ in ev)
X = rng.normal(size=(20_000, 30)).astype(np.float32)
Y = X[:, :2].copy()
equal = np.ones_like(X)
q = np.arange(3000, dtype=np.uint32)


def left(f, kernel):  # the tile kernel behind the filter
    ev = events(f)
    return sum(kernel in name for name, _ in ev), max(t for name, t in ev if "k_knn_tile" in name)


out["knn"] = left(lambda: umapcu.knn_exact(X, 15), "k_refine")
out["knn_equal"] = left(lambda: umapcu.knn_exact(equal, 15), "k_refine")
out["rank"] = left(lambda: umapcu.embedding_quality(X, Y, None, 15, q), "k_rank_refine")
out["rank_equal"] = left(lambda: umapcu.embedding_quality(equal, Y, None, 15, q), "k_rank_refine")
print("RESULT " + json.dumps(out))
"""


def test_paths_taken_on_ordinary_data():
    pytest.importorskip("torch")
    from tests.conftest import PKG_ROOT, ROOT
    r = subprocess.run([sys.executable, "-c", CHILD, PKG_ROOT, ROOT], capture_output=True, text=True, timeout=300)
    lines = [x for x in r.stdout.splitlines() if x.startswith("RESULT ")]
    assert r.returncode == 0 and lines, r.stdout + r.stderr
    out = json.loads(lines[-1][7:])
    if not out["resident"] and not out["epochs"]:
        pytest.skip("the profiler lists no kernels here")
    assert out["resident"] == 1 and out["epochs"] == 0  # one launch, not repeated
    # (18 MB in 1 MiB chunks)
    assert out["staged_up"] >= 17 and out["staged_down"] >= 34
    for what in ("knn", "rank"):
        used, ordinary = out[what]
        assert used >= 1
        # nothing was left to the tile kernel, which takes all queries of equal rows
        assert ordinary < 0.1 * out[what + "_equal"][1], out
