"""Large copies in a context that is not the device's primary one: the calling
thread keeps its context and the results are those of the primary one. In a
process of its own, as a second context is created."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

pytest.importorskip("umapcu")

CHILD = r"""
import ctypes as C
import sys
sys.path[:0] = sys.argv[1:]
import numpy as np
import umapcu
cu = C.CDLL("libcuda.so.1")
d = np.sort(np.random.default_rng(0).exponential(size=(4_500_007, 1)), axis=1).astype(np.float32)
want = umapcu.smooth_knn_dist(d)  # 18 MB up and 2 x 18 MB down, the primary context
assert cu.cuInit(0) == 0
dev, ctx, now = C.c_int(), C.c_void_p(), C.c_void_p()
assert cu.cuDeviceGet(C.byref(dev), 0) == 0
assert cu.cuCtxCreate_v2(C.byref(ctx), C.c_uint(0), dev) == 0
small = umapcu.smooth_knn_dist(d[:1000])
got = umapcu.smooth_knn_dist(d)
assert cu.cuCtxGetCurrent(C.byref(now)) == 0 and now.value == ctx.value, (now.value, ctx.value)
assert np.array_equal(small[0], want[0][:1000])
assert all(np.array_equal(a, b) for a, b in zip(got, want))
assert cu.cuCtxDestroy_v2(ctx) == 0
again = umapcu.smooth_knn_dist(d)
assert all(np.array_equal(a, b) for a, b in zip(again, want))
print("context kept")
"""


def test_large_copies_keep_the_callers_context():
    from tests.conftest import PKG_ROOT, ROOT
    r = subprocess.run([sys.executable, "-c", CHILD, PKG_ROOT, ROOT], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "context kept" in r.stdout, r.stdout + r.stderr
