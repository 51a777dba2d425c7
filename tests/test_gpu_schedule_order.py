"""Epochs enqueued straight behind the kernels that build their schedule: they
read the words of this graph, not what another graph left in the cached block."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

umapcu = pytest.importorskip("umapcu")
from tests.test_gpu_layout_resident import _graph

EPOCHS = 12


# eight warps a segment, six, three (2D: 700 segments and a third of 5920), one
@pytest.mark.parametrize("n,n_dim", [(9_001, 2), (40_000, 2), (200_000, 2), (130_000, 2), (30_000, 3)])
def test_bitmasks_then_run(n, n_dim):
    adj, old = _graph(n, 6, n), _graph(n + 501, 7, n + 1)
    rng = np.random.default_rng(n)
    y0 = rng.uniform(-10, 10, (n, n_dim)).astype(np.float32)
    p = umapcu.UmapOptimParams(n_epochs=EPOCHS)
    st = umapcu.UmapGpuState(y0, adj, p, None, 3)
    st.set_schedule(umapcu.SCHED_SCAN)
    st.reset(y0)
    st.run(0, EPOCHS)
    want = st.read()[:3]
    for _ in range(3):
        st.set_schedule(umapcu.SCHED_SCAN)
        st.reset(y0)
        # another graph's words into the block the next build takes
        other = umapcu.UmapGpuState(rng.uniform(-10, 10, (n + 501, n_dim)).astype(np.float32), old, p, None, 4)
        other.set_schedule(umapcu.SCHED_BITS)
        other.close()
        st.set_schedule(umapcu.SCHED_BITS)
        st.run(0, EPOCHS)
        for a, b in zip(st.read()[:3], want):
            assert np.array_equal(a, b)
    st.close()
