"""The batched form's launches per epoch at the lines where they stop overlapping
the one before: each layout equals its own run from a resident state, bit for
bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

umapcu = pytest.importorskip("umapcu")
from tests.test_gpu_layout_resident import _graph


# four warps, and 32-point segments, a block: 444 blocks in two dimensions, 148 in
# three, 296 in four, 592 outside the fast configuration, 1184 all
@pytest.mark.parametrize("n_dim,blocks,neg", [(2, 444, 5), (2, 445, 5), (3, 148, 5), (3, 149, 5), (4, 296, 5), (4, 297, 5),
                                              (3, 592, 3), (3, 593, 3), (2, 1184, 5), (2, 1185, 5)])
def test_lines_of_the_launch_forms(n_dim, blocks, neg):
    segments = 4 * blocks
    sizes = [32 * 100, 32 * 37, 32 * (segments - 137)]
    p = umapcu.UmapOptimParams(n_epochs=9)
    p.neg_sample_rate = neg
    graphs = [_graph(n, 6, n) for n in sizes]
    starts = [np.random.default_rng(n).uniform(-10, 10, (n, n_dim)).astype(np.float32) for n in sizes]
    b = umapcu.UmapBatch(starts, graphs, p, [5, 6, 7])
    b.run(2)
    got = [b.read(i) for i in range(3)]
    b.close()
    for i in range(3):
        st = umapcu.UmapGpuState(starts[i], graphs[i], p, None, 5 + i)
        st.run(0, 9)
        assert np.array_equal(got[i], st.read()[0])
        st.close()
