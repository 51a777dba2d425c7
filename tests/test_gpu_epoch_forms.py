"""Every way an epoch is launched -- three, six or eight warps a segment, one
warp a segment, dependent on the previous kernel or after it -- at the sizes
where one gives way to the next: bitmasks and lists against the cursor scan,
bit for bit, over a run of epochs and in pieces."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

umapcu = pytest.importorskip("umapcu")
from tests.test_gpu_layout_resident import _graph

EPOCHS = 9

# segments x 32 points; on 148 SMs: 444, 700, 1000, a third of 5920 = 1973, half
# = 2960, 0.78 = 4602, 5920, 1.27 = 7493; six blocks an SM: half of 3552 = 1776,
# 3552, 7104
SEGMENTS_2D = [444, 445, 699, 700, 1001, 1973, 1974, 2960, 2961, 4602, 4603, 5920, 5921, 7493, 7494]


def _check(n, n_dim, dens=None):
    adj = _graph(n, 6, n)
    y0 = np.random.default_rng(n).uniform(-10, 10, (n, n_dim)).astype(np.float32)
    p = umapcu.UmapOptimParams(n_epochs=EPOCHS)
    st = umapcu.UmapGpuState(y0, adj, p, dens, 3)
    got = []
    for form in (umapcu.SCHED_SCAN, umapcu.SCHED_BITS, umapcu.SCHED_LISTS):
        st.set_schedule(form)
        assert st.schedule_form() == form
        st.reset(y0)
        st.run(0, 4)
        st.run(4, EPOCHS - 4)
        got.append(st.read()[:3])
    st.close()
    for other in got[1:]:
        for a, b in zip(got[0], other):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("segments", SEGMENTS_2D)
def test_two_dimensions(segments):
    _check(32 * segments - (segments % 3), 2)


@pytest.mark.parametrize("segments", [699, 700, 1776, 1777, 3552, 7104, 7105])
def test_three_dimensions(segments):
    _check(32 * segments - 1, 3)


@pytest.mark.parametrize("segments", [1331, 1332, 1776, 1777, 3552, 3553, 7105])
def test_density_term(segments):
    n = 32 * segments - 5
    rng = np.random.default_rng(segments)
    dens = umapcu.DensState(umapcu.DensParams(frac=0.5), rng.normal(size=n).astype(np.float32), np.ones(n, np.float32), float(n))
    _check(n, 2, dens)
