"""The lines where one way of launching an epoch gives way to another in more
than two dimensions, with the density term, and in the configurations that only
the general kernels take: bitmasks and lists against the cursor scan, bit for
bit, over a run of epochs and in pieces."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

umapcu = pytest.importorskip("umapcu")
from tests.test_gpu_layout_resident import _graph

EPOCHS = 7


def _check(segments, n_dim, dens=False, neg=5, precise=False, sampler=None):
    n = 32 * segments - segments % 5
    adj = _graph(n, 6, n)
    rng = np.random.default_rng(n)
    y0 = rng.uniform(-10, 10, (n, n_dim)).astype(np.float32)
    p = umapcu.UmapOptimParams(n_epochs=EPOCHS)
    p.neg_sample_rate = neg
    d = None
    if dens:
        d = umapcu.DensState(umapcu.DensParams(frac=0.6), rng.normal(size=n).astype(np.float32), np.ones(n, np.float32), float(n))
    st = umapcu.UmapGpuState(y0, adj, p, d, 3, umapcu.NEG_REF_HASH if sampler is None else sampler)
    if precise:
        st.set_precise_pow(True)
    got = []
    for form in (umapcu.SCHED_SCAN, umapcu.SCHED_BITS, umapcu.SCHED_LISTS):
        st.set_schedule(form)
        st.reset(y0)
        st.run(0, 4)
        st.run(4, EPOCHS - 4)
        got.append(st.read()[:3])
    st.close()
    for other in got[1:]:
        for a, b in zip(got[0], other):
            assert np.array_equal(a, b)


# lists in 3 (900 and 1331 segments), 4 (850, 1150, 1331; bitmasks 1776, 3552)
# and 5 dimensions (800, 1331)
@pytest.mark.parametrize("n_dim,segments", [(3, 900), (3, 901), (4, 850), (4, 851), (4, 1150), (4, 1151), (4, 1331), (4, 1776),
                                            (4, 1777), (4, 3552), (4, 3553), (5, 800), (5, 801), (5, 1331), (5, 1332),
                                            (8, 7105)])
def test_more_dimensions(n_dim, segments):
    _check(segments, n_dim)


# scans to 444, bitmasks to 500, lists to 560, 1000, 1331 / 1332, 0.53 x 3552 =
# 1882; P = 3552, 1.3 P = 4617, 4 P / 3 = 4736, three warps to 1.8 P = 6390 (2-D)
# and 2 P = 7104
@pytest.mark.parametrize("n_dim,segments", [(2, 444), (2, 445), (2, 500), (2, 501), (2, 560), (2, 561), (2, 1000), (2, 1001),
                                            (2, 1331), (2, 1332), (2, 1882), (2, 1883), (2, 3552), (2, 3553), (2, 4617),
                                            (2, 4618), (2, 4736), (2, 4737), (2, 6390), (2, 6391), (3, 440), (3, 561),
                                            (3, 1332), (3, 3553), (4, 1000), (4, 3553), (4, 4737), (4, 7104), (5, 444),
                                            (5, 445), (5, 1332), (5, 1883), (5, 4737), (6, 7105)])
def test_density_term(n_dim, segments):
    _check(segments, n_dim, dens=True)


# a warp per segment launched after its predecessor (1777 to 3552 segments) and
# dependent, from 4617 on with powf; general kernels in one and two dimensions
@pytest.mark.parametrize("segments", [700, 701, 1331, 1776, 1777, 3552, 3553, 4617, 4618])
@pytest.mark.parametrize("kw", [dict(neg=4), dict(precise=True), dict(sampler=umapcu.NEG_PHILOX), dict(neg=3, dens=True),
                                dict(precise=True, dens=True)])
def test_general_kernels(segments, kw):
    _check(segments, 2 if segments % 2 else 1, **kw)
