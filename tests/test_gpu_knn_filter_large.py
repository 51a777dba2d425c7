"""The kNN filter at more points than 32 bits hold threads for them (32 threads
a row from 2^27 rows on): neighbours of queries on both sides of that row
against distances in 64 bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

umapcu = pytest.importorskip("umapcu")


def test_more_than_two_to_27_points():
    torch = pytest.importorskip("torch")
    n, dim, k, nq, checked = 2 ** 27 + 1000, 3, 5, 2048, 24
    if torch.cuda.mem_get_info()[0] < 60 << 30:
        pytest.skip("needs 60 GB of device memory")
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.rand(n, dim, generator=g, device="cuda")
    q = torch.randint(0, n, (nq,), generator=g, device="cuda", dtype=torch.int64)
    q[: checked // 2] = torch.arange(n - checked // 2, n, device="cuda")  # rows past 2^27
    q = q.to(torch.int32)
    idx = torch.empty(nq, k, dtype=torch.int32, device="cuda")
    dist = torch.empty(nq, k, device="cuda")
    umapcu._check(umapcu._lib.umapcu_knn_exact_dev(x.data_ptr(), n, dim, q.data_ptr(), nq, k, 0, idx.data_ptr(),
                                                   dist.data_ptr(), None))
    torch.cuda.synchronize()
    for i in range(checked):
        row = int(q[i])
        d = torch.zeros(n, dtype=torch.float64, device="cuda")
        for c in range(dim):
            d += (x[:, c].double() - x[row, c].double()) ** 2
        d[row] = float("inf")
        v, want = torch.topk(d, k, largest=False)
        # distances of three terms in 32 bits: within 8 roundings; no two of the
        # nearest are nearer to one another than that
        assert torch.equal(idx[i].long(), want)
        assert np.allclose(dist[i].double().cpu().numpy(), v.cpu().numpy(), rtol=8 * 2.0 ** -24, atol=0)
        del d, v, want
    del x
    torch.cuda.empty_cache()
