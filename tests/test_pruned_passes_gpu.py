"""Which exact searches take the tensor-core passes, and a batch of several passes with queries left to the scan in each."""
import numpy as np
import pytest

from tests.test_pruned_exact_gpu import _data, _plain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nq,k,taken", [
    (4095, 5, 10, False), (4096, 5, 64, True), (4096, 5, 65, False), (8191, 3, 10, False), (8192, 2, 100, True),
    (8191, 1, 64, False), (8192, 1, 64, True), (16383, 1, 63, False), (16384, 1, 63, True), (32768, 1, 10, False),
    (199999, 1, 10, False), (200000, 1, 10, True), (32768, 9, 512, True), (32767, 9, 512, False),
])
def test_rule(cuda, n, nq, k, taken):
    import torch
    from annvedi_b200.linear import LinearIndex
    x, q = _data("normal", n, 24, nq, np.random.default_rng(n))
    ix = LinearIndex(device=0, mode="exact")
    ix.fit(torch.from_numpy(x).cuda())
    qd = torch.from_numpy(q).cuda()
    ix.search_tc(qd[:1], 1)  # the BF16 copy is there
    ids, d = ix.search(qd, k)
    torch.cuda.synchronize()
    s = ix.get_prune_stats()
    assert s["passes"] == int(taken)
    if taken:
        assert (s["queries"], s["left"]) == (nq, 0)
    wi, wd = _plain(ix, qd, k)
    np.testing.assert_array_equal(ids.cpu().numpy(), wi)
    np.testing.assert_array_equal(d.cpu().numpy(), wd)


@pytest.mark.parametrize("metric", ["l2", "ip"])
def test_several_passes(cuda, metric):
    """10,300 queries: two passes, the second with a shorter last chunk; uncovered queries in both."""
    import torch
    from annvedi_b200.linear import LinearIndex
    n, dim, nq, k = 8192, 32, 10300, 10
    x, q = _data("normal", n, dim, nq, np.random.default_rng(1))
    bad = [0, 77, 5000, 5151, 5152, 5247, 5248, 10239, 10240, 10299]
    q[bad[::2]] = np.nan
    q[bad[1::2]] *= np.float32(1e17)
    ix = LinearIndex(device=0, metric=metric, mode="exact")
    ix.fit(torch.from_numpy(x).cuda())
    qd = torch.from_numpy(q).cuda()
    ix.search_tc(qd[:1], 1)  # the BF16 copy is there
    ids, d = ix.search(qd, k)
    torch.cuda.synchronize()
    s = ix.get_prune_stats()
    assert s["passes"] == 2 and s["left"] > 0
    wi, wd = _plain(ix, qd, k)
    np.testing.assert_array_equal(ids.cpu().numpy(), wi)
    np.testing.assert_array_equal(d.cpu().numpy(), wd)
