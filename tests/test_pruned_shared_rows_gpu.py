"""Few queries with wide windows: a query's rows are shared by several blocks of the finishing kernel. Ids and distances of the
plain scan, bit for bit, at the edges of a block's round (512 or 256 rows) and of the survivors' buffer."""
import numpy as np
import pytest

from tests.test_pruned_exact_gpu import _data, _plain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("metric", ["l2", "ip"])
@pytest.mark.parametrize("n,dim,nq,k,group", [
    (20000, 64, 1, 100, 400), (20000, 64, 1, 100, 513), (40000, 96, 5, 10, 1025), (40000, 96, 3, 100, 2000),
    (30000, 200, 18, 50, 3000), (30000, 64, 74, 20, 900), (30000, 64, 75, 20, 900), (50000, 33, 8, 400, 6000),
    (20000, 3000, 2, 300, 1500), (70000, 48, 37, 1, 4000),
])
def test_wide_windows(cuda, metric, n, dim, nq, k, group):
    """Groups of near-copies around each query: their keys lie within the window of the k-th, their FP32 distances differ."""
    import torch
    from annvedi_b200.linear import LinearIndex
    rng = np.random.default_rng(n + dim + nq + group)
    x = rng.standard_normal((n, dim)).astype(np.float32)
    q = rng.standard_normal((nq, dim)).astype(np.float32)
    at = rng.permutation(n)
    for i in range(min(nq, n // group)):
        x[at[i * group:(i + 1) * group]] = q[i] * (2 if metric == "ip" else 1) + 1e-3 * rng.standard_normal((group, dim))
    ix = LinearIndex(device=0, metric=metric, mode="exact")
    ix.fit(torch.from_numpy(x).cuda())
    qd = torch.from_numpy(q).cuda()
    ix.search_tc(qd[:1], 1)  # the BF16 copy is there: the next exact search prunes
    wi, wd = _plain(ix, qd, k)
    for _ in range(3):
        ids, d = ix.search(qd, k)
        torch.cuda.synchronize()
        np.testing.assert_array_equal(ids.cpu().numpy(), wi)
        np.testing.assert_array_equal(d.cpu().numpy(), wd)
        if ix.get_prune_stats()["skip"]:
            break
    assert ix.get_prune_stats()["passes"] >= 1
