"""NaN queries in a batch of the exact IVF form answer as they do in calls of 8: no list compares with them and no key of
theirs is a number, so ids are -1 and distances +inf; the batch's other queries are untouched."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(c, dim, nq, k, npc, R, sizes, seed):
    import torch
    from annvedi_b200.ivf import IVFIndex
    rng = np.random.default_rng(seed)
    cen = rng.standard_normal((c, dim)).astype(np.float32)
    assign = np.repeat(np.arange(c), sizes).astype(np.int32)
    x = (cen[assign] + 0.3 * rng.standard_normal((len(assign), dim))).astype(np.float32)
    q = (cen[rng.integers(0, c, nq)] + 0.3 * rng.standard_normal((nq, dim))).astype(np.float32)
    bad = rng.permutation(nq)[: max(1, nq // 9)]
    q[bad, rng.integers(0, dim, len(bad))] = np.nan
    ix = IVFIndex(device=0, mode="exact")
    ix.fit(x, 1, 0, c, centroids=cen, assign=assign)
    qd = torch.from_numpy(q).cuda()
    out = torch.full((nq, k), -7, dtype=torch.int64, device="cuda"), torch.full((nq, k), -7.0, device="cuda")
    ids, d = ix.search(qd, k, 0, npc, R, out_ids=out[0], out_dists=out[1])
    small = [ix.search(qd[s:s + 8].contiguous(), k, 0, npc, R) for s in range(0, nq, 8)]
    np.testing.assert_array_equal(ids.cpu().numpy(), torch.cat([s[0] for s in small]).cpu().numpy())
    np.testing.assert_array_equal(d.cpu().numpy(), torch.cat([s[1] for s in small]).cpu().numpy())
    assert (ids[torch.from_numpy(bad).cuda()] == -1).all() and torch.isinf(d[torch.from_numpy(bad).cuda()]).all()
    return ix


@pytest.mark.parametrize("c,dim,nq,k,npc,R", [(20, 48, 100, 50, 2, 100), (40, 100, 300, 20, 3, 20)])
def test_nan_queries_that_scan_every_row(cuda, c, dim, nq, k, npc, R):
    """Lists of 5 rows among longer ones: a query of no list is one short of k, which scans every row."""
    _check(c, dim, nq, k, npc, R, [5, 5, 5] + [150] * (c - 3), c)


@pytest.mark.parametrize("c,dim,nq,k,npc,R", [(256, 48, 64, 10, 4, 40), (300, 384, 200, 20, 8, 80), (2048, 33, 90, 5, 32, 20)])
def test_nan_queries_ranked_by_centroid_keys(cuda, c, dim, nq, k, npc, R):
    """256 lists and more: the batch's coarse ranking by keys."""
    _check(c, dim, nq, k, npc, R, [21 + i % 7 for i in range(c)], c + dim)
