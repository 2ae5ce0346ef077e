"""Batches with queries whose probed lists hold fewer than k rows: those are set apart by the plan and scored over every
row together. Each query's result equals its own small call's, for all three scoring forms, and the counter counts
every row for them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["exact", "tc", "tc_sq8"])
@pytest.mark.parametrize("n,k,R,short", [(6000, 50, 100, 1), (6000, 50, 300, 90), (700, 60, 900, 40)])
def test_short_queries_in_a_batch(cuda, mode, n, k, R, short):
    import torch
    from annvedi_b200.ivf import IVFIndex
    rng = np.random.default_rng(n + short)
    c, dim, nq = 20, 48, 300
    cen = rng.standard_normal((c, dim)).astype(np.float32)
    # lists 0 and 1 are tiny twins, far from the others: a query there probes both and stays short of k
    cen[0] += 20.0
    cen[1] = cen[0] + 0.05
    assign = rng.integers(2, c, n).astype(np.int32)
    assign[:15], assign[15:25] = 0, 1
    x = (cen[assign] + 0.2 * rng.standard_normal((n, dim))).astype(np.float32)
    x[400:500] = x[300:400]  # equal keys among the rows
    own = rng.integers(2, c, nq)
    own[rng.permutation(nq)[:short]] = 0
    q = (cen[own] + 0.2 * rng.standard_normal((nq, dim))).astype(np.float32)
    ix = IVFIndex(device=0, mode=mode)
    ix.fit(x, 1, 0, c, centroids=cen, assign=assign)
    qd = torch.from_numpy(q).cuda()
    sizes = np.bincount(assign, minlength=c)
    ix.reset_distances_count()
    ids, d = ix.search(qd, k, 0, 2, R)
    torch.cuda.synchronize()
    probes = np.argsort(((cen[None].astype(np.float64) - q[:, None]) ** 2).sum(-1), axis=1, kind="stable")[:, :2]
    cands = sizes[probes].sum(1)
    assert (cands < k).sum() == short
    assert ix.total_distances_count() == int(np.where(cands < k, n, cands).sum())
    ids, d = ids.cpu().numpy(), d.cpu().numpy()
    for i in np.flatnonzero(cands < k)[:12]:  # alone, by the exact form: the SQ8 keys of every row
        one, od = ix.search(qd[i:i + 1], k, 0, 2, R, mode="exact")
        np.testing.assert_array_equal(ids[i], one[0].cpu().numpy())
        np.testing.assert_array_equal(d[i], od[0].cpu().numpy())
