"""Small tensor-core IVF batches, set up by one CTA: the same results as the sampled path's (another set-up and
selection) for the same queries, the plan's candidate counts, and shards of the lists."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["tc", "tc_sq8"])
@pytest.mark.parametrize("nq,npc,shard,cap", [(1, 1, False, 0), (1, 4, False, 0), (3, 7, False, 0), (33, 31, False, 0),
                                              (128, 8, False, 0), (255, 4, True, 0), (40, 9, False, 900), (17, 40, True, 0)])
def test_equals_the_sampled_path(cuda, mode, nq, npc, shard, cap):
    import torch
    from annvedi_b200.ivf import IVFIndex
    rng = np.random.default_rng(nq + npc)
    c, dim, n = 40, 56, 12000
    cen = rng.standard_normal((c, dim)).astype(np.float32)
    sizes = rng.integers(60, 560, c)
    assign = rng.permutation(np.repeat(np.arange(c), sizes)[:n]).astype(np.int32)
    n = len(assign)
    x = (cen[assign] + 0.4 * rng.standard_normal((n, dim))).astype(np.float32)
    q = (cen[rng.integers(0, c, nq)] + 0.4 * rng.standard_normal((nq, dim))).astype(np.float32)
    ix = IVFIndex(device=0, mode=mode)
    ix.fit(x, 1, 0, c, centroids=cen, assign=assign)
    qd = torch.from_numpy(q).cuda()
    k, R = 20, 50
    out = []
    for sampled_min in (256, 1):
        ix.set_option("sampled_min_queries", sampled_min)
        ix.reset_distances_count()
        ids, d = ix.search(qd, k, 0, npc, R, max_candidates=cap, shard=shard)
        torch.cuda.synchronize()
        out.append((ids.cpu().numpy(), d.cpu().numpy(), ix.total_distances_count()))
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])
    assert out[0][2] == out[1][2]
