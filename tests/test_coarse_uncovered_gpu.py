"""Coarse rankings by keys of queries at the ends of the keys' range, in the tensor-core forms and the exact one: tiny and
zero queries rank the centroids by their FP32 distances like any other, and in the tensor-core forms a query that compares
with no centroid (NaN, an infinite component) probes list 0 for each of its probes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["tc", "tc_sq8", "exact"])
@pytest.mark.parametrize("c,dim,nq", [(300, 48, 40), (700, 200, 300)])
def test_probes_of_uncovered_queries(cuda, mode, c, dim, nq):
    import torch
    from annvedi_b200.ivf import IVFIndex
    rng = np.random.default_rng(c)
    npc, k = 4, 10
    sizes = 30 + np.arange(c)  # a list's size names it
    cen = rng.standard_normal((c, dim)).astype(np.float32)
    assign = np.repeat(np.arange(c), sizes).astype(np.int32)
    x = (cen[assign] + 0.1 * rng.standard_normal((len(assign), dim))).astype(np.float32)
    ix = IVFIndex(device=0, mode=mode)
    ix.fit(x, 1, 0, c, centroids=cen, assign=assign)

    def probed(q):
        ix.reset_distances_count()
        ix.search(torch.from_numpy(q).cuda(), k, 0, npc, 40)
        torch.cuda.synchronize()
        return ix.total_distances_count()

    for scale in (1.0, 1e-13, 1e-20, 1e-23, 1e-30, 1e-41, 0.0):
        q = (cen[rng.integers(0, c, nq)] * np.float32(scale)).astype(np.float32)
        d = ((q[:, None].astype(np.float64) - cen[None]) ** 2).sum(-1)
        want = sizes[np.argsort(d, axis=1, kind="stable")[:, :npc]].sum()
        assert probed(q) == want, scale
    if mode != "exact":
        for bad in (np.nan, np.inf, -np.inf):
            q = cen[rng.integers(0, c, nq)].copy()
            q[:, dim // 2] = bad
            assert probed(q) == nq * npc * sizes[0], bad
