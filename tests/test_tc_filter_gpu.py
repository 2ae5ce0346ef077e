"""The dense tensor-core filter pass at the edges of its tiles, through search_tc.

The oracle takes the key of every (query, row) from the key-matrix GEMM (scores_tc, another kernel), keeps the best R
per query and re-ranks them in FP64. Sizes: one CTA a tile (up to 128 queries) and pairs, the last pair half empty,
a ragged last base tile, a last k-block of one MMA, query tiles that stay in shared memory and that do not.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,metric", [("bf16", "l2"), ("bf16", "ip"), ("e4m3", "l2"), ("e4m3", "ip")])
@pytest.mark.parametrize("n,dim,nq", [
    (131072, 20, 1), (140001, 64, 128), (140001, 384, 129), (150000, 126, 257), (140255, 700, 300),
])
def test_filter_keeps_the_best_keys(cuda, precision, metric, n, dim, nq):
    import torch
    from annvedi_b200.linear import LinearIndex
    g = torch.Generator(device="cuda").manual_seed(n + dim + nq)
    c = torch.randn(40, dim, generator=g, device="cuda")
    base = c[torch.randint(0, 40, (n,), generator=g, device="cuda")] + 0.5 * torch.randn(n, dim, generator=g, device="cuda")
    q = c[torch.randint(0, 40, (nq,), generator=g, device="cuda")] + 0.5 * torch.randn(nq, dim, generator=g, device="cuda")
    ix = LinearIndex(device=0, metric=metric, mode="exact")
    ix.fit(base)
    ix.set_tc_precision(precision)
    k, R = 10, 60
    ids, d = ix.search_tc(q, k, refine_r=R)
    keys = ix.scores_tc(q)
    cand = torch.topk(keys, R, largest=False).indices
    x = base[cand].double()
    want = (x * q.double()[:, None, :]).sum(-1) if metric == "ip" else ((x - q.double()[:, None, :]) ** 2).sum(-1)
    want = torch.sort(want, 1, descending=metric == "ip").values[:, :k]
    # FP32 sums of dim terms against FP64: relative to the terms' absolute sum, dim 2^-24 at most
    scale = (base[cand].abs().double() * q.abs().double()[:, None, :]).sum(-1).amax(1) if metric == "ip" else want[:, -1]
    tol = (dim + 8) * 2.0 ** -24 * scale.cpu().numpy()[:, None]
    assert (np.abs(d.double().cpu().numpy() - want.cpu().numpy()) <= tol).all()
    got = base[ids].double()
    got = (got * q.double()[:, None, :]).sum(-1) if metric == "ip" else ((got - q.double()[:, None, :]) ** 2).sum(-1)
    assert (np.abs(got.cpu().numpy() - want.cpu().numpy()) <= tol).all()  # the ids hold those distances
