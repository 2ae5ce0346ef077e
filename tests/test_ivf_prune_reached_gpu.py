"""The exact IVF form's SQ8 selection by tensor-core keys, at sizes that take it: batches that it settled and batches that it
left equal the same queries in calls of 8 (the scan), bit for bit. Among them: groups of equal rows (ties at the R-th distance),
lists shorter than k, constant dimensions, data far from the origin, and queries outside the keys' range (the batch is left)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c,per,dim,npc,nq,k,R,kind", [
    (64, 1200, 256, 8, 700, 100, 400, "normal"), (64, 1200, 256, 8, 700, 1, 1, "normal"),
    (300, 500, 100, 32, 900, 10, 100, "normal"), (40, 2500, 500, 3, 900, 60, 80, "ties"),
    (64, 1200, 129, 16, 1000, 10, 513, "constant"), (64, 1200, 384, 3, 1900, 20, 64, "offset"),
    (50, 1500, 768, 8, 500, 50, 200, "normal"), (64, 1500, 384, 8, 700, 100, 1024, "normal"),
    (64, 1200, 256, 8, 700, 100, 400, "odd"), (64, 1200, 256, 2, 4000, 50, 100, "short"),
])
def test_batch_equals_small_calls(cuda, c, per, dim, npc, nq, k, R, kind):
    import torch
    from annvedi_b200.ivf import IVFIndex
    rng = np.random.default_rng(c + dim + npc)
    cen = rng.standard_normal((c, dim))
    if kind == "offset":
        cen += 300.0
    n = per * c
    assign = rng.integers(0, c, n).astype(np.int32)
    assign[: n // 3] = assign[: n // 3] // 5 * 5 % c  # uneven lists
    if kind == "short":  # lists of a few rows beside the others: their queries scan every row
        cen[:4] = cen[0] + 0.01 * rng.standard_normal((4, dim))
        assign[assign < 4] = 7
        assign[:12] = np.arange(12) % 4
    x = (cen[assign] + 0.3 * rng.standard_normal((n, dim))).astype(np.float32)
    if kind == "ties":
        x = x[np.arange(n) // 3 * 3]
    if kind == "constant":
        x[:, ::3] = 7.0
    own = rng.integers(4 if kind == "short" else 0, c, nq)
    if kind == "short":
        own[::50] = 1
    q = (cen[own] + 0.3 * rng.standard_normal((nq, dim))).astype(np.float32)
    if kind == "odd":
        q[3] = 0.0
        q[5] *= 1e17
    ix = IVFIndex(device=0, mode="exact")
    ix.fit(x, 1, 0, c, centroids=cen.astype(np.float32), assign=assign)
    qd = torch.from_numpy(q).cuda()
    calls = [ix.search(qd, k, 0, npc, R) for _ in range(12)]
    s = ix.get_prune_stats()
    assert s["batches"] >= 1  # taken
    # left: queries out of range; constant dimensions, whose codes' distance from their centre widens every window; a buffer of
    # 16 survivors. Such a batch is not tried again by the 16 calls that follow.
    left = kind in ("odd", "constant") or R == 1
    assert s == ({"batches": 1, "settled": 0} if left else {"batches": s["batches"], "settled": s["batches"]})
    pick = np.concatenate([np.arange(24), nq // 2 + np.arange(24), np.arange(nq - 16, nq)])
    for p0 in range(0, len(pick), 8):
        rows = torch.from_numpy(pick[p0:p0 + 8]).cuda()
        i8, d8 = ix.search(qd[rows].contiguous(), k, 0, npc, R)
        for ids, d in (calls[0], calls[-1]):
            np.testing.assert_array_equal(ids[rows].cpu().numpy(), i8.cpu().numpy(), err_msg=f"queries {pick[p0:p0 + 8]}")
            np.testing.assert_array_equal(d[rows].cpu().numpy(), d8.cpu().numpy(), err_msg=f"queries {pick[p0:p0 + 8]}")
    for ids, d in calls[1:]:
        assert torch.equal(ids, calls[0][0]) and torch.equal(d, calls[0][1])
