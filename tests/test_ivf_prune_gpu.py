"""The exact IVF form's SQ8 selection by tensor-core keys gives what the scan of every candidate gives: a large batch,
called until the index has laid its operand out and after, returns the ids and distances of the same queries in calls of 8
(scan), bit for bit. Among them: rows in equal groups (ties at the R-th distance), lists shorter than k, constant
dimensions, data far from the origin, and queries outside the keys' range (the batch then falls back)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c,per,dim,npc,nq,k,R,kind", [
    (256, 120, 384, 8, 700, 100, 400, "normal"), (300, 200, 100, 32, 400, 1, 1, "normal"),
    (256, 150, 500, 5, 640, 60, 80, "ties"), (400, 100, 129, 16, 1000, 10, 513, "constant"),
    (256, 120, 384, 3, 1900, 20, 64, "offset"), (256, 100, 768, 8, 500, 50, 200, "normal"), (256, 120, 384, 8, 700, 100, 1024, "odd"),
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
    x = (cen[assign] + 0.3 * rng.standard_normal((n, dim))).astype(np.float32)
    if kind == "ties":
        x = x[np.arange(n) // 3 * 3]
    if kind == "constant":
        x[:, ::3] = 7.0
    q = (cen[rng.integers(0, c, nq)] + 0.3 * rng.standard_normal((nq, dim))).astype(np.float32)
    if kind == "odd":
        q[3] = 0.0
        q[5] *= 1e17
    ix = IVFIndex(device=0, mode="exact")
    ix.fit(x, 1, 0, c, centroids=cen.astype(np.float32), assign=assign)
    qd = torch.from_numpy(q).cuda()
    calls = [ix.search(qd, k, 0, npc, R) for _ in range(12)]
    pick = np.concatenate([np.arange(24), nq // 2 + np.arange(24), np.arange(nq - 16, nq)])
    for s in range(0, len(pick), 8):
        rows = torch.from_numpy(pick[s:s + 8]).cuda()
        i8, d8 = ix.search(qd[rows].contiguous(), k, 0, npc, R)
        for ids, d in (calls[0], calls[-1]):
            np.testing.assert_array_equal(ids[rows].cpu().numpy(), i8.cpu().numpy(), err_msg=f"queries {pick[s:s + 8]}")
            np.testing.assert_array_equal(d[rows].cpu().numpy(), d8.cpu().numpy(), err_msg=f"queries {pick[s:s + 8]}")
    for ids, d in calls[1:]:
        assert torch.equal(ids, calls[0][0]) and torch.equal(d, calls[0][1])
