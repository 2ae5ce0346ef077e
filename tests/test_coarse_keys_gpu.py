"""The exact IVF form's coarse ranking by tensor-core keys gives the probes of the exact scan over the centroids: a
batch (keys) returns the ids and distances of the same queries in calls of 8 (scan), bit for bit. Queries set apart
because their lists hold fewer than k rows are among them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c,dim,npc,nq,kind", [
    (256, 40, 1, 32, "normal"), (300, 384, 8, 200, "normal"), (2048, 96, 32, 130, "normal"),
    (257, 500, 5, 64, "twins"), (300, 20, 2, 70, "odd"), (300, 24, 3, 40, "offset"),
])
def test_batch_equals_small_calls(cuda, c, dim, npc, nq, kind):
    import torch
    from annvedi_b200.ivf import IVFIndex
    rng = np.random.default_rng(c + dim + npc)
    cen = rng.standard_normal((c, dim))
    if kind == "twins":  # centroids in equal pairs: their order is by id
        cen[1::2] = cen[:-1:2]
    if kind == "offset":  # the window holds every centroid
        cen = 40.0 + 0.01 * cen
    n = 60 * c
    assign = rng.integers(0, c, n).astype(np.int32)
    assign[: n // 2] = assign[: n // 2] // 3 * 3 % c  # uneven lists, some short
    x = (cen[assign] + 0.3 * rng.standard_normal((n, dim))).astype(np.float32)
    q = (cen[rng.integers(0, c, nq)] + 0.3 * rng.standard_normal((nq, dim))).astype(np.float32)
    if kind == "odd":
        q[3] = 0.0
        q[5] *= 1e17
    ix = IVFIndex(device=0, mode="exact")
    ix.fit(x, 1, 0, c, centroids=cen.astype(np.float32), assign=assign)
    qd = torch.from_numpy(q).cuda()
    k, R = 60, 80
    ids, d = ix.search(qd, k, 0, npc, R)
    for s in range(0, nq, 8):
        e = nq if nq - s < 13 else s + 8  # never a rest of 4 or fewer: another sum order
        i8, d8 = ix.search(qd[s:e], k, 0, npc, R)
        np.testing.assert_array_equal(ids[s:e].cpu().numpy(), i8.cpu().numpy(), err_msg=f"queries {s}..{e}")
        np.testing.assert_array_equal(d[s:e].cpu().numpy(), d8.cpu().numpy(), err_msg=f"queries {s}..{e}")
        if e == nq:
            break
