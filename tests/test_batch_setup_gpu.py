"""The set-up of an IVF batch (pairs grouped by list, offsets, tiles, operand rows) at list and query counts around its
block's 1,024 threads: a batch gives what calls of other sizes, set up differently or not at all, give, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,c,nq,npc,small", [
    ("exact", 1, 32, 1, 31), ("exact", 1023, 40, 33, 20), ("exact", 1024, 1025, 3, 16), ("exact", 2100, 3000, 2, 25),
    ("tc", 1, 300, 1, 100), ("tc", 1023, 257, 40, 128), ("tc", 1025, 1024, 5, 200), ("tc", 2100, 3001, 2, 250),
    ("tc_sq8", 1024, 1025, 4, 255), ("tc_sq8", 65, 2500, 64, 250),
])
def test_batch_equals_small_calls(cuda, mode, c, nq, npc, small):
    import torch
    from annvedi_b200.ivf import IVFIndex
    rng = np.random.default_rng(c + nq)
    dim, n = 24, max(4000, 40 * c)
    cen = rng.standard_normal((c, dim)).astype(np.float32)
    assign = rng.integers(0, c, n).astype(np.int32)
    assign[: n // 2] = assign[: n // 2] // 4 * 4  # uneven lists, some empty-handed
    x = (cen[assign] + 0.3 * rng.standard_normal((n, dim))).astype(np.float32)
    q = torch.from_numpy((cen[rng.integers(0, c, nq)] + 0.3 * rng.standard_normal((nq, dim))).astype(np.float32)).cuda()
    ix = IVFIndex(device=0, mode=mode)
    ix.fit(x, 1, 0, c, centroids=cen, assign=assign)
    k, R = 10, 40
    ids, d = ix.search(q, k, 0, npc, R)
    for s in range(0, nq, small):
        i2, d2 = ix.search(q[s:s + small], k, 0, npc, R)
        np.testing.assert_array_equal(ids[s:s + small].cpu().numpy(), i2.cpu().numpy(), err_msg=f"from {s}")
        np.testing.assert_array_equal(d[s:s + small].cpu().numpy(), d2.cpu().numpy(), err_msg=f"from {s}")
        if s > 8 * small:
            break
