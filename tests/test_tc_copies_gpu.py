"""Tensor-core searches of bases with more copies of a row than a query's survivor buffer holds, among ordinary queries: every
query's distances are those of its exact nearest rows (the re-rank is exact, and R takes in every nearer row), and the
ordinary queries' results are those of the same base without the copies' queries beside them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["bf16", "e4m3"])
@pytest.mark.parametrize("n,dim,copies,nq,near,k,R", [
    (200000, 9, 60000, 5, 2, 100, 100), (200000, 9, 60000, 5, 5, 100, 200), (140001, 64, 3000, 400, 3, 10, 100),
    (300000, 40, 250000, 130, 130, 20, 50), (140001, 64, 1700, 257, 200, 10, 100),
])
def test_many_copies(cuda, precision, n, dim, copies, nq, near, k, R):
    import torch
    from annvedi_b200.linear import LinearIndex
    rng = np.random.default_rng(n + copies + nq)
    x = rng.standard_normal((n, dim)).astype(np.float32)
    x[rng.permutation(n)[:copies]] = x[0]
    q = rng.standard_normal((nq, dim)).astype(np.float32) * 3
    at = rng.permutation(nq)[:near]
    q[at] = x[0] + 0.01 * rng.standard_normal((near, dim)).astype(np.float32)
    ix = LinearIndex(device=0, mode="exact")
    ix.fit(x)
    ix.set_tc_precision(precision)
    ix.set_pruning(False)
    qd = torch.from_numpy(q).cuda()
    ids, d = ix.search_tc(qd, k, refine_r=R)
    torch.cuda.synchronize()
    # the copies are nearer to `at` than anything else: k distances, all that of x[0], in FP32 as the re-rank forms it
    near_d = d[torch.from_numpy(at).cuda()].cpu().numpy()
    want = ((q[at].astype(np.float64) - x[0]) ** 2).sum(1)
    np.testing.assert_allclose(near_d, np.repeat(want[:, None], k, 1), rtol=dim * 2.0 ** -23)
    got = np.sort(ids[torch.from_numpy(at).cuda()].cpu().numpy(), 1)
    assert (np.diff(got, axis=1) > 0).all()  # k different rows
    assert (np.abs(x[got.ravel()] - x[0]).max(1) == 0).all()
    rest = np.setdiff1d(np.arange(nq), at)
    if len(rest):
        alone = ix.search_tc(qd[torch.from_numpy(rest).cuda()].contiguous(), k, refine_r=R)
        assert torch.equal(d[torch.from_numpy(rest).cuda()], alone[1])
