"""Searches whose device waits run out (the self-test option: no copies are issued): the kernels wind down, the status says so,
and the same index answers the next call as before."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TIMEOUT = -5
FLAT_OPT_WAIT_SELFTEST = 2


def _flat(n, dim, nq, precision, rng):
    import torch
    from annvedi_b200.linear import LinearIndex
    ix = LinearIndex(device=0, mode="exact")
    ix.fit(torch.from_numpy(rng.standard_normal((n, dim)).astype(np.float32)).cuda())
    ix.set_tc_precision(precision)
    return ix, torch.from_numpy(rng.standard_normal((nq, dim)).astype(np.float32)).cuda()


# 200,000 rows: the sampled form (tc_filter.cu, one CTA a tile and CTA pairs); 20,000: the key matrix (tc_gemm.cu)
@pytest.mark.parametrize("n,dim,nq,precision", [(200000, 40, 3, "bf16"), (200000, 1000, 20, "bf16"), (200000, 64, 300, "bf16"),
                                                (200000, 64, 300, "e4m3"), (20000, 64, 40, "bf16"), (300, 32, 2, "e4m3")])
def test_flat_tensor_core_search(cuda, n, dim, nq, precision):
    import torch
    ix, q = _flat(n, dim, nq, precision, np.random.default_rng(nq))
    lib = ix._lib
    want = ix.search_tc(q, 10)
    assert lib.ann_flat_device_status(ix._h) == 0
    assert lib.ann_flat_set_option(ix._h, FLAT_OPT_WAIT_SELFTEST, ctypes.c_int64(100000)) == 0
    ix.search_tc(q, 10)
    torch.cuda.synchronize()
    assert lib.ann_flat_device_status(ix._h) == TIMEOUT
    assert lib.ann_flat_device_status(ix._h) == 0  # read and cleared
    with pytest.raises(RuntimeError):
        ix.search_tc(q.cpu().numpy(), 10)
    assert lib.ann_flat_set_option(ix._h, FLAT_OPT_WAIT_SELFTEST, ctypes.c_int64(0)) == 0
    got = ix.search_tc(q, 10)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    assert lib.ann_flat_device_status(ix._h) == 0


@pytest.mark.parametrize("mode", ["tc", "tc_sq8"])
@pytest.mark.parametrize("nq", [1, 40, 400])
def test_ivf_tensor_core_search(cuda, mode, nq):
    import torch
    from annvedi_b200.ivf import IVFIndex
    rng = np.random.default_rng(nq)
    x = rng.standard_normal((20000, 96)).astype(np.float32)
    ix = IVFIndex(device=0, mode=mode)
    ix.fit(x, 1, 0, 64, centroids=x[:64])
    q = torch.from_numpy(rng.standard_normal((nq, 96)).astype(np.float32)).cuda()
    want = ix.search(q, 10, 0, 4, 40)
    assert ix._lib.ann_ivf_device_status(ix._h) == 0
    ix.set_option("wait_selftest", 100000)
    ix.search(q, 10, 0, 4, 40)
    torch.cuda.synchronize()
    assert ix._lib.ann_ivf_device_status(ix._h) == TIMEOUT
    ix.set_option("wait_selftest", 0)
    got = ix.search(q, 10, 0, 4, 40)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    assert ix._lib.ann_ivf_device_status(ix._h) == 0


@pytest.mark.parametrize("metric", ["l2", "ip"])
@pytest.mark.parametrize("n,dim,nq", [(60000, 64, 1), (60000, 64, 40), (40000, 100, 300)])
def test_exact_search_falls_back_to_the_scan(cuda, metric, n, dim, nq):
    """The exact search's tensor-core passes certify nothing where a wait gave up: the scan answers, and no error is left."""
    import torch
    from annvedi_b200.linear import LinearIndex
    from tests.test_pruned_exact_gpu import _plain
    rng = np.random.default_rng(nq)
    ix = LinearIndex(device=0, metric=metric, mode="exact")
    ix.fit(torch.from_numpy(rng.standard_normal((n, dim)).astype(np.float32)).cuda())
    q = torch.from_numpy(rng.standard_normal((nq, dim)).astype(np.float32)).cuda()
    ix.search_tc(q[:1], 1)  # the BF16 copy is there: the next exact search prunes
    good = ix.search(q, 20)
    wi, wd = _plain(ix, q, 20)
    assert ix._lib.ann_flat_set_option(ix._h, FLAT_OPT_WAIT_SELFTEST, ctypes.c_int64(100000)) == 0
    for ids, d in (good, ix.search(q, 20), ix.search(q.cpu().numpy(), 20)):
        np.testing.assert_array_equal(np.asarray(ids.cpu() if torch.is_tensor(ids) else ids), wi)
        np.testing.assert_array_equal(np.asarray(d.cpu() if torch.is_tensor(d) else d), wd)
    assert ix._lib.ann_flat_device_status(ix._h) == 0


@pytest.mark.parametrize("c,sizes,nq,k,npc", [(300, 40, 200, 10, 8), (300, 6, 64, 20, 2), (64, 1200, 600, 20, 8)])
def test_exact_ivf_batch_takes_the_scans(cuda, c, sizes, nq, k, npc):
    """The exact form's rankings by keys: where their waits give up, the batch has the small calls' results and count.
    (300 lists: the coarse ranking; 64: the SQ8 selection, from the call on that has laid its operand out.)"""
    import torch
    from annvedi_b200.ivf import IVFIndex
    rng = np.random.default_rng(c)
    dim = 256
    cen = rng.standard_normal((c, dim)).astype(np.float32)
    assign = np.repeat(np.arange(c), sizes).astype(np.int32)
    x = (cen[assign] + 0.3 * rng.standard_normal((len(assign), dim))).astype(np.float32)
    ix = IVFIndex(device=0, mode="exact")
    ix.fit(x, 1, 0, c, centroids=cen, assign=assign)
    q = torch.from_numpy((cen[rng.integers(0, c, nq)] + 0.3 * rng.standard_normal((nq, dim))).astype(np.float32)).cuda()
    for _ in range(8):
        ix.search(q, k, 0, npc, 4 * k)
    ix.reset_distances_count()
    parts = [ix.search(q[s:s + 8].contiguous(), k, 0, npc, 4 * k) for s in range(0, nq, 8)]
    torch.cuda.synchronize()
    count = ix.total_distances_count()
    ix.set_option("wait_selftest", 100000)
    ix.reset_distances_count()
    ids, d = ix.search(q, k, 0, npc, 4 * k)
    torch.cuda.synchronize()
    assert torch.equal(ids, torch.cat([p[0] for p in parts])) and torch.equal(d, torch.cat([p[1] for p in parts]))
    assert ix.total_distances_count() == count
    assert ix._lib.ann_ivf_device_status(ix._h) == 0


@pytest.mark.parametrize("given", [False, True])
def test_fit_runs_its_rounds_by_the_scan(cuda, given):
    """k-means assignments by keys: where their waits give up, the fit's centroids and lists are the same."""
    from annvedi_b200.ivf import IVFIndex
    rng = np.random.default_rng(3)
    x = rng.standard_normal((9000, 40)).astype(np.float32)
    states = []
    for wait in (0, 100000):
        ix = IVFIndex(device=0, mode="exact", num_threads=4)
        ix.set_option("wait_selftest", wait)
        ix.fit(x, 1, 0, 30, kmeans_iters=4, centroids=x[:30] if given else None)
        states.append(ix.export_state())
    for key in ("centroids", "reordered_to_original", "table_offsets", "quantized_data"):
        np.testing.assert_array_equal(states[0][key], states[1][key])
