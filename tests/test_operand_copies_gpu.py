"""The operand copies that the exact searches lay out for themselves: none for rows that the keys' bounds do not cover, and one
that did not fit beside what the card holds is not asked for again until the next fit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


class _Filled:
    """All but `left` bytes of the card's free memory held."""

    def __init__(self, left):
        self.left = left

    def __enter__(self):
        import torch
        torch.cuda.empty_cache()
        self.block = torch.empty(_free() - self.left, dtype=torch.uint8, device="cuda")

    def __exit__(self, *exc):
        import torch
        del self.block
        torch.cuda.empty_cache()


def test_uncovered_rows_get_no_copy(cuda):
    import torch
    from annvedi_b200.linear import LinearIndex
    n, dim = 200_000, 256
    x = torch.randn(n, dim, device="cuda")
    x[5, 7] = float("inf")
    ix = LinearIndex(device=0, mode="exact")
    ix.fit(x)
    q = torch.randn(500, dim, device="cuda")
    ix.search(q, 10, mode="exact")  # (this call's estimated savings are beyond the copy's cost)
    torch.cuda.empty_cache()
    before = _free()
    for _ in range(3):
        ix.search(q, 10, mode="exact")
    torch.cuda.empty_cache()
    assert before - _free() < 64 << 20 and ix.get_prune_stats()["passes"] == 0
    fresh = LinearIndex(device=0, mode="exact")
    fresh.fit(x)
    torch.cuda.empty_cache()
    before = _free()
    fresh.search(q, 10, mode="exact")
    torch.cuda.empty_cache()
    assert before - _free() < n * dim * 2  # the scan's scratch, no copy


def test_refused_copy_is_not_asked_for_again(cuda):
    import torch
    from annvedi_b200.linear import LinearIndex
    n, dim = 1_000_000, 512  # the copy: 1.06 GB
    x = torch.randn(n, dim, device="cuda")
    ix = LinearIndex(device=0, mode="exact")
    ix.fit(x)
    q = torch.randn(64, dim, device="cuda")
    want = ix.search(q, 10, mode="exact", workspace=None)
    ix.fit(x)  # (the copy that the call laid out is given back)
    ix.search(q[:1], 10)  # the scan's scratch is there
    with _Filled(1500 << 20):
        for _ in range(3):
            ids, d = ix.search(q, 10)
        torch.cuda.synchronize()
        assert torch.equal(ids, want[0]) and torch.equal(d, want[1])
    for _ in range(3):
        ix.search(q, 10)
    assert ix.get_prune_stats()["passes"] == 1  # the first index state's
    ix.fit(x)
    ids, d = ix.search(q, 10)
    torch.cuda.synchronize()
    assert ix.get_prune_stats()["passes"] == 2
    assert torch.equal(ids, want[0]) and torch.equal(d, want[1])


def test_fit_gives_the_keys_buffers_back(cuda):
    """A k-means fit of rows by tensor-core keys needs no more beside the rows and its state than the scan's: the keys' copy of
    the rows is freed before the lists are laid out."""
    import torch
    from annvedi_b200.ivf import IVFIndex
    n, dim, c = 1_000_000, 256, 256
    x = torch.randn(n, dim, device="cuda")
    want = None
    for left in (None, (n * dim * 9) + (400 << 20)):  # the rows, the lists' rows and codes, and room for the sorts
        ix = IVFIndex(device=0, mode="exact", num_threads=4)
        if left is None:
            ix.fit(x, 1, 0, c, kmeans_iters=1)
        else:
            with _Filled(left):
                ix.fit(x, 1, 0, c, kmeans_iters=1)
        st = ix.export_state()
        ix.close()
        if want is None:
            want = st
        for key in ("centroids", "reordered_to_original", "quantized_data"):
            np.testing.assert_array_equal(st[key], want[key])


@pytest.mark.parametrize("mode,nq,c,sizes,npc,left", [
    ("exact", 16000, 2048, [25] * 2048, 1, 90 << 20),            # 131 MB of coarse keys
    ("tc", 150, 40, [100000] + [60] * 39, 1, 40 << 20),          # 60 MB of stream keys by the largest list
    ("exact", 60, 40, [40000] * 30 + [3] * 10, 2, 20 << 20),     # 192 MB of keys of every row, 40 queries (8 MB of streams)
])
def test_batches_in_little_memory(cuda, mode, nq, c, sizes, npc, left):
    """Batches whose faster form does not fit take the one that does, with the same results."""
    import torch
    from annvedi_b200.ivf import IVFIndex
    rng = np.random.default_rng(nq)
    dim, k = 32, 10
    cen = (10 * rng.standard_normal((c, dim))).astype(np.float32)
    cen[-10:] = cen[-1] + 0.01 * rng.standard_normal((10, dim)).astype(np.float32)
    assign = np.repeat(np.arange(c), sizes).astype(np.int32)
    x = (cen[assign] + 0.3 * rng.standard_normal((len(assign), dim))).astype(np.float32)
    own = rng.integers(1, c - 10, nq)
    if sizes[-1] < k:
        own[:40] = c - 1
    q = torch.from_numpy((cen[own] + 0.3 * rng.standard_normal((nq, dim))).astype(np.float32)).cuda()
    out = [torch.empty(nq, k, dtype=torch.int64, device="cuda"), torch.empty(nq, k, device="cuda")]
    ix = IVFIndex(device=0, mode=mode)
    ix.fit(x, 1, 0, c, centroids=cen, assign=assign)
    want = ix.search(q, k, 0, npc, 20)
    other = IVFIndex(device=0, mode=mode)
    other.fit(x, 1, 0, c, centroids=cen, assign=assign)
    other.search(q[:1], k, 0, npc, 20)
    with _Filled(left):
        got = other.search(q, k, 0, npc, 20, out_ids=out[0], out_dists=out[1])
        torch.cuda.synchronize()
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
