"""A set query tile changes the exact scan's tile alone: the search still prunes, and gives the staged scan's ids and distances
bit for bit for every batch size; set_pruning(False) gives them without a pass. What the tuner leaves set prunes too."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq", [1, 3, 40])
@pytest.mark.parametrize("metric", ["l2", "ip"])
def test_pruned_with_a_set_tile(cuda, metric, nq):
    import torch
    from annvedi_b200.linear import LinearIndex
    rng = np.random.default_rng(nq)
    ix = LinearIndex(device=0, metric=metric, mode="exact")
    ix.fit(rng.standard_normal((30000, 100)).astype(np.float32))
    q = torch.from_numpy(rng.standard_normal((nq, 100)).astype(np.float32)).cuda()
    ix.search_tc(q[:1], 1)  # the BF16 copy is there: the next exact search prunes
    for tile in (8, 16, 32):
        ix.set_query_tile(tile)
        ix.set_pruning(False)
        before = ix.get_prune_stats()["passes"]
        want = ix.search(q, 64)
        assert ix.get_prune_stats()["passes"] == before
        ix.set_pruning(True)
        got = ix.search(q, 64)
        torch.cuda.synchronize()
        s = ix.get_prune_stats()
        assert (s["passes"], s["queries"], s["left"]) == (before + 1, nq, 0)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


def test_tuned_tile_keeps_pruning(cuda):
    import torch
    from annvedi_b200 import autotune
    from annvedi_b200.linear import LinearIndex
    rng = np.random.default_rng(1)
    ix = LinearIndex(device=0, mode="exact")
    ix.fit(rng.standard_normal((100000, 64)).astype(np.float32))
    q = torch.from_numpy(rng.standard_normal((500, 64)).astype(np.float32)).cuda()
    autotune.tune_flat_tile(ix, q, k=10)
    before = ix.get_prune_stats()["passes"]
    ix.search(q, 10)
    assert ix.get_prune_stats()["passes"] == before + 1
