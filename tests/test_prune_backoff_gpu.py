"""The exact search over bases on which its tensor-core passes settle few queries: it goes back to the scan alone, tries again
ever more rarely, and the results are the plain scan's throughout (as in test_pruned_exact_gpu)."""
import numpy as np
import pytest

from tests.test_pruned_exact_gpu import _data, _plain

pytestmark = pytest.mark.gpu


def _index(x, metric="l2"):
    import torch
    from annvedi_b200.linear import LinearIndex
    ix = LinearIndex(device=0, metric=metric, mode="exact")
    ix.fit(torch.from_numpy(x).cuda())
    ix.search_tc(torch.from_numpy(x[:1]).cuda(), 1)  # the BF16 copy is there: the next exact search prunes
    return ix


def _run(ix, q, k, calls):
    import torch
    wi, wd = _plain(ix, q, k)
    for _ in range(calls):
        ids, d = ix.search(q, k)
        torch.cuda.synchronize()
        np.testing.assert_array_equal(ids.cpu().numpy(), wi)
        np.testing.assert_array_equal(d.cpu().numpy(), wd)
    return ix.get_prune_stats()


@pytest.mark.parametrize("kind,metric,n,dim,nq,k", [("offset", "ip", 40000, 32, 37, 50), ("offset", "l2", 20000, 64, 1, 100),
                                                    ("copies", "l2", 30000, 48, 300, 20)])
def test_passes_that_settle_nothing_become_rare(cuda, kind, metric, n, dim, nq, k):
    import torch
    if kind == "copies":
        rng = np.random.default_rng(n)
        x = rng.standard_normal((n, dim)).astype(np.float32)
        x[rng.permutation(n)[: n // 3]] = x[0]
        q = (x[:1] + 0.1 * rng.standard_normal((nq, dim))).astype(np.float32)
    else:
        x, q = _data("offset", n, dim, nq, np.random.default_rng(n))
    ix = _index(x, metric)
    s = _run(ix, torch.from_numpy(q).cuda(), k, 60)
    assert s["queries"] == nq and s["left"] == nq
    # calls 1, 6 (after 4), 15 (8), 32 (16); the next would be 65
    assert s["passes"] == 4 and s["skip"] > 0


def test_a_settled_pass_ends_it(cuda):
    """Queries far outside the bound, then ordinary ones: the next try settles and every call after it prunes; a new fit starts
    afresh."""
    import torch
    x, q = _data("normal", 30000, 64, 20, np.random.default_rng(4))
    ix = _index(x)
    s = _run(ix, torch.from_numpy(q * np.float32(1e17)).cuda(), 10, 1)
    assert (s["passes"], s["left"]) == (1, 20)
    s = _run(ix, torch.from_numpy(q).cuda(), 10, 5)
    assert (s["passes"], s["left"], s["skip"]) == (2, 0, 0)
    s = _run(ix, torch.from_numpy(q).cuda(), 10, 5)
    assert (s["passes"], s["left"]) == (7, 0)
    # a few query tiles of many are not a reason (5 queries of 400 are one tile of 13 at most)
    mixed = np.tile(q, (20, 1))
    mixed[:5] = np.nan
    s = _run(ix, torch.from_numpy(mixed).cuda(), 10, 3)
    assert (s["passes"], s["left"]) == (10, 5)
    s = _run(ix, torch.from_numpy(q * np.float32(1e17)).cuda(), 10, 1)
    ix.fit(torch.from_numpy(x + 1).cuda())
    ix.search_tc(torch.from_numpy(q[:1]).cuda(), 1)
    assert _run(ix, torch.from_numpy(q).cuda(), 10, 2)["passes"] == 13


def test_one_query_of_a_small_batch_is_its_whole_scan(cuda):
    """The scan of one left query of 6 reads the base as for all six: such passes are backed off from."""
    import torch
    x, q = _data("normal", 30000, 64, 6, np.random.default_rng(5))
    q[2] = np.nan
    ix = _index(x)
    s = _run(ix, torch.from_numpy(q).cuda(), 10, 7)
    assert (s["passes"], s["left"], s["skip"]) == (2, 1, 7)  # calls 1 and 6; the seventh reads the sixth's end: 8 calls


def test_a_new_fit_reads_no_old_end(cuda):
    """Two passes under way, the first leaving every query and the second none, then a new base: its passes are its own."""
    import torch
    x, q = _data("normal", 30000, 64, 20, np.random.default_rng(6))
    good, bad = torch.from_numpy(q).cuda(), torch.from_numpy(q * np.float32(1e17)).cuda()
    ix = _index(x)
    ix.search(good, 10)
    torch.cuda.synchronize()
    busy = torch.randn(8192, 8192, device="cuda")
    for _ in range(8):
        busy = busy @ busy * 1e-4  # the passes below are queued behind this
    ix.search(bad, 10)
    ix.search(good, 10)
    assert ix.get_prune_stats()["passes"] == 3
    ix.fit(torch.from_numpy(x + 1).cuda())
    ix.search_tc(good[:1], 1)
    s = _run(ix, good, 10, 3)
    assert (s["passes"], s["left"], s["skip"]) == (6, 0, 0)
