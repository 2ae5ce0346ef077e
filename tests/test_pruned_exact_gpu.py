"""The pruned exact scan returns the plain scan's ids and distances bit for bit.

The plain scan is reached through ann_flat_query_noalloc, which never prunes and picks the same query tile by the
batch size (the streaming sums for up to 4 queries, the staged sums above). Bit equality is the property itself, so
no tolerance is involved.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _plain(ix, q, k):
    """ids, distances of the plain scan, in batches of the pruned call's own form that fit the fixed scratch."""
    import torch
    from annvedi_b200 import _lib
    lib = _lib.load()
    nq = q.shape[0]
    step = nq if nq <= 4 else max(5, min(64, (8 << 20) // (k * 8)))
    ids, ds = [], []
    s = 0
    while s < nq:
        e = nq if nq - s < step + 5 else s + step  # never a rest of 4 or fewer: another sum order
        x = q[s:e].contiguous()
        i = torch.empty(e - s, k, dtype=torch.int64, device=q.device)
        d = torch.empty(e - s, k, dtype=torch.float32, device=q.device)
        _lib.check(lib.ann_flat_query_noalloc(ix._h, ctypes.c_void_p(x.data_ptr()), e - s, x.stride(0), k,
                                              ctypes.c_void_p(i.data_ptr()), ctypes.c_void_p(d.data_ptr()),
                                              ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        ids.append(i.cpu().numpy())
        ds.append(d.cpu().numpy())
        s = e
    return np.concatenate(ids), np.concatenate(ds)


def _data(kind, n, dim, nq, rng):
    if kind == "normal":
        x, q = rng.standard_normal((n, dim)), rng.standard_normal((nq, dim))
    elif kind == "clusters":  # a few large clusters: many rows inside the window
        c = rng.standard_normal((12, dim))
        x = c[rng.integers(0, 12, n)] + 0.3 * rng.standard_normal((n, dim))
        q = c[rng.integers(0, 12, nq)] + 0.3 * rng.standard_normal((nq, dim))
    elif kind == "ties":  # copies of few rows: equal distances across the k-th place
        d = rng.standard_normal((300, dim))
        x, q = d[rng.integers(0, 300, n)], rng.standard_normal((nq, dim))
    else:  # "offset": a common offset far above the spread, so that the keys' error covers every row
        x, q = 50.0 + 0.01 * rng.standard_normal((n, dim)), 50.0 + 0.01 * rng.standard_normal((nq, dim))
    return x.astype(np.float32), q.astype(np.float32)


def _check(x, q, k, metric):
    import torch
    from annvedi_b200.linear import LinearIndex
    ix = LinearIndex(device=0, metric=metric, mode="exact")
    ix.fit(torch.from_numpy(x).cuda())
    qd = torch.from_numpy(q).cuda()
    ix.search_tc(qd[:1], 1)  # the BF16 copy is there: the next exact search prunes
    ids, d = ix.search(qd, k)
    wi, wd = _plain(ix, qd, min(k, x.shape[0]))
    np.testing.assert_array_equal(ids.cpu().numpy(), wi)
    np.testing.assert_array_equal(d.cpu().numpy(), wd)
    hi, hd = ix.search(q, k)  # host buffers
    np.testing.assert_array_equal(hi, wi)
    np.testing.assert_array_equal(hd, wd)


@pytest.mark.parametrize("kind,n,dim,nq,k,metric", [
    ("normal", 32768, 20, 5, 1, "l2"),
    ("normal", 70001, 100, 33, 100, "ip"),
    ("normal", 70001, 384, 300, 10, "l2"),
    ("normal", 40000, 64, 9, 512, "l2"),
    ("normal", 140000, 600, 7, 129, "ip"),
    ("normal", 65536, 96, 1, 100, "l2"),
    ("normal", 65536, 96, 2, 10, "ip"),
    ("normal", 65536, 48, 3, 50, "l2"),
    ("clusters", 100003, 128, 40, 100, "l2"),
    ("clusters", 100003, 128, 4, 100, "l2"),
    ("clusters", 50000, 40, 70, 128, "ip"),
    ("ties", 60000, 64, 20, 100, "l2"),
    ("ties", 60000, 64, 1, 100, "ip"),
    ("offset", 40000, 32, 40, 100, "l2"),
    ("offset", 40000, 32, 3, 20, "ip"),
])
def test_equals_the_plain_scan(cuda, kind, n, dim, nq, k, metric):
    x, q = _data(kind, n, dim, nq, np.random.default_rng(n + dim + nq))
    _check(x, q, k, metric)


def test_queries_the_bound_does_not_cover(cuda):
    """A zero query, one of huge norm and one of NaN among ordinary ones: the last two go to the plain scan."""
    rng = np.random.default_rng(5)
    x, q = _data("normal", 40000, 32, 12, rng)
    q[3] = 0.0
    q[5] *= 1e17
    q[7, 2] = np.nan
    _check(x, q, 30, "ip")


@pytest.mark.parametrize("bad", [np.nan, np.inf, 1e20])
def test_rows_the_bound_does_not_cover(cuda, bad):
    rng = np.random.default_rng(6)
    x, q = _data("normal", 40000, 32, 12, rng)
    x[17, 3] = bad
    _check(x, q, 30, "l2")


def test_graph_capture_and_replay(cuda):
    """A captured pruned search replays on new queries with the eager call's results (no host synchronisation)."""
    import torch
    from annvedi_b200 import graphs
    from annvedi_b200.linear import LinearIndex
    x, q = _data("normal", 50000, 64, 48, np.random.default_rng(8))
    ix = LinearIndex(device=0, mode="exact")
    ix.fit(torch.from_numpy(x).cuda())
    ix.search_tc(torch.from_numpy(q[:1]).cuda(), 1)
    g = graphs.flat_exact(ix, 24, 20)
    for s in (0, 24):
        part = torch.from_numpy(q[s:s + 24]).cuda()
        ids, d = g(part)
        torch.cuda.synchronize()
        wi, wd = _plain(ix, part, 20)
        np.testing.assert_array_equal(ids.cpu().numpy(), wi)
        np.testing.assert_array_equal(d.cpu().numpy(), wd)
