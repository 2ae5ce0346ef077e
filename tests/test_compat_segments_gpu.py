"""The reference ranking of the linear scan where its rows are cut into segments: ids and ranking values equal the
CPU restatement's, bit for bit, at the segments' edges."""
import numpy as np
import pytest

from oracle import refmod

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dim,k,order", [
    (1023, 20, 64, "random"), (1024, 100, 65, "random"), (1025, 16, 1, "random"), (3000, 512, 100, "ties"),
    (5000, 530, 63, "random"), (131072, 8, 100, "falling"), (140001, 24, 512, "random"), (20000, 96, 100, "rising"),
])
def test_reference_ranking_equals_the_restatement(cuda, n, dim, k, order):
    from annvedi_b200.linear import LinearIndex
    rng = np.random.default_rng(n + dim + k)
    x = rng.standard_normal((n, dim)).astype(np.float32)
    if order == "ties":  # copies of 40 rows: equal distances across every threshold and across the k-th place
        x = x[:40][rng.integers(0, 40, n)]
    elif order != "random":  # distances to the origin fall (an insertion at every row) or rise (none after the first)
        r = np.linspace(2.0, 1.0, n) if order == "falling" else np.linspace(1.0, 2.0, n)
        x = (x / np.linalg.norm(x, axis=1, keepdims=True) * r[:, None]).astype(np.float32)
    q = rng.standard_normal((3, dim)).astype(np.float32)
    if order in ("falling", "rising"):
        q *= 1e-3
    ix = LinearIndex(device=0, mode="reference")
    ix.fit(x)
    ids, vals = ix.search(q, k)
    oids, ovals = refmod.linear_query(x, q, k, lanes=16)
    np.testing.assert_array_equal(ids, oids)
    np.testing.assert_array_equal(vals, ovals)
