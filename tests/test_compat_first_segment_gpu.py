"""The reference ranking of the linear scan where the first segment's walk is cut (rows 64, 128, 256, 512 and 1024): ids
and ranking values equal the CPU restatement's, bit for bit, with thresholds that fall at every row, equal distances,
and rows whose distance is not finite."""
import numpy as np
import pytest

from oracle import refmod

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 63, 64, 65, 128, 129, 256, 300, 512, 1024, 1100, 200000])
@pytest.mark.parametrize("k,order", [(1, "random"), (63, "falling"), (64, "random"), (100, "falling"), (64, "ties"),
                                     (100, "inf")])
def test_reference_ranking_equals_the_restatement(cuda, n, k, order):
    from annvedi_b200.linear import LinearIndex
    if k > n:
        k = n
    rng = np.random.default_rng(n + k)
    dim = 112
    x = rng.standard_normal((n, dim)).astype(np.float32)
    if order == "ties":
        x = x[: max(1, n // 50)][rng.integers(0, max(1, n // 50), n)]
    if order == "falling":
        r = np.linspace(2.0, 1.0, n)
        x = (x / np.linalg.norm(x, axis=1, keepdims=True) * r[:, None]).astype(np.float32)
    if order == "inf" and n > 300:  # never held by the heap, and not among the best
        x[rng.integers(0, 300, 40)] = 1e25
    q = rng.standard_normal((2, dim)).astype(np.float32)
    if order == "falling":
        q *= 1e-3
    ix = LinearIndex(device=0, mode="reference")
    ix.fit(x)
    ids, vals = ix.search(q, k)
    oids, ovals = refmod.linear_query(x, q, k, lanes=16)
    np.testing.assert_array_equal(ids, oids)
    np.testing.assert_array_equal(vals, ovals)
