"""The reference ranking under NaN: a row of NaN distance is never held by the heap and orders after every number, and a
query whose distances are all NaN gets the first rows with NaN values."""
import numpy as np
import pytest

from oracle import refmod

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dim,k", [(300, 20, 5), (1500, 33, 70), (9000, 96, 200)])
def test_nan_rows_order_last(cuda, n, dim, k):
    from annvedi_b200.linear import LinearIndex
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, dim)).astype(np.float32)
    bad = rng.permutation(n)[: n // 10]
    x[bad, dim // 2] = np.nan
    bad = np.isnan(x).any(1)
    q = rng.standard_normal((3, dim)).astype(np.float32)
    ix = LinearIndex(device=0, mode="reference")
    ix.fit(x)
    ids, v = ix.search(q, k)
    # rows that never enter the heap change nothing for the others: the oracle over the rest
    wi, wv = refmod.linear_query(np.ascontiguousarray(x[~bad]), q, k, lanes=16)
    np.testing.assert_array_equal(ids, np.flatnonzero(~bad)[wi])
    np.testing.assert_array_equal(v, wv)
    kk = min(n, 512)
    ids, v = ix.search(q[:1], kk)
    if kk == n:  # every row is returned: the NaN rows last, by row
        np.testing.assert_array_equal(ids[0, (~bad).sum():], np.flatnonzero(bad))
        assert np.isnan(v[0, (~bad).sum():]).all()


@pytest.mark.parametrize("n,k", [(263, 6), (5000, 100)])
def test_nan_query(cuda, n, k):
    from annvedi_b200.linear import LinearIndex
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, 110)).astype(np.float32)
    q = rng.standard_normal((2, 110)).astype(np.float32)
    q[1, 55] = np.nan
    ix = LinearIndex(device=0, mode="reference")
    ix.fit(x)
    ids, v = ix.search(q, k)
    np.testing.assert_array_equal(ids[1], np.arange(k))
    assert np.isnan(v[1]).all() and not np.isnan(v[0]).any()
