"""The reference ranking over the dimensions at which the partials kernel's row pieces change, and over the batch sizes at which
the rows are one segment: ids and values of the restatement, bit for bit."""
import numpy as np
import pytest

from oracle import refmod

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [1, 7, 15, 16, 17, 32, 33, 48, 64, 65, 100, 128, 129, 256, 257, 384, 385, 400, 512, 513])
def test_dimensions(cuda, dim):
    from annvedi_b200.linear import LinearIndex
    rng = np.random.default_rng(dim)
    x = rng.standard_normal((2500, dim)).astype(np.float32)
    q = rng.standard_normal((5, dim)).astype(np.float32)
    ix = LinearIndex(device=0, mode="reference")
    ix.fit(x)
    ids, v = ix.search(q, 70)
    wi, wv = refmod.linear_query(x, q, 70, lanes=16)
    np.testing.assert_array_equal(ids, wi)
    np.testing.assert_array_equal(v, wv)


@pytest.mark.parametrize("n,nq,k", [(10240, 256, 9), (10241, 256, 9), (10240, 255, 9), (1030, 300, 512), (64, 257, 64), (5000, 256, 200)])
def test_one_segment(cuda, n, nq, k):
    from annvedi_b200.linear import LinearIndex
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, 20)).astype(np.float32)
    q = rng.standard_normal((nq, 20)).astype(np.float32)
    ix = LinearIndex(device=0, mode="reference")
    ix.fit(x)
    ids, v = ix.search(q, k)
    pick = np.r_[0:6, nq - 6:nq]
    wi, wv = refmod.linear_query(x, np.ascontiguousarray(q[pick]), k, lanes=16)
    np.testing.assert_array_equal(ids[pick], wi)
    np.testing.assert_array_equal(v[pick], wv)
