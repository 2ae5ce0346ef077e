"""The pruned exact scan at the smallest bases that take it: ids and distances of the plain scan, bit for bit (the plain
scan as in test_pruned_exact_gpu)."""
import numpy as np
import pytest

from tests.test_pruned_exact_gpu import _check, _data

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("metric", ["l2", "ip"])
@pytest.mark.parametrize("n,dim,nq,k,kind", [
    (4095, 24, 5, 10, "normal"), (4096, 24, 5, 64, "normal"), (4097, 100, 33, 1, "ties"), (4352, 384, 64, 64, "clusters"),
    (8191, 48, 3, 10, "normal"), (8192, 48, 2, 100, "normal"), (8193, 48, 4, 128, "clusters"), (11999, 96, 1, 10, "normal"),
    (12000, 96, 1, 10, "ties"), (8192, 96, 1, 64, "offset"), (6000, 64, 700, 20, "offset"), (30000, 33, 300, 400, "normal"),
])
def test_pruned_equals_plain(cuda, metric, n, dim, nq, k, kind):
    x, q = _data(kind, n, dim, nq, np.random.default_rng(n + nq))
    _check(x, q, k, metric)
