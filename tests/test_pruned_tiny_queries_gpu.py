"""Queries whose squares underflow, beside ordinary ones: the exact search gives the plain scan's ids and distances bit for
bit (the plain scan as in test_pruned_exact_gpu)."""
import numpy as np
import pytest

from tests.test_pruned_exact_gpu import _check, _data

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("metric", ["ip", "l2"])
@pytest.mark.parametrize("scale", [1e-11, 1e-13, 1e-18, 1e-23, 1e-25, 1e-30, 1e-36, 0.0])
@pytest.mark.parametrize("n,dim,nq,k", [(50021, 100, 40, 100), (30000, 384, 3, 10)])
def test_tiny_queries(cuda, metric, scale, n, dim, nq, k):
    x, q = _data("normal", n, dim, nq, np.random.default_rng(dim))
    q[nq // 3:] *= np.float32(scale)
    _check(x, q, k, metric)


def test_rows_far_below_the_largest(cuda):
    """Rows of very different norms: the tiny ones' own squares underflow, the window is the largest row's."""
    x, q = _data("normal", 40000, 64, 20, np.random.default_rng(2))
    x[::3] *= np.float32(1e-24)
    x[1::3] = np.round(x[1::3])
    q[::2] *= np.float32(1e-9)
    _check(x, q, 50, "ip")
    _check(x, q, 50, "l2")
