"""The k-means assignment from tensor-core keys and the update by ThreadPool chunks, bit for bit against the CPU
restatement of the reference's k-means (oracle/restate_kmeans.cpp)."""
import numpy as np
import pytest

from oracle import refmod

pytestmark = pytest.mark.gpu


def _rows(kind, n, dim, seed):
    rng = np.random.default_rng(seed)
    if kind == "clusters":  # fewer clusters than lists: lists split clusters, several centroids in a row's window
        c = rng.standard_normal((9, dim))
        x = c[rng.integers(0, 9, n)] + 0.2 * rng.standard_normal((n, dim))
    elif kind == "offset":  # the keys' error covers every centroid
        x = 30.0 + 0.01 * rng.standard_normal((n, dim))
    elif kind == "huge":    # norms the keys' bound does not cover: the FP32 scan assigns
        x = 1e16 * rng.standard_normal((n, dim))
    else:
        x = rng.standard_normal((n, dim))
    x = x.astype(np.float32)
    if kind == "zeros":
        x[5:25] = 0.0
    return x


@pytest.mark.parametrize("kind,n,dim,c,threads", [
    ("normal", 4001, 13, 33, 1), ("normal", 3000, 100, 64, 40), ("clusters", 6000, 48, 47, 16),
    ("clusters", 2500, 520, 70, 5), ("offset", 2500, 24, 31, 3), ("zeros", 3000, 16, 40, 17), ("huge", 2500, 16, 32, 4),
    ("normal", 2100, 8, 2048, 2),
])
def test_fit_equals_the_restatement(cuda, kind, n, dim, c, threads):
    from annvedi_b200.ivf import IVFIndex
    x = _rows(kind, n, dim, n + dim)
    cent, assign = refmod.kmeans(x, c, threads)
    ix = IVFIndex(device=0, num_threads=threads)
    ix.fit(x, 1, 0, c)
    st = ix.export_state()
    np.testing.assert_array_equal(st["centroids"], cent)
    np.testing.assert_array_equal(st["reordered_to_original"], np.argsort(assign, kind="stable"))
