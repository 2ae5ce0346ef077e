"""The restated LSH projections against those recorded from the reference's own fit, and their orthonormality."""
import os

import numpy as np
import pytest

from oracle import refmod
from tests.golden import make_golden as mg


def test_restatement_equals_the_recorded(golden_dir):
    with np.load(os.path.join(golden_dir, "ivf_ref.npz")) as fx:
        want = fx["lsh_8k_64_t3b4/projections"]
    got = refmod.lsh_projections(3, 4, want.shape[1])
    # FP32 sums of 64 terms of unit rows, four deep: 64 * 4 * 2^-24 of the largest component at most
    np.testing.assert_allclose(got, want, atol=64 * 4 * 2.0 ** -24)


@pytest.mark.parametrize("t,b,d", [(3, 6, 64), (1, 8, 64), (2, 5, 33), (1, 9, 4)])
def test_shapes(t, b, d):
    p = mg.projections_from_reference(t, b, d)
    assert p.shape == (t * b, d) and p.dtype == np.float32
    if b <= d:
        for i in range(t):
            rows = p[i * b:(i + 1) * b].astype(np.float64)
            np.testing.assert_allclose(rows @ rows.T, np.eye(b), atol=1e-6)
