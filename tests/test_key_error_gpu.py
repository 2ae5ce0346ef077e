"""What the certified windows take for granted, measured: the BF16 keys of the tensor cores against 64-bit sums.

The accumulation of the operands' dim + 3 products loses at most 2^-21 of their absolute sum each (half of the allowance's slack is
left out here), and a key is within half the window of |x|^2 - 2 x.q (or -x.q) of the FP32 vectors (key_window_l2 / _ip)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bf16(a):
    import torch
    return torch.from_numpy(a).to(torch.bfloat16).to(torch.float64).numpy()


@pytest.mark.parametrize("metric", ["l2", "ip"])
@pytest.mark.parametrize("kind,scale", [("normal", 1.0), ("normal", 1e9), ("normal", 1e-9), ("offset", 1.0), ("spread", 1.0)])
@pytest.mark.parametrize("dim", [5, 64, 100, 384, 1536, 4096])
def test_keys(cuda, metric, kind, scale, dim):
    import torch
    from annvedi_b200.linear import LinearIndex
    rng = np.random.default_rng(dim)
    x, q = rng.standard_normal((1500, dim)), rng.standard_normal((40, dim))
    if kind == "offset":
        x, q = x + 20, q + 20
    if kind == "spread":  # terms of very different size
        f = 10.0 ** rng.uniform(-4, 4, dim)
        x, q = x * f, q / f
    x, q = (scale * x).astype(np.float32), (scale * q).astype(np.float32)
    ix = LinearIndex(device=0, metric=metric, mode="exact")
    ix.fit(torch.from_numpy(x).cuda())
    keys = ix.scores_tc(torch.from_numpy(q).cuda()).cpu().numpy().astype(np.float64)
    x64, q64 = x.astype(np.float64), q.astype(np.float64)
    xb, qb = _bf16(x), _bf16(q)
    f = 2.0 if metric == "l2" else 1.0
    dots, absdots = f * qb @ xb.T, f * np.abs(qb) @ np.abs(xb).T
    sq = (x64 ** 2).sum(1)
    if metric == "l2":
        # the operands' norm: an FP32 sum of FP32 squares (dim 2^-24 of it at most) in three BF16 pieces (2^-24 of it left)
        err = np.abs(keys - (sq - dots))
        assert (err <= (dim + 3) * 2.0 ** -21 * (absdots + sq) + (dim + 2) * 2.0 ** -24 * sq).all()
    else:
        err = np.abs(keys + dots)
        assert (err <= dim * 2.0 ** -21 * absdots).all()
    cm, rm = np.sqrt(sq.max()), np.sqrt(((x64 - xb) ** 2).sum(1).max())
    qn, rq = np.sqrt((q64 ** 2).sum(1)), np.sqrt(((q64 - qb) ** 2).sum(1))
    acc = (dim + 19) * 2.0 ** -21
    cross = rm * qn + (cm + rm) * rq
    eps = 2 * cross + acc * (2 * (cm + rm) * (qn + rq) + cm * cm) if metric == "l2" else cross + acc * (cm + rm) * (qn + rq)
    real = sq - 2 * q64 @ x64.T if metric == "l2" else -(q64 @ x64.T)
    assert (np.abs(keys - real) <= eps[:, None]).all()
