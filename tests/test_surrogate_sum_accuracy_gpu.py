"""The loss's sums are as exact as FP64 sums, bias included, against exact integer arithmetic."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from modlefork_gb300 import surrogate_ops as ops  # noqa: E402

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def test_loss_of_one_thread():
    """Sixteen groups of four values a whole grid apart (1216 blocks of 256 threads) meet in one thread and all others are
    zero, so nothing but that thread's sum rounds: two additions in FP64 and what the floats lose, allowed
    eight units of 2^-53.  (FP64 squares added one by one may lose 64; pairs of floats with a single low part lost
    up to 300.)"""
    step, chunk = 1216 * 256, 16
    pred = torch.zeros(chunk * step // 64, 256, device=DEV)
    target = torch.zeros_like(pred)
    groups = pred.view(chunk, step, 4)
    rng = np.random.default_rng(1)
    for j in rng.integers(0, step, 40):
        v = rng.standard_normal((chunk, 4)).astype(np.float32)
        groups[:, j] = torch.from_numpy(v).to(DEV)
        loss = torch.zeros(1, dtype=torch.float64, device=DEV)
        ops.mse(pred, target, loss)
        groups[:, j] = 0
        q = [int(x) for x in (np.abs(v).astype(np.float64) * 2.0 ** 50).ravel()]  # whole: |v| >= 2^-26 here
        assert all(float(x) == float(y) * 2.0 ** 50 for x, y in zip(q, np.abs(v).ravel()))
        want = sum(x * x for x in q)
        got = int(loss.item() * 2.0 ** 60) << 40
        assert abs(got - want) * 2 ** 50 <= want, abs(got - want) / want  # 8 * 2^-53
