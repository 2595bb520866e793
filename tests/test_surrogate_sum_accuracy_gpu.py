"""The loss's and the scores' sums are as exact as FP64 sums, bias included, against exact integer arithmetic."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from modlefork_gb300 import surrogate_ops as ops  # noqa: E402

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _exact(x):
    """Sum of an int64 array of values below 2^54 in size, as a Python integer."""
    pad = np.concatenate([x, np.zeros(-x.size % 256, dtype=np.int64)])
    return sum(pad.reshape(-1, 256).sum(axis=1).tolist())


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


def _maps(n, maps, seed):
    """Float maps in [1, 16), whole multiples of 2^-23, and means that leave no deviation exact in a float."""
    rng = np.random.default_rng(seed)
    ref = np.clip(np.exp(rng.normal(1.2, 0.5, (maps, n))), 1.0, 15.5).astype(np.float32)
    pred = np.clip(ref + 0.1 * rng.standard_normal(ref.shape), 1.0, 15.5).astype(np.float32)
    return pred, ref, np.array([1.3700001, 1.7300003], dtype=np.float32)


@pytest.mark.parametrize("n,maps", [(2_400_000, 16), (700_001, 16)])
def test_map_sums_are_unbiased(n, maps):
    """Sums about float means.  The blocks' FP64 sums meet in some 40 additions in any order, a random walk of
    about 2e-16 per map; what each element loses must not add up: 1.5e-15 for one map, 2e-16 for the mean of 16
    (dropping the squares of the deviations' low parts lost 4e-16 to 7e-16 of every map)."""
    pred, ref, mean = _maps(n, maps, n)
    out = torch.zeros(maps, 6, dtype=torch.float64, device=DEV)
    ops.map_sums(torch.from_numpy(pred).to(DEV), torch.from_numpy(ref).to(DEV), n, maps, out,
                 means=torch.from_numpy(np.tile(mean.astype(np.float64), (maps, 1))).to(DEV))
    got = out.cpu().numpy()
    unit = 2.0 ** 23
    mp, mr = (int(float(m) * unit) for m in mean)
    err = np.zeros((maps, 6))
    for k in range(maps):
        p, r = ((x[k].astype(np.float64) * unit).astype(np.int64) for x in (pred, ref))
        a, b, d = p - mp, r - mr, p - r
        for j, v in enumerate((a, b, a * a, b * b, a * b, d * d)):
            want, scale = _exact(v), unit if j < 2 else unit * unit
            err[k, j] = (int(got[k, j] * scale * 2 ** 20) - (want << 20)) / (want << 20)
    assert np.abs(err).max() <= 1.5e-15, np.abs(err).max(axis=0)
    assert np.abs(err.mean(axis=0)).max() <= 2e-16, err.mean(axis=0)


def test_scores_of_whole_maps():
    """Pearson r and relative L2 of 4000 x 600 maps against exact sums: 2e-15 (FP64 sums: up to 1e-15)."""
    from fractions import Fraction as F

    n, maps = 2_400_000, 8
    pred, ref, _ = _maps(n, maps, 5)
    r, l2 = ops.map_scores(torch.from_numpy(pred).to(DEV), torch.from_numpy(ref).to(DEV), n, maps)
    for k in range(maps):
        p, q = ((x[k].astype(np.float64) * 2.0 ** 23).astype(np.int64) for x in (pred, ref))
        sp, sq = _exact(p), _exact(q)
        spp, sqq, spq, sdd = _exact(p * p), _exact(q * q), _exact(p * q), _exact((p - q) ** 2)
        cov, vp, vq = F(spq) - F(sp * sq, n), F(spp) - F(sp * sp, n), F(sqq) - F(sq * sq, n)
        # r^2 and l2^2 are ratios of integers: compare the squares, whose relative error is twice as large
        assert abs(F(float(r[k])) ** 2 / (cov * cov / (vp * vq)) - 1) <= 4e-15
        assert abs(F(float(l2[k])) ** 2 / F(sdd, sqq) - 1) <= 4e-15


@pytest.mark.parametrize("mean", [1e39, -3e300, np.inf, -np.inf, np.nan, 2.0 ** 60])
@pytest.mark.parametrize("n", [5000, 40_001])
def test_map_sums_about_means_beyond_floats(n, mean):
    """Deviations from means that no float holds, as FP64 numpy gives them (1e-13 of each sum, infinities and NaN
    as they come); threads without elements add nothing."""
    rng = np.random.default_rng(n)
    p, r = (rng.random(n).astype(np.float32) for _ in range(2))
    out = torch.zeros(1, 6, dtype=torch.float64, device=DEV)
    ops.map_sums(torch.from_numpy(p).to(DEV), torch.from_numpy(r).to(DEV), n, 1, out,
                 means=torch.tensor([[mean, 0.5]], dtype=torch.float64, device=DEV))
    with np.errstate(all="ignore"):
        a, b, d = p.astype(np.float64) - mean, r.astype(np.float64) - 0.5, p.astype(np.float64) - r
        want = np.array([a.sum(), b.sum(), (a * a).sum(), (b * b).sum(), (a * b).sum(), (d * d).sum()])
        size = np.array([np.abs(x).sum() for x in (a, b, a * a, b * b, a * b, d * d)])
    got = out.cpu().numpy()[0]
    for k in range(6):
        if np.isfinite(size[k]):
            assert abs(got[k] - want[k]) <= 1e-13 * size[k], (k, got[k], want[k])
        else:
            assert got[k] == want[k] or (np.isnan(got[k]) and np.isnan(want[k])), (k, got[k], want[k])


@pytest.mark.parametrize("B,L,cin,cout,taps,splits", [(64, 1000, 256, 256, 3, (76, 38)), (64, 4000, 64, 64, 3, (304, 152)),
                                                      (64, 2000, 128, 128, 1, (304, 152))])
def test_weight_gradient_accumulation_length(B, L, cin, cout, taps, splits):
    """The automatic split adds its accumulations to dw often enough: its error (norm against FP64) is that of as many
    splits as give each accumulation two waves' share of the positions (76, 304), not that of one wave of splits with a
    single accumulation each (38, 152), which is about twice as large."""
    g = torch.Generator(device=DEV).manual_seed(B + L)
    x = torch.nn.functional.silu(torch.randn(B, L, cin, generator=g, device=DEV)).to(torch.bfloat16)
    dz = (torch.randn(B, L, cout, generator=g, device=DEV) * 1e-2).to(torch.bfloat16)
    pad = (taps - 1) // 2
    xp = torch.zeros(B, L + 2 * pad, cin, dtype=torch.float64, device=DEV)
    xp[:, pad:pad + L] = x.double()
    zd = dz.double().reshape(B * L, cout)
    want = torch.stack([zd.T @ xp[:, t:t + L].reshape(B * L, cin) for t in range(taps)], dim=1)

    def error(k):
        dw = torch.zeros(cout, taps, cin, device=DEV)
        ops.conv_wgrad(x, dz, dw, splits=k)
        return float((dw.double() - want).norm() / want.norm())

    auto, short, long = error(0), error(splits[0]), error(splits[1])
    assert auto <= 1.15 * short and auto <= 0.85 * long, (auto, short, long)
