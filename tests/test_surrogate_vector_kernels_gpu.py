"""The vectorised forms of the surrogate's memory-bound kernels at the sizes and alignments where they change
path, against FP64 numpy: sums in float pairs (scores, loss), the bias gradient, Adam, the list of weight
transposes and the weight gradient's bulk reductions."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from modlefork_gb300 import surrogate_ops as ops  # noqa: E402

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _sums64(p, r, mp, mr):
    a, b = p.astype(np.float64) - mp, r.astype(np.float64) - mr
    d = p.astype(np.float64) - r
    return np.array([a.sum(), b.sum(), (a * a).sum(), (b * b).sum(), (a * b).sum(), (d * d).sum()])


@pytest.mark.parametrize("scale", [1.0, 1e-12, 1e12])
@pytest.mark.parametrize("n,off", [(1, 0), (3, 0), (4, 0), (1023, 0), (16384, 0), (16388, 1), (16384 * 5 + 7, 0),
                                   (60_000, 2)])
def test_map_sums(n, off, scale):
    """FP64-like accuracy (1e-13 of the sum of magnitudes) inside and outside the float pairs' range, aligned and
    not, with and without means."""
    rng = np.random.default_rng(n)
    nm = 3
    p = (rng.random((nm, n + off)) * scale).astype(np.float32)
    r = (p + 0.1 * scale * rng.standard_normal(p.shape)).astype(np.float32)
    p[1, off:] = 0.0  # a map of zeros
    tp, tr = (torch.from_numpy(x).to(DEV) for x in (p, r))
    means = np.stack([p[:, off:].mean(1), r[:, off:].mean(1)], axis=1).astype(np.float64)
    for mm in (None, means):
        out = torch.zeros(nm, 6, dtype=torch.float64, device=DEV)
        ops.map_sums(tp.view(-1)[off:], tr.view(-1)[off:], n, nm, out, n + off, n + off,
                     means=None if mm is None else torch.from_numpy(mm).to(DEV))
        got = out.cpu().numpy()
        for m in range(nm):
            mp, mr = (0.0, 0.0) if mm is None else mm[m]
            want = _sums64(p[m, off:], r[m, off:], mp, mr)
            a, b = np.abs(p[m, off:].astype(np.float64) - mp), np.abs(r[m, off:].astype(np.float64) - mr)
            size = np.array([a.sum() + n * abs(mp) * 1e-3, b.sum() + n * abs(mr) * 1e-3, (a * a).sum(), (b * b).sum(),
                             (a * b).sum(), want[5]])
            assert np.all(np.abs(got[m] - want) <= 1e-13 * size + 1e-300), (m, got[m], want)


def test_map_sums_keep_infinities_and_nan():
    p = torch.ones(2, 5000, device=DEV)
    r = torch.ones(2, 5000, device=DEV) * 2
    p[0, 77], p[1, 4999] = float("inf"), float("nan")
    out = torch.zeros(2, 6, dtype=torch.float64, device=DEV)
    ops.map_sums(p, r, 5000, 2, out)
    got = out.cpu().numpy()
    assert got[0, 0] == np.inf and got[0, 2] == np.inf and got[0, 5] == np.inf and got[0, 1] == 10000.0
    assert np.isnan(got[1, 0]) and np.isnan(got[1, 4]) and got[1, 3] == 20000.0


@pytest.mark.parametrize("rows,n_valid,dstride", [(1, 4, 4), (50, 600, 640), (333, 36, 64), (50, 601, 640), (7, 5, 9)])
def test_mse(rows, n_valid, dstride):
    rng = np.random.default_rng(rows)
    pred = rng.standard_normal((rows, n_valid)).astype(np.float32)
    tgt = rng.standard_normal((rows, n_valid)).astype(np.float32)
    loss = torch.zeros(1, dtype=torch.float64, device=DEV)
    dp = torch.full((rows, dstride), 9.0, dtype=torch.bfloat16, device=DEV)
    ops.mse(torch.from_numpy(pred).to(DEV), torch.from_numpy(tgt).to(DEV), loss, dp=dp, scale=0.5)
    d = (pred - tgt).astype(np.float64)
    assert abs(loss.item() - (d * d).sum()) <= 1e-13 * (d * d).sum()
    want = torch.from_numpy((0.5 * (pred - tgt)).astype(np.float32)).to(torch.bfloat16)
    assert torch.equal(dp[:, :n_valid].cpu(), want) and not dp[:, n_valid:].any()


@pytest.mark.parametrize("rows,C,stride", [(1, 8, 8), (31, 64, 64), (129, 72, 80), (4001, 640, 640), (515, 200, 640),
                                           (100, 30, 30)])
def test_bias_grad(rows, C, stride):
    rng = np.random.default_rng(rows + C)
    dz = torch.from_numpy(rng.standard_normal((rows, stride)).astype(np.float32)).to(torch.bfloat16)
    db = torch.ones(C, device=DEV)
    ops.bias_grad(dz.to(DEV), db, n_valid=C)
    x = dz.float().numpy().astype(np.float64)[:, :C]
    assert np.all(np.abs(db.cpu().numpy() - 1 - x.sum(0)) <= 2e-6 * (1 + np.abs(x).sum(0)))


@pytest.mark.parametrize("n", [4, 1000, 1003])
def test_adam_forms_agree(n):
    """Aligned and offset buffers take different kernels with the same arithmetic."""
    rng = np.random.default_rng(n)
    cols = [torch.from_numpy(np.abs(rng.standard_normal(n + 4)).astype(np.float32)).to(DEV) for _ in range(4)]
    res = []
    for off in (0, 1):
        p, g, m, v = (torch.zeros(n + 8, device=DEV)[off:off + n].copy_(c[:n]) for c in cols)
        pb = torch.zeros(n + 8, dtype=torch.bfloat16, device=DEV)[off:off + n]
        ops.adam(p, g, m, v, 3, 1e-3, wd=0.01, gscale=0.5, p_bf16=pb)
        res.append([t.cpu() for t in (p, m, v, pb)])
    for a, b in zip(*res):
        assert torch.equal(a, b)


def test_transpose_list():
    rng = np.random.default_rng(3)
    shapes = [(64, 3, 64), (640, 1, 64), (128, 3, 200), (72, 5, 8), (512, 3, 1024)]
    ws = [torch.from_numpy(rng.standard_normal(s).astype(np.float32)).to(torch.bfloat16).to(DEV) for s in shapes]
    wts = [torch.zeros(s[2], s[1], s[0], dtype=torch.bfloat16, device=DEV) for s in shapes]
    ops.TransposeList(zip(ws, wts)).run()
    for w, wt in zip(ws, wts):
        assert torch.equal(wt, w.flip(1).permute(2, 1, 0))


@pytest.mark.parametrize("B,L,Cin,Cout,taps,off", [(1, 5, 8, 8, 3, 0), (2, 70, 136, 200, 3, 0), (3, 129, 64, 128, 3, 0),
                                                   (2, 100, 72, 264, 1, 0), (2, 70, 136, 200, 3, 1),
                                                   (16, 125, 512, 512, 3, 0)])
def test_wgrad_reductions(B, L, Cin, Cout, taps, off):
    """dw 16-byte aligned (bulk reductions) and not (word by word), ragged channel tiles."""
    rng = np.random.default_rng(Cin + Cout)
    x = torch.from_numpy(rng.standard_normal((B, L, Cin)).astype(np.float32)).to(torch.bfloat16).to(DEV)
    dz = torch.from_numpy(rng.standard_normal((B, L, Cout)).astype(np.float32)).to(torch.bfloat16).to(DEV)
    buf = torch.ones(Cout * taps * Cin + 8, device=DEV)
    dw = buf[off:off + Cout * taps * Cin].view(Cout, taps, Cin)
    ops.conv_wgrad(x, dz, dw)
    xd, zd = x.double(), dz.double()
    pad = (taps - 1) // 2
    xp = torch.nn.functional.pad(xd, (0, 0, pad, pad))
    want = torch.stack([torch.einsum("bln,blc->nc", zd, xp[:, t:t + L]) for t in range(taps)], dim=1)
    assert (dw.double() - 1 - want).abs().max() <= 2e-5 * want.abs().max()
    assert torch.all(buf[:off] == 1) and torch.all(buf[off + dw.numel():] == 1)
    assert ops.take_error() == 0
