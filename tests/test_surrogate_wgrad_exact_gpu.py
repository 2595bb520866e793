"""Weight gradients (and, per case, bias gradients) of small whole numbers: every product and every partial sum is a
whole number below 2^24, exact in FP32 in any order, so the results must equal the FP64 sums exactly.  A row lost or
read twice, or a column that a diverged warp gave another value, shows at once.  Run several times each."""

import pytest

torch = pytest.importorskip("torch")

from modlefork_gb300 import surrogate_ops as ops  # noqa: E402

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _inputs(B, L, cin, cout, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    x = torch.randint(-2, 3, (B, L, cin), generator=g, device=DEV).to(torch.bfloat16)
    dz = torch.randint(-2, 3, (B, L, cout), generator=g, device=DEV).to(torch.bfloat16)
    return x, dz


def _want(x, dz, taps):
    B, L, cin = x.shape
    pad = (taps - 1) // 2
    xp = torch.zeros(B, L + 2 * pad, cin, dtype=torch.float64, device=DEV)
    xp[:, pad:pad + L] = x.double()
    zd = dz.double().reshape(B * L, -1)
    return torch.stack([zd.T @ xp[:, t:t + L].reshape(B * L, cin) for t in range(taps)], dim=1), zd.sum(0)


# output channels that end inside a warp's 32 rows, with one and several accumulations per split, both input-tile
# widths, bulk reductions and (off = 1) word by word
@pytest.mark.parametrize("B,L,cin,cout,taps,off", [(16, 999, 136, 136, 3, 0), (16, 999, 72, 8, 3, 0),
                                                   (16, 2000, 64, 200, 3, 0), (40, 500, 128, 600, 1, 0),
                                                   (16, 999, 136, 136, 3, 1), (1, 65, 264, 40, 3, 0)])
def test_ragged_output_channels(B, L, cin, cout, taps, off):
    x, dz = _inputs(B, L, cin, cout, B + cout)
    want, _ = _want(x, dz, taps)
    for _ in range(5):
        buf = torch.ones(cout * taps * cin + 8, device=DEV)
        dw = buf[off:off + cout * taps * cin].view(cout, taps, cin)
        ops.conv_wgrad(x, dz, dw)
        assert torch.equal(dw.double() - 1, want)
        assert torch.all(buf[:off] == 1) and torch.all(buf[off + dw.numel():] == 1)
    assert ops.take_error() == 0


@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("L", [1, 33, 127, 130, 161])
def test_unstaged_epilogue_at_ragged_lengths(L, form):
    """Rows past the end leave their warp's stores out; the next columns' accumulators are right all the same."""
    B, cin, cout = 3, 64, 256
    x, w = _inputs(B, L, cin, cout, L)[0], _inputs(1, cout * 3, cin, 8, 5)[0].view(cout, 3, cin)
    out = torch.full((B, L, cout), 7.0, device=DEV)
    saved = ops.conv_get_form(256)
    ops.conv_set_form(256, form)
    try:
        ops.conv_forward(x, w, out_f32=out)
    finally:
        ops.conv_set_form(256, saved)
    xp = torch.zeros(B, L + 2, cin, dtype=torch.float64, device=DEV)
    xp[:, 1:1 + L] = x.double()
    want = sum(xp[:, t:t + L] @ w[:, t].double().T for t in range(3))
    assert torch.equal(out.double(), want)
    assert ops.take_error() == 0


# the bias gradient's warps read the stages of a long ring while copies refill it: many blocks per split at full-rate
# copies, the head's five output tiles, one tap and three, ragged channels, lengths that end inside a block
@pytest.mark.parametrize("B,L,cin,cout,taps", [(64, 1000, 256, 256, 3), (32, 4000, 64, 640, 1), (64, 4000, 64, 64, 3),
                                               (32, 2000, 384, 128, 3), (16, 999, 72, 136, 3), (256, 125, 512, 512, 3),
                                               (300, 65, 8, 8, 1)])
def test_bias_gradient_of_the_weight_gradient(B, L, cin, cout, taps):
    x, dz = _inputs(B, L, cin, cout, L + cout)
    want, wantb = _want(x, dz, taps)
    for k in range(20):
        dw, db = torch.zeros(cout, taps, cin, device=DEV), torch.ones(cout, device=DEV)
        ops.run((ops.Op * 1)(ops.op(ops.OP_WGRAD, (x, dz, dw, db), (B, L, cin, cout, taps, 0))))
        assert torch.equal(db.double() - 1, wantb), k
        assert torch.equal(dw.double(), want), k
    assert ops.take_error() == 0
