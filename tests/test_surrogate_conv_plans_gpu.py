"""The persistent convolution's ways of using shared memory, lists of operations, and selections of map sums.

The persistent kernel adds the same products in the same order as the one-tile-per-CTA kernel (which is compared with
FP64 elsewhere), whatever stays in shared memory, so the two must agree bit for bit.  The shapes reach every
plan (weights and activation slots resident, slots with a weight ring, both operands by stage, one tap, more taps than
slots hold), every tile width (64, 128, 192, 256) and its narrowing, more than one tile per CTA, ragged last tiles."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from modlefork_gb300 import surrogate_ops as ops  # noqa: E402

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

SHAPES = [  # (B, L, Cin, Cout, taps)
    (1400, 130, 64, 64, 3),    # weights stay, one chunk
    (700, 130, 128, 128, 3),   # weights stay, two chunks
    (500, 131, 192, 64, 3),    # weights stay, three chunks
    (400, 130, 64, 384, 3),    # weights stay, two N tiles of 192
    (300, 257, 384, 128, 3),   # slots and a weight ring
    (200, 260, 256, 256, 3),
    (200, 257, 384, 384, 3),
    (100, 130, 640, 256, 3),   # both operands by stage
    (150, 130, 896, 384, 3),
    (400, 129, 64, 640, 1),    # one tap
    (400, 129, 128, 128, 9),   # as many taps as slots hold
    (300, 129, 64, 64, 11),    # more
    (1, 125, 512, 512, 3),     # narrowed tiles
    (1, 4000, 64, 64, 3),
    (2, 999, 256, 384, 3),
]


@pytest.fixture(autouse=True)
def _no_timeouts():
    torch.cuda.synchronize()
    yield
    torch.cuda.synchronize()
    assert ops.take_error() == 0, "a tensor-core kernel's barrier wait ran out"


def _inputs(B, L, cin, cout, taps):
    g = torch.Generator(device=DEV).manual_seed(B + L + cin + cout)
    x = torch.randn(B, L, cin, generator=g, device=DEV).to(torch.bfloat16)
    w = (torch.randn(cout, taps, cin, generator=g, device=DEV) * (1.0 / (taps * cin)) ** 0.5).to(torch.bfloat16)
    b = torch.randn(cout, generator=g, device=DEV)
    z = torch.randn(B, L, cout, generator=g, device=DEV).to(torch.bfloat16)
    return x, w, b, z


def _run(form, B, L, cout, fn):
    saved = {bn: ops.conv_get_form(bn) for bn in (64, 128, 256)}
    for bn in saved:
        ops.conv_set_form(bn, form)
    try:
        return fn()
    finally:
        for bn, f in saved.items():
            ops.conv_set_form(bn, f)


@pytest.mark.parametrize("B,L,cin,cout,taps", SHAPES)
def test_persistent_equals_tile_kernel(B, L, cin, cout, taps):
    x, w, b, z = _inputs(B, L, cin, cout, taps)
    nv = 600 if cout == 640 else cout  # the head: 600 of 640 channels

    def both():
        post, pre = (torch.full((B, L, nv), 7.0, dtype=torch.bfloat16, device=DEV) for _ in range(2))
        ops.conv_forward(x, w, b, act=ops.ACT_SILU, out_pre=pre, out_post=post, n_valid=nv)
        return pre, post

    def f32():
        out = torch.full((B, L, nv), 7.0, device=DEV)
        ops.conv_forward(x, w, b, out_f32=out, n_valid=nv)
        return (out,)

    def gated():
        out = torch.full((B, L, nv), 7.0, dtype=torch.bfloat16, device=DEV)
        ops.conv_forward(x, w, None, out_post=out, n_valid=nv, gate=z[:, :, :nv].contiguous())
        return (out,)

    for fn in (both, f32, gated):
        want = _run(0, B, L, cout, fn)
        for form in (1, 2, 3):
            for a, c in zip(_run(form, B, L, cout, fn), want):
                assert torch.equal(a, c), (fn.__name__, form, (a != c).sum().item())


@pytest.mark.parametrize("B,L,cin,cout,taps", [s for s in SHAPES if s[1] % 2 == 0 and s[3] != 640])
def test_persistent_fused_copies(B, L, cin, cout, taps):
    x, w, b, _ = _inputs(B, L, cin, cout, taps)

    def fused():
        cat = torch.zeros(B, L, cout + 64, dtype=torch.bfloat16, device=DEV)
        up = torch.zeros(B, 2 * L, cout + 64, dtype=torch.bfloat16, device=DEV)
        pool = torch.zeros(B, L // 2, cout, dtype=torch.bfloat16, device=DEV)
        ops.conv_forward_fused(x, w, b, act=ops.ACT_SILU, skip=cat[:, :, 64:], dup=up[:, :, :cout], pool=pool)
        return cat, up, pool

    def plain():
        post = torch.empty(B, L, cout, dtype=torch.bfloat16, device=DEV)
        ops.conv_forward(x, w, b, act=ops.ACT_SILU, out_post=post)
        pool = torch.empty(B, L // 2, cout, dtype=torch.bfloat16, device=DEV)
        ops.pool2(post, pool)
        return post, pool

    post, pool = _run(2, B, L, cout, plain)
    for form in (2, 3):
        cat, up, p = _run(form, B, L, cout, fused)
        assert torch.equal(cat[:, :, 64:], post) and not cat[:, :, :64].any()
        assert torch.equal(up[:, 0::2, :cout], post) and torch.equal(up[:, 1::2, :cout], post) and not up[:, :, cout:].any()
        assert torch.equal(p, pool)


def test_list_of_operations_equals_them_one_by_one():
    """A chain in which every operation reads what the one before it wrote, run as one list without a wait and one
    operation at a time; and an unknown kind is refused."""
    B, L, C = 40, 500, 64
    x, w, b, z = _inputs(B, L, C, C, 3)

    def chain(run):
        bf = lambda *s: torch.zeros(*s, dtype=torch.bfloat16, device=DEV)  # noqa: E731
        pre, post, pool, post2 = bf(B, L, C), bf(B, L, C), bf(B, L // 2, C), bf(B, L // 2, C)
        cat, dcat, dz, dw = bf(B, L, 2 * C), bf(B, L, 2 * C), bf(B, L // 2, C), torch.zeros(C, 3, C, device=DEV)
        db = torch.zeros(C, device=DEV)
        w2 = torch.cat([w, w], 0).contiguous()
        lst = [ops.conv_op(x, w, bias=b, act=ops.ACT_SILU, pre=pre, post=post),
               ops.op(ops.OP_POOL2, (post, pool), (B, L // 2, C)),
               ops.conv_op(pool, w, bias=b, act=ops.ACT_SILU, post=post2),
               ops.op(ops.OP_UPCAT, (post2, post, cat), (B, L, C, C)),
               ops.conv_op(post, w2, post=dcat),
               ops.op(ops.OP_UPCAT_BWD, (dcat, post2, dz), (B, L // 2, C, 2 * C)),
               ops.op(ops.OP_WGRAD, (pool, dz, dw, db), (B, L // 2, C, C, 3, 1))]
        run(lst)
        torch.cuda.synchronize()
        return pre, post, pool, post2, cat, dcat, dz, dw, db

    def one_by_one(lst):
        for o in lst:
            ops.run((ops.Op * 1)(o))
            torch.cuda.synchronize()

    want = chain(one_by_one)
    got = chain(lambda lst: ops.run((ops.Op * len(lst))(*lst)))
    for k, (a, c) in enumerate(zip(got, want)):
        assert torch.equal(a, c), k
    bad = ops.op(99, (x,), (B,))
    with pytest.raises(ops.SurrogateKernelError):
        ops.run((ops.Op * 1)(bad))


def test_selected_map_sums():
    rng = np.random.default_rng(3)
    p, r = (torch.from_numpy(rng.random((3, 40_001), dtype=np.float32)).to(DEV) for _ in range(2))
    means = torch.rand(3, 2, dtype=torch.float64, device=DEV)
    for which, mm in ((ops.SUMS_RAW, None), (ops.SUMS_CENTRED, means)):
        full, part = (torch.zeros(3, 6, dtype=torch.float64, device=DEV) for _ in range(2))
        ops.map_sums(p, r, 40_001, 3, full, means=mm)
        ops.map_sums(p, r, 40_001, 3, part, means=mm, which=which)
        for k in range(6):
            if which >> k & 1:  # the blocks' sums meet in any order
                assert ((part[:, k] - full[:, k]).abs() <= 1e-13 * 40_001).all(), k
            else:
                assert not part[:, k].any(), k


@pytest.mark.parametrize("B,L,cin,cout,taps", [(16, 999, 256, 256, 3), (3, 130, 64, 64, 3), (5, 64, 128, 600, 1),
                                               (1, 63, 8, 8, 3), (2, 1, 192, 136, 3), (40, 65, 896, 384, 3)])
def test_weight_and_bias_gradient_in_one(B, L, cin, cout, taps):
    """Against FP64: products and sums of BF16 values in FP32, K terms each (error of any order of adding: at most
    (K + 1) 2^-24 of the sum of magnitudes; 16 times its square root covers a random walk many times over), added to
    what was there; rows and columns past the tiles' edges."""
    x, _, _, z = _inputs(B, L, cin, cout, taps)
    dw = torch.ones(cout, taps, cin, device=DEV)
    db = torch.ones(cout, device=DEV)
    o = ops.op(ops.OP_WGRAD, (x, z, dw, db), (B, L, cin, cout, taps, 0))
    ops.run((ops.Op * 1)(o))
    pad = (taps - 1) // 2
    xp = torch.zeros(B, L + 2 * pad, cin, dtype=torch.float64, device=DEV)
    xp[:, pad:pad + L] = x.double()
    zd = z.double()
    tol = 16 * (B * L + 2) ** 0.5 * 2.0 ** -24
    assert ((db - 1 - zd.sum((0, 1))).abs() <= tol * (zd.abs().sum((0, 1)) + 1)).all()
    for t in range(taps):
        xt = xp[:, t:t + L]
        want = torch.einsum("bln,blc->nc", zd, xt)
        size = torch.einsum("bln,blc->nc", zd.abs(), xt.abs()) + 1
        assert ((dw[:, t] - 1 - want).abs() <= tol * size).all()
