"""Copies and saved objects of a network that has run: their own tensors, the same results, nothing shared."""

import copy
import io

import pytest

torch = pytest.importorskip("torch")

from modlefork_gb300 import surrogate as S  # noqa: E402
from modlefork_gb300 import surrogate_ops as ops  # noqa: E402

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _saved(net):
    buf = io.BytesIO()
    torch.save(net, buf)
    buf.seek(0)
    return torch.load(buf, weights_only=False)


@pytest.mark.parametrize("how", [copy.deepcopy, _saved, copy.copy])
def test_copy_of_a_used_network(how):
    net = S.UNet(widths=(64, 128), mid=128, length=64, seed=4)
    g = torch.Generator(device=DEV).manual_seed(1)
    x = torch.randn(3, 64, S.IN_CH, generator=g, device=DEV).to(torch.bfloat16)
    target = torch.rand(3, 64, S.NROWS, generator=g, device=DEV)
    want = net.forward(x).clone()
    loss = net.loss_and_grad(x, target).clone()
    grad = net.g.clone()
    net.adam_step(0.0)
    other = how(net)
    assert torch.equal(other.forward(x), want)
    assert torch.allclose(other.loss_and_grad(x, target), loss, rtol=1e-12)
    assert (other.g - grad).abs().max() <= 1e-5 * grad.abs().max()  # the splits' sums meet in any order
    other.adam_step(1e-2)
    for name, w in other.wb.items():
        assert torch.equal(other.wt[name], w.flip(1).permute(2, 1, 0)), name
    if how is not copy.copy:
        assert torch.equal(net.forward(x), want) and not torch.equal(other.forward(x), want)
    assert ops.take_error() == 0
