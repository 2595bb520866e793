"""The network's input at sequence lengths where three channel strides pass 2^31, and at small ragged ones."""

import pytest

torch = pytest.importorskip("torch")

from modlefork_gb300 import surrogate_ops as ops  # noqa: E402

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("B,L,C", [(1, 1, 8), (3, 77, 64), (1, 716_000_003, 8)])
def test_assemble_input(B, L, C):
    if L > 1 << 20 and torch.cuda.mem_get_info()[0] < 64 << 30:
        pytest.skip("needs 24 GB of device memory")
    track = torch.zeros(B, 4, L, device=DEV)
    at = torch.tensor([0, L // 3, L - 1], device=DEV)
    for c in range(4):
        track[:, c, at] = torch.arange(1.0, 4.0, device=DEV) * (c + 1)
    params = torch.arange(1.0, 5.0, device=DEV).repeat(B, 1)
    x = torch.full((B, L, C), 9.0, dtype=torch.bfloat16, device=DEV)
    ops.assemble_input(track, params, x)
    for i in at.tolist():
        assert torch.equal(x[:, i, :4].float(), track[:, :, i])
        assert torch.equal(x[:, i, 4:8].float(), params) and not x[:, i, 8:].any()
