"""A list of weight transposes holds addresses for its calls; copies and pickles of it take the tensors only."""

import copy
import io

import pytest

torch = pytest.importorskip("torch")

from modlefork_gb300 import surrogate_ops as ops  # noqa: E402


def _addresses(lst):
    return [[list(c[1]), list(c[5])] for c in lst._arguments()]


def test_transpose_list_copies():
    pairs = [(torch.zeros(8 * k, 3, 8), torch.zeros(8, 3, 8 * k)) for k in range(1, 71)]
    lst = ops.TransposeList(pairs)
    lst.calls = lst._arguments()
    held = {"list": lst, "w": [w for w, _ in pairs]}
    deep = copy.deepcopy(held)
    buf = io.BytesIO()
    torch.save(held, buf)
    buf.seek(0)
    for other in (deep, torch.load(buf, weights_only=False)):
        new = other["list"]
        assert new.calls is None and len(new.pairs) == 70
        got = [a for call in _addresses(new) for a in call[0]]
        assert got == [w.data_ptr() for w in other["w"]] and not set(got) & {w.data_ptr() for w, _ in pairs}
        assert [c[0] for c in new._arguments()] == [64, 6]
