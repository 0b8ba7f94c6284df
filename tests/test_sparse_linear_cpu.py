"""CPU: an input of the wrong width to ``SparseLinear`` is an error on the host, whichever way the
layer would have taken; no call reaches the native side."""
import pytest
import torch
from torch import nn

from intrasm_engine_b200 import ops
from intrasm_engine_b200.pytorch.huggingface_rewriter import SparseLinear
from intrasm_engine_b200.pytorch.utils import DenseCopy


class _SaysCuda(torch.Tensor):
    """A host tensor that takes the branches of a CUDA tensor."""

    is_cuda = True


class _Native:
    def __init__(self):
        self.widths = []

    def sparse_linear(self, x, values, ro, ci, m, *rest):
        self.widths.append(x.size(1))
        return torch.zeros(x.size(0), m, dtype=x.dtype)


def _layer(in_features, out_features):
    layer = SparseLinear.__new__(SparseLinear)
    nn.Module.__init__(layer)
    layer.in_features, layer.out_features, layer.bias = in_features, out_features, None
    layer.values = nn.Parameter(torch.ones(4, dtype=torch.float16), requires_grad=False)
    layer.row_offsets = layer.column_indices = torch.zeros(1, dtype=torch.int32)
    layer._dense = DenseCopy(out_features, in_features)
    return layer


@pytest.mark.parametrize("shape", [(3, 8), (4, 32), (1, 15), (2, 3, 8), (16, 1), (3, 0)])
@pytest.mark.parametrize("grad", [False, True])
def test_wrong_width_raises_before_any_call(monkeypatch, shape, grad):
    native = _Native()
    monkeypatch.setattr(ops, "native", native)
    x = torch.zeros(shape, dtype=torch.float16).as_subclass(_SaysCuda)
    with pytest.raises(RuntimeError, match="16 input features"):
        _layer(16, 24)(x.requires_grad_(grad))
    assert native.widths == []


@pytest.mark.parametrize("shape", [(3, 16), (16,), (2, 5, 16), (0, 16), (0, 7)])
def test_right_width_passes(monkeypatch, shape):
    native = _Native()
    monkeypatch.setattr(ops, "native", native)
    x = torch.zeros(shape, dtype=torch.float16).as_subclass(_SaysCuda)
    assert _layer(16, 24)(x).shape == (*shape[:-1], 24)
    assert native.widths == [16]
