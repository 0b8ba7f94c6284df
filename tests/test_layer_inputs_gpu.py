"""GPU: what the layers do with inputs of the wrong size (an error on the host, before any launch) and
with inputs that are only aligned to their element size (the same result as from an aligned copy)."""
import pytest
import torch

from intrasm_engine_b200 import _lib, ops
from intrasm_engine_b200.pytorch.huggingface_rewriter import SparseLinear

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _weight(out_features, in_features, density, seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    w = (torch.randn(out_features, in_features, generator=g, device=DEV) * 0.05).half()
    return torch.where(torch.rand(out_features, in_features, generator=g, device=DEV) < density, w, torch.zeros_like(w))


@pytest.mark.parametrize("density", [0.1, 0.5])  # without and with a dense copy of the weight
@pytest.mark.parametrize("tokens", [1, 2, 40, 300])
def test_sparse_linear_width(density, tokens):
    layer = SparseLinear(_weight(264, 512, density, 1))
    for width in (256, 504, 520, 1024):
        x = torch.randn(tokens, width, device=DEV).half()
        with pytest.raises(RuntimeError):
            layer(x)
        with pytest.raises(RuntimeError):
            layer(x[None])
        with pytest.raises(RuntimeError):
            ops.native.sparse_linear(x, layer.values, layer.row_offsets, layer.column_indices, 264, 512, None)
    assert layer(torch.zeros(tokens, 512, device=DEV).half()).shape == (tokens, 264)
    assert _lib.lib.iex_last_device_status(1) == 0
