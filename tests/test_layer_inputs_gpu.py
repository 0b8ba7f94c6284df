"""GPU: what the layers do with inputs of the wrong size (an error on the host, before any launch) and
with inputs that are only aligned to their element size (the same result as from an aligned copy)."""
import pytest
import torch

from intrasm_engine_b200 import _lib, ops
from intrasm_engine_b200.pytorch.ffn import relu_down_proj
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


def _misaligned(t, by=1):
    """The same values at an address that is `by` elements off a 16-byte boundary, contiguous."""
    buf = torch.empty(t.numel() + 8, dtype=t.dtype, device=t.device)
    out = buf[by:by + t.numel()].view(t.shape)
    out.copy_(t)
    assert out.data_ptr() % 16 != 0 and out.is_contiguous()
    return out


@pytest.mark.parametrize("density", [0.1, 0.5])
@pytest.mark.parametrize("tokens", [1, 2, 3, 64, 300])
def test_sparse_linear_misaligned(density, tokens):
    """The activations, and the nonzeros, at odd addresses."""
    w = _weight(264, 512, density, 2)
    layer = SparseLinear(w)
    x = torch.randn(tokens, 512, device=DEV).half()
    ref = (x.double() @ w.double().t())
    bound = 2.0 ** -10 * ref.abs() + 1e-5 * (x.double().abs() @ w.double().abs().t()) + 2.0 ** -24  # one rounding, fp32 sums
    for by in (1, 2, 4):
        assert bool(((layer(_misaligned(x, by)).double() - ref).abs() <= bound).all())
    for dense in (layer.dense_copy(), None):
        y = ops.native.sparse_linear(x, _misaligned(layer.values.detach()), layer.row_offsets,
                                     _misaligned(layer.column_indices), 264, 512, dense)
        assert bool(((y.double() - ref).abs() <= bound).all())
    assert _lib.lib.iex_last_device_status(1) == 0


@pytest.mark.parametrize("tokens,k", [(1, 8), (32, 1000), (200, 4104)])
def test_relu_down_proj_misaligned(tokens, k):
    hidden = torch.randn(tokens, k, device=DEV).half()
    hidden[0, 3], hidden[0, 5] = float("nan"), -float("inf")  # the ReLU makes zeros of both
    w = (torch.randn(136, k, device=DEV) * 0.05).half()
    ref = relu_down_proj(hidden, w)
    act = torch.where(hidden > 0, hidden, torch.zeros_like(hidden)).double()
    bound = 2.0 ** -10 * (act @ w.double().t()).abs() + 1e-5 * (act @ w.double().abs().t()) + 2.0 ** -24
    assert bool(((ref.double() - act @ w.double().t()).abs() <= bound).all())
    for by in (1, 4, 7):
        assert torch.equal(relu_down_proj(_misaligned(hidden, by), w), ref)
