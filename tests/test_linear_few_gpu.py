"""GPU: the linear layer for a handful of tokens against fp64: rows and columns around a block's and a pass's edges, the
dense copy of a CSR weight with inputs that are not finite, and the layers that reach it."""
import pytest
import torch

from intrasm_engine_b200 import _lib
from intrasm_engine_b200.pytorch.cpp_extensions.layers_and_funcs.torch import MyLinear
from intrasm_engine_b200.pytorch.huggingface_rewriter import SparseLinear

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _rand(shape, seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return torch.randn(shape, generator=g, device=DEV).half()


def _close(y, x, w):
    ref = x.double() @ w.double().t()
    bound = 2.0 ** -10 * ref.abs() + 1e-5 * (x.double().abs() @ w.double().abs().t()) + 2.0 ** -24  # one rounding, fp32 sums
    return bool(((y.double() - ref).abs() <= bound).all())


@pytest.mark.parametrize("tokens", [1, 2, 3, 4, 5, 8])
@pytest.mark.parametrize("out_features,in_features", [
    (1, 8), (3, 2048), (5, 2056), (296, 16), (297, 2040), (1188, 512), (18945, 64), (40, 4096)])
def test_few_tokens(tokens, out_features, in_features):
    x, w = _rand((tokens, in_features), tokens), _rand((out_features, in_features), out_features)
    y = torch.full((tokens * out_features + 8,), 7.0, dtype=torch.float16, device=DEV)
    st = _lib.lib.iex_linear_f16_few(tokens, in_features, out_features, x.data_ptr(), w.data_ptr(), y.data_ptr(), 0, 0, 0, 0,
                                     torch.cuda.current_stream().cuda_stream)
    assert st == 0 and _lib.lib.iex_linear_f16_few_supported(tokens, in_features)
    assert _close(y[:tokens * out_features].view(tokens, out_features), x, w)
    assert bool((y[tokens * out_features:] == 7).all())


def test_what_is_refused():
    few = _lib.lib.iex_linear_f16_few_supported
    assert not few(9, 64) and not few(0, 64) and not few(1, 12) and not few(8, 4104) and few(8, 4096) and few(1, 32768)
    x, w, y = _rand((1, 72), 1), _rand((9, 72), 2), _rand((1, 9), 3)
    assert _lib.lib.iex_linear_f16_few(1, 64, 8, x.data_ptr() + 2, w.data_ptr(), y.data_ptr(), 0, 0, 0, 0, 0) == -2


@pytest.mark.parametrize("tokens", [1, 2, 4])
def test_layers_with_a_handful_of_tokens(tokens):
    x, w = _rand((tokens, 1032), 4), _rand((1099, 1032), 5) * 0.05
    assert _close(MyLinear.run(x, w), x, w)
    kept = torch.where(torch.rand(w.shape, device=DEV) < 0.5, w, torch.zeros_like(w))
    kept[:, 3] = 0
    layer = SparseLinear(kept)
    assert layer.dense_copy() is not None and _close(layer(x), x, kept)
    clean, finite = layer(x), x.clone()
    x[0, 3] = float("inf")  # stored nowhere
    finite[0, 3] = 0
    assert _close(layer(x), finite, kept)
    x[0, 4] = float("nan")
    stored = kept[:, 4] != 0
    y = layer(x)
    assert bool(torch.isnan(y[0, stored]).all()) and bool(torch.isfinite(y[0, ~stored]).all()) and torch.equal(y[1:], clean[1:])
