"""GPU: the linear layer for a handful of tokens against fp64: rows and columns around a block's, a row tile's and a piece's edges, the
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


@pytest.mark.parametrize("tokens", [1, 2, 5, 8, 9, 16])
@pytest.mark.parametrize("out_features,in_features", [
    (1, 8), (3, 2048), (9, 2056), (296, 16), (1184, 40), (1185, 2040), (2369, 520), (4737, 512), (11009, 72), (14209, 64),
    (30000, 24), (40, 4096)])
def test_few_tokens(tokens, out_features, in_features):
    x, w = _rand((tokens, in_features), tokens), _rand((out_features, in_features), out_features)
    y = torch.full((tokens * out_features + 8,), 7.0, dtype=torch.float16, device=DEV)
    st = _lib.lib.iex_linear_f16_few(tokens, in_features, out_features, x.data_ptr(), w.data_ptr(), y.data_ptr(), tokens % 2, 0, 0, 0, 0,
                                     torch.cuda.current_stream().cuda_stream)
    assert st == 0 and _lib.lib.iex_linear_f16_few_supported(tokens, in_features)
    assert _close(y[:tokens * out_features].view(tokens, out_features), x, w)
    assert bool((y[tokens * out_features:] == 7).all())


@pytest.mark.parametrize("settled", [0, 1])
@pytest.mark.parametrize("tokens,features", [(1, 4096), (3, 2048), (16, 1024)])
def test_chained_calls_see_each_other(tokens, features, settled):
    """Each call reads what the one in front, which it may overlap, has written."""
    stream = torch.cuda.current_stream().cuda_stream
    weights = [_rand((features, features), i) * (1.0 / features ** 0.5) for i in range(5)]
    bufs = [_rand((tokens, features), 9)] + [torch.empty((tokens, features), dtype=torch.float16, device=DEV) for _ in range(5)]

    def chain(one_by_one):
        for i, w in enumerate(weights):
            assert _lib.lib.iex_linear_f16_few(tokens, features, features, bufs[i].data_ptr(), w.data_ptr(),
                                               bufs[i + 1].data_ptr(), settled, 0, 0, 0, 0, stream) == 0
            if one_by_one:
                torch.cuda.synchronize()
        return [b.clone() for b in bufs]

    ref = chain(True)
    for turn in range(40):
        for b in bufs[1:]:
            b.fill_(float(turn % 7))
        assert all(torch.equal(a, b) for a, b in zip(ref, chain(False)))


def test_a_weight_written_by_the_call_in_front():
    """Not settled: the weight is the result of the launch in front."""
    stream = torch.cuda.current_stream().cuda_stream
    x, m, w0 = _rand((8, 2048), 1), _rand((8, 2048), 2), _rand((2048, 2048), 3) * 0.02
    w = torch.empty((8, 2048), dtype=torch.float16, device=DEV)
    y, ref = torch.empty((8, 8), dtype=torch.float16, device=DEV), torch.empty((8, 8), dtype=torch.float16, device=DEV)

    def run(out, one_by_one):
        assert _lib.lib.iex_linear_f16_few(8, 2048, 2048, m.data_ptr(), w0.data_ptr(), w.data_ptr(), 0, 0, 0, 0, 0, stream) == 0
        if one_by_one:
            torch.cuda.synchronize()
        assert _lib.lib.iex_linear_f16_few(8, 2048, 8, x.data_ptr(), w.data_ptr(), out.data_ptr(), 0, 0, 0, 0, 0, stream) == 0

    run(ref, True)
    for _ in range(40):
        w.zero_()
        run(y, False)
        assert torch.equal(y, ref)


def test_what_is_refused():
    few = _lib.lib.iex_linear_f16_few_supported
    assert not few(17, 64) and not few(0, 64) and not few(1, 12) and few(16, 4104) and few(1, 32768)
    x, w, y = _rand((1, 72), 1), _rand((9, 72), 2), _rand((1, 9), 3)
    assert _lib.lib.iex_linear_f16_few(1, 64, 8, x.data_ptr() + 2, w.data_ptr(), y.data_ptr(), 0, 0, 0, 0, 0, 0) == -2


@pytest.mark.parametrize("tokens", [1, 2, 4, 12])
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


@pytest.mark.parametrize("tokens,in_features,out_features,shift", [(9, 2048, 5001, 0), (16, 4096, 5001, 0), (12, 8192, 2001, 0), (9, 4096, 4096, 1)])
def test_compared_with_the_gemm_that_can_run(tokens, in_features, out_features, shift):
    """Odd numbers of features, and results at odd addresses, rule the weight-as-A product out: its estimate, the lower one, does not count."""
    few = 1.15 * _lib.lib.iex_linear_f16_few_estimate_us(tokens, in_features, out_features, 0)
    assert _lib.lib.iex_gemm_f16_estimate_us(out_features, tokens, in_features, 0, 1) < few
    assert few <= _lib.lib.iex_gemm_f16_estimate_us(tokens, out_features, in_features, 0, 0)
    x, w = _rand((tokens, in_features), 6), _rand((out_features, in_features), 7)
    y, own = (torch.zeros(tokens * out_features + 8, dtype=torch.float16, device=DEV)[shift:tokens * out_features + shift] for _ in range(2))
    stream = torch.cuda.current_stream().cuda_stream
    assert _lib.lib.iex_linear_f16_any(tokens, in_features, out_features, x.data_ptr(), w.data_ptr(), y.data_ptr(), stream) == 0
    assert _lib.lib.iex_linear_f16_few(tokens, in_features, out_features, x.data_ptr(), w.data_ptr(), own.data_ptr(), 0, 0, 0, 0, 0,
                                       stream) == 0
    assert _close(y.view(tokens, out_features), x, w) and torch.equal(y, own)  # its order of summation
