"""GPU: what records, transforms or differentiates a program sees the operator classes and layers, although
their usual calls go past the dispatcher: tracing, dispatch modes, tensor subclasses, forward-mode
derivatives, hooks on saved tensors, in-place changes before the backward pass, second derivatives."""
import contextlib

import pytest
import torch
from torch.autograd import forward_ad

from intrasm_engine_b200.pytorch.cpp_extensions.layers_and_funcs.sputnik import MySpMM
from intrasm_engine_b200.pytorch.cpp_extensions.layers_and_funcs.torch import MyLinear
from intrasm_engine_b200.pytorch.cpp_extensions.layers_and_funcs.utils import default_fwd_kwargs
from intrasm_engine_b200.pytorch.horizontal_rewriter import SparseDenseLayer
from intrasm_engine_b200.pytorch.huggingface_rewriter import SparseLinear
from intrasm_engine_b200.pytorch.utils import dense_to_sparse_cuda, get_transpose_info

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
M, K, N = 96, 64, 64


def _pattern(dtype, seed=0):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    w = torch.randn(M, K, generator=g, device=DEV).to(dtype)
    w = torch.where(torch.rand(M, K, generator=g, device=DEV) < 0.4, w, torch.zeros_like(w))
    values, ri, ro, ci = dense_to_sparse_cuda(w)
    return w, values, ri, ro, ci, get_transpose_info(M, K, ri, ro, ci)


def _spmm(dtype, auto):
    _w, values, ri, ro, ci, transp = _pattern(dtype)

    def call(b):
        return MySpMM.run(b, ri, values, ro, ci, M, transp, fwd_kwargs_1=default_fwd_kwargs(use_tensor_cores=auto))
    return call, torch.randn(K, N, device=DEV).to(dtype)


def _call(name):
    """A function of one tensor and an input of it."""
    if name.startswith("spmm"):
        return _spmm(torch.float32 if name == "spmm-f32" else torch.float16, "auto" if name.endswith("auto") else False)
    w, values, ri, ro, ci, _t = _pattern(torch.float16)
    weight = torch.randn(40, K, device=DEV).half()
    if name == "linear":
        return lambda x: MyLinear.run(x, weight), torch.randn(8, K, device=DEV).half()
    if name == "sparse-linear":
        return SparseLinear(w), torch.randn(8, K, device=DEV).half()
    both = SparseDenseLayer(values, ri, ro, ci, M, weight)
    return lambda x: torch.cat([t.flatten() for t in both(x)]), torch.randn(K, N, device=DEV).half()


@pytest.fixture(params=["spmm-f32", "spmm-f16", "spmm-f16-auto", "linear", "sparse-linear", "sparse-dense"])
def call(request):
    return _call(request.param)


def _same(a, b):
    return torch.allclose(a.float(), b.float(), rtol=2e-3, atol=2e-3 * float(b.float().abs().max()))


def test_trace_follows_the_input(call):
    f, x = call
    traced = torch.jit.trace(f, (x,), check_trace=False)
    other = torch.randn_like(x)
    assert _same(traced(other), f(other))


def test_dispatch_mode_sees_the_operators(call):
    from torch.fx.experimental.proxy_tensor import make_fx
    f, x = call
    graph = make_fx(f)(x)
    assert any("iex_ops" in str(node.target) for node in graph.graph.nodes)
    other = torch.randn_like(x)
    assert _same(graph(other), f(other))


def test_tangents_are_not_dropped(call):
    f, x = call
    with forward_ad.dual_level(), pytest.raises(NotImplementedError):
        f(forward_ad.make_dual(x, torch.ones_like(x)))


def test_vmap_is_refused(call):
    f, x = call
    with pytest.raises(RuntimeError):
        torch.vmap(f)(torch.stack([x, x]))


def test_negative_view(call):
    """A tensor that only says it is negated."""
    f, x = call
    assert _same(f(torch._neg_view(x)), f(-x))


def test_subclass_reaches_its_own_dispatch():
    class Wrapped(torch.Tensor):
        @staticmethod
        def __new__(cls, inner):
            return torch.Tensor._make_wrapper_subclass(cls, inner.shape, dtype=inner.dtype, device=inner.device)

        def __init__(self, inner):
            self.inner = inner

        @classmethod
        def __torch_dispatch__(cls, func, types, args=(), kwargs=None):
            seen.append(str(func))
            unwrap = lambda t: t.inner if isinstance(t, cls) else t
            return func(*(unwrap(a) for a in args), **(kwargs or {}))

    seen = []
    _w, values, ri, ro, ci, transp = _pattern(torch.float32)
    b = torch.randn(K, N, device=DEV)
    out = MySpMM.run(Wrapped(b), ri, values, ro, ci, M, transp)
    assert seen and torch.equal(out, MySpMM.run(b, ri, values, ro, ci, M, transp))


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_saved_tensors(dtype):
    """Hooks see the operands and the pattern; changing one of them in place before the backward pass raises."""
    _w, values, ri, ro, ci, transp = _pattern(dtype)
    b = torch.randn(K, N, device=DEV).to(dtype)

    def run(hooks=None):
        x, v = b.clone().requires_grad_(True), values.clone().requires_grad_(True)
        with torch.autograd.graph.saved_tensors_hooks(*hooks) if hooks else contextlib.nullcontext():
            return MySpMM.run(x, ri, v, ro, ci, M, transp), x, v

    packed = []
    y, x, v = run((lambda t: packed.append(t.shape) or t.cpu(), lambda t: t.to(DEV)))
    ref = torch.autograd.grad(*(lambda r: (r[0].float().sum(), r[1:]))(run()))
    got = torch.autograd.grad(y.float().sum(), (x, v))
    assert len(packed) == 9 and all(torch.equal(a, r) for a, r in zip(got, ref))
    y, x, v = run()
    ci.add_(0)
    with pytest.raises(RuntimeError, match="inplace"):
        y.float().sum().backward()
    y, x, v = run()
    y.float().sum().backward()
    with pytest.raises(RuntimeError, match="second time"):
        y.float().sum().backward()


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_second_derivatives_of_the_product_are_an_error(dtype):
    _w, values, ri, ro, ci, transp = _pattern(dtype)
    x = torch.randn(K, N, device=DEV).to(dtype).requires_grad_(True)
    v = values.clone().requires_grad_(True)
    y = MySpMM.run(x, ri, v, ro, ci, M, transp).float()
    gx, gv = torch.autograd.grad(y.pow(2).sum(), (x, v), create_graph=True)
    once = torch.autograd.grad(MySpMM.run(x, ri, v, ro, ci, M, transp).float().pow(2).sum(), (x, v))
    assert torch.equal(gx, once[0]) and torch.equal(gv, once[1])
    for g in (gx, gv):
        with pytest.raises(RuntimeError, match="twice"):
            torch.autograd.grad(g.float().sum(), (x, v), retain_graph=True)


@pytest.mark.parametrize("features", [40, 41])
def test_second_derivatives_of_the_linear(features):
    """Features that are no multiple of 8 take library products in the backward pass, which have one."""
    x0, w0 = torch.randn(8, K, device=DEV).half(), torch.randn(features, K, device=DEV).half()
    results = []
    for own, f in ((True, MyLinear.run), (False, lambda x, w: x @ w.t())):
        x, w = x0.clone().requires_grad_(True), w0.clone().requires_grad_(True)
        gx, gw = torch.autograd.grad(f(x, w).float().pow(2).sum(), (x, w), create_graph=True)
        loss = gx.float().mean() + gw.float().mean()
        if own and features % 8 == 0:
            with pytest.raises(RuntimeError, match="twice"):
                torch.autograd.grad(loss, (x, w))
            return
        results.append(torch.autograd.grad(loss, (x, w)))
    assert all(_same(a, b) for a, b in zip(*results))
