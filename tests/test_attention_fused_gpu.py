"""GPU: masked attention over heads in one launch against fp64: tile, band and part edges, bands cut between
CTAs, one-tile bands, values of v that are not finite outside and inside the mask."""
import numpy as np
import pytest
import torch

from intrasm_engine_b200 import _lib
from intrasm_engine_b200.pytorch.attention import SparseAttentionChain
from intrasm_engine_b200.pytorch.utils import dense_to_sparse_cuda

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _mask(m, n, density, seed):
    rng = np.random.default_rng(seed)
    mask = torch.as_tensor(rng.random((m, n)) < density).to(DEV)
    _values, _ri, ro, ci = dense_to_sparse_cuda(mask.to(torch.float16))
    return mask, ro, ci


def _qkv(heads, m, n, d, dv, seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return tuple(torch.randn(s, generator=g, device=DEV) for s in ((heads, m, d), (heads, n, d), (heads, n, dv)))


@pytest.mark.parametrize("heads,m,n,d,dv,density", [
    (1, 128, 64, 64, 64, 0.5), (2, 129, 65, 32, 32, 0.3), (3, 300, 520, 48, 48, 0.1), (2, 100, 900, 80, 80, 0.1),
    (2, 260, 33, 96, 20, 0.3), (1, 500, 700, 4, 4, 0.1), (2, 200, 300, 32, 96, 0.1), (2, 140, 200, 100, 116, 0.2),
    (300, 128, 64, 64, 64, 0.2), (150, 128, 128, 64, 64, 0.2), (100, 130, 100, 32, 64, 0.2), (18, 1179, 200, 64, 64, 0.05),
    (60, 300, 100, 128, 128, 0.1), (1, 130, 3000, 64, 64, 0.1), (5, 600, 900, 80, 80, 0.1), (70, 250, 700, 64, 64, 0.1),
    (76, 250, 333, 48, 64, 0.1)])
def test_one_launch_chain(heads, m, n, d, dv, density):
    mask, ro, ci = _mask(m, n, density, heads + m)
    chain = SparseAttentionChain(ro, ci, m, n)
    assert chain.bits is not None and _lib.lib.iex_attention_f32_supported(heads, m, n, d, dv)
    q, k, v = _qkv(heads, m, n, d, dv, m + n)
    out = chain(q, k, v)
    ref = torch.where(mask, q.double() @ k.double().transpose(1, 2), torch.zeros((), dtype=torch.float64, device=DEV)) @ v.double()
    err = (out.double() - ref).flatten(1).norm(dim=1) / ref.flatten(1).norm(dim=1)
    assert float(err.max()) < 1e-6
    assert torch.equal(out, chain(q, k, v))  # the pieces of a shared band are added in order
    assert _lib.lib.iex_last_device_status(1) == 0


def test_values_that_are_not_finite():
    mask, ro, ci = _mask(300, 200, 0.1, 3)
    mask[:, 7] = False
    _v, _ri, ro, ci = dense_to_sparse_cuda(mask.to(torch.float16))
    chain = SparseAttentionChain(ro, ci, 300, 200)
    q, k, v = _qkv(3, 300, 200, 64, 64, 9)
    clean = chain(q, k, v)
    v[1, 7] = float("nan")    # masked everywhere: must not be seen
    v[2, 11, 5] = float("inf")
    out = chain(q, k, v)
    assert torch.equal(out[0], clean[0])
    assert torch.allclose(out[1], clean[1], rtol=1e-5, atol=1e-4)
    seen = mask[:, 11]
    assert bool(torch.isinf(out[2, seen, 5]).all()) and bool(torch.isfinite(out[2, ~seen]).all())


def test_repeated_position_takes_the_operators():
    ro = torch.tensor([0, 2], dtype=torch.int32, device=DEV)
    ci = torch.tensor([1, 1], dtype=torch.int32, device=DEV)
    chain = SparseAttentionChain(ro, ci, 1, 4)
    assert chain.bits is None
    q, k, v = _qkv(1, 1, 4, 32, 32, 1)
    ref = 2 * (q[0] @ k[0, 1]) * v[0, 1]
    assert torch.allclose(chain(q, k, v)[0, 0], ref, rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("heads,m,d,width", [(2, 16384, 64, 32), (3, 4096, 128, 64), (1, 8192, 80, 16)])
def test_sparse_bands_take_the_operators(heads, m, d, width):
    """Large masks with few positions: no launch over every tile and, where no width of q and v would want one,
    no bits of the whole matrix."""
    rows = torch.arange(m, device=DEV)[:, None]
    cols = rows + torch.arange(-width // 2, width // 2, device=DEV)[None, :]
    inside = (cols >= 0) & (cols < m)
    ro = torch.zeros(m + 1, dtype=torch.int32, device=DEV)
    ro[1:] = torch.cumsum(inside.sum(1), 0)
    ci = cols[inside].to(torch.int32)
    nnz = ci.numel()
    before = torch.cuda.memory_allocated()
    chain = SparseAttentionChain(ro, ci, m, m)
    assert not _lib.lib.iex_attention_f32_prefers(heads, m, m, d, d, nnz)
    if m == 16384:
        assert chain.bits is None and torch.cuda.memory_allocated() - before < m * m // 16
    q, k, v = _qkv(heads, m, m, d, d, m)
    out = chain(q, k, v)
    index = cols.clamp(0, m - 1)
    for h in range(heads):
        s = torch.einsum("rd,rwd->rw", q[h].double(), k[h].double()[index]) * inside
        ref = torch.einsum("rw,rwd->rd", s, v[h].double()[index])
        assert float((out[h].double() - ref).norm() / ref.norm()) < 1e-6
    scored, scores = chain(q, k, v, return_scores=True)
    assert torch.equal(out, scored) and scores.shape == (heads, nnz)


def test_chain_made_while_a_stream_is_recorded():
    """Making a chain reads nothing back then; it works without the bits."""
    mask, ro, ci = _mask(200, 300, 0.1, 5)
    q, k, v = _qkv(2, 200, 300, 64, 64, 1)
    ref = SparseAttentionChain(ro, ci, 200, 300)(q, k, v)
    SparseAttentionChain(ro, ci, 200, 300)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        chain = SparseAttentionChain(ro, ci, 200, 300)
        out = chain(q, k, v)
    assert chain.bits is None
    graph.replay()
    torch.cuda.synchronize()
    assert torch.allclose(out, ref, rtol=1e-5, atol=1e-3)
    del graph
