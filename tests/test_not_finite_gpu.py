"""GPU: infinities and NaN in the dense operand of a CSR product reach the outputs whose row stores a position
there, and no other, whichever way the product takes; elsewhere results equal those without them."""
import numpy as np
import pytest
import torch

from intrasm_engine_b200 import _lib
from intrasm_engine_b200.pytorch.cpp_extensions.layers_and_funcs.sputnik import MySpMM
from intrasm_engine_b200.pytorch.cpp_extensions.layers_and_funcs.utils import default_fwd_kwargs
from intrasm_engine_b200.pytorch.huggingface_rewriter import SparseLinear
from intrasm_engine_b200.pytorch.utils import dense_to_sparse_cuda, get_transpose_info

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _weight(m, k, density, seed):
    rng = np.random.default_rng(seed)
    w = (rng.integers(1, 4, (m, k)) * (rng.random((m, k)) < density)).astype(np.float16)
    w[0], w[1] = 0, 1  # an empty and a full row
    w[:, 5] = 0        # a column nobody stores
    return torch.as_tensor(w).to(DEV)


def _spoil(x, rows):
    """Small integers with values that are not finite in some rows [k, n]."""
    x[rows[0], 0], x[rows[1], -1] = float("inf"), float("nan")
    x[rows[1], 0] = -float("inf")
    x[5] = float("nan")
    return x


def _ref(w, x):
    """The stored positions' terms only, exactly: [m, k] x [k, n] of small integers."""
    finite = torch.nan_to_num(x.double(), 0.0, 0.0, 0.0)
    out = w.double() @ finite
    stored = (w != 0).double()
    nan = stored @ torch.isnan(x).double() > 0
    plus, minus = stored @ (x == float("inf")).double() > 0, stored @ (x == -float("inf")).double() > 0
    out[plus], out[minus] = float("inf"), -float("inf")
    out[nan | (plus & minus)] = float("nan")
    return out.half()


def _equal(a, b):
    return bool(((a == b) | (torch.isnan(a) & torch.isnan(b))).all())


@pytest.mark.parametrize("m,n,k", [(200, 72, 136), (304, 264, 520), (40, 520, 72)])
@pytest.mark.parametrize("a_mn,b_mn,out_t,parts", [(0, 1, 0, 1), (1, 1, 0, 1), (0, 0, 1, 1), (0, 0, 0, 2), (1, 1, 1, 2), (0, 1, 1, 1)])
@pytest.mark.parametrize("operand", [0, 1])
def test_gemm_of_a_dense_copy(m, n, k, a_mn, b_mn, out_t, parts, operand):
    rows, cols = (m, n) if operand == 0 else (n, m)
    w = _weight(rows, k, 0.3, m + n)
    x = _spoil(torch.randint(-2, 3, (k, cols), device=DEV).half(), (7, 11))
    values, _ri, ro, ci = dense_to_sparse_cuda(w)
    ref = _ref(w, x)
    a, b = (w, x.t()) if operand == 0 else (x.t(), w)  # [m, k], [n, k]
    if operand == 1:
        ref = ref.t()
    da, db = (a.t() if a_mn else a).contiguous(), (b.t() if b_mn else b).contiguous()
    out = torch.full((n, m) if out_t else (m, n), 9.0, dtype=torch.float16, device=DEV)
    perm = torch.randperm(values.numel(), device=DEV)
    shuffled = torch.empty_like(values)
    shuffled[perm] = values
    for v, p in ((values, None), (shuffled, perm.data_ptr())):
        _lib.call("iex_gemm_f16_csr", m, n, k, da.data_ptr(), a_mn, da.stride(0), db.data_ptr(), b_mn, db.stride(0),
                  out.data_ptr(), out_t, out.stride(0), operand, ro.data_ptr(), ci.data_ptr(), 32, v.data_ptr(), p, 64 * parts,
                  parts, torch.cuda.current_stream().cuda_stream)
        assert _equal(out.t() if out_t else out, ref)
    assert _lib.lib.iex_last_device_status(1) == 0


@pytest.mark.parametrize("n", [3, 10, 64, 100, 256, 300])
@pytest.mark.parametrize("m,k,density", [(300, 520, 0.5), (600, 1001, 0.2), (90, 64, 0.6)])
@pytest.mark.parametrize("auto", ["auto", True])
@pytest.mark.parametrize("index", [torch.int16, torch.int32])
def test_spmm_forward_and_backward(n, m, k, density, auto, index):
    w = _weight(m, k, density, m + k)
    values, ri, ro, ci = dense_to_sparse_cuda(w, index_dtype=index)
    info = get_transpose_info(m, k, ri, ro, ci)
    x = _spoil(torch.randint(-1, 2, (k, n), device=DEV).half(), (7, 11)).requires_grad_(True)
    out = MySpMM.run(x, ri, values, ro, ci, m, info, fwd_kwargs_1=default_fwd_kwargs(use_tensor_cores=auto))
    assert _equal(out.detach(), _ref(w, x.detach()))
    grad = torch.randint(-1, 2, (m, n), device=DEV).half()
    grad[3, 0], grad[4, -1], grad[0] = float("inf"), float("nan"), float("nan")  # row 0 stores nothing
    (gx,) = torch.autograd.grad(out, x, grad)
    assert _equal(gx, _ref(w.t().contiguous(), grad))
    assert _lib.lib.iex_last_device_status(1) == 0


@pytest.mark.parametrize("tokens", [1, 2, 3, 40, 64, 130, 300])
@pytest.mark.parametrize("density", [0.1, 0.5])  # without and with a dense copy
@pytest.mark.parametrize("out_features,in_features", [(264, 512), (100, 1000), (1000, 200)])
def test_sparse_linear(tokens, density, out_features, in_features):
    w = _weight(out_features, in_features, density, tokens)
    layer = SparseLinear(w)
    x = _spoil(torch.randint(-1, 2, (in_features, tokens), device=DEV).half(), (7, 11))
    assert _equal(layer(x.t().contiguous()), _ref(w, x).t())
    assert _lib.lib.iex_last_device_status(1) == 0


def test_decoder_with_bias_and_two_blocks_of_tokens():
    """The block decoder's own epilogue: bias and ReLU after the second sum (NaN becomes 0 there), 200 tokens."""
    m, k, n = 333, 640, 200
    w = _weight(m, k, 0.3, 9)
    values, _ri, ro, ci = dense_to_sparse_cuda(w, index_dtype=torch.int16)
    x = _spoil(torch.randint(-1, 2, (k, n), device=DEV).half(), (7, 300))
    bias = torch.arange(m, device=DEV).float()
    ref = _ref(w, x).float()
    ref = torch.where(ref + bias[:, None] > 0, ref + bias[:, None], torch.zeros_like(ref)).half()
    for tokens_major in (0, 1):
        dx = x.t().contiguous() if tokens_major else x
        out = torch.full((n, m) if tokens_major else (m, n), 9.0, dtype=torch.float16, device=DEV)
        _lib.call("iex_spmm_linear_f16_tile", m, 0, k, n, values.numel(), ro.data_ptr(), ci.data_ptr(), 16,
                  values.data_ptr(), None, dx.data_ptr(), tokens_major, bias.data_ptr(), out.data_ptr(), tokens_major, None, 0,
                  torch.cuda.current_stream().cuda_stream)
        assert _equal(out.t() if tokens_major else out, ref)
    assert _lib.lib.iex_last_device_status(1) == 0


def test_everything_not_finite_ends():
    """Every output is summed again, on several waves of tiles, within the waits' limits."""
    w = _weight(4096, 2048, 0.5, 1)
    layer = SparseLinear(w)
    x = torch.full((2000, 2048), float("nan"), device=DEV).half()
    out = layer(x)
    assert bool(torch.isnan(out[:, 1:]).all()) and not bool(out[:, 0].any())
    assert _lib.lib.iex_last_device_status(1) == 0


@pytest.mark.parametrize("m,k", [(700, 300), (700, 4608), (600, 4616), (40, 200), (300, 6144), (30, 6152), (900, 25000)])
@pytest.mark.parametrize("index", [torch.int16, torch.int32])
def test_columns_out_of_order_and_stored_twice(m, k, index):
    """Rows in falling order, rows with repeated columns next to each other, far apart and three times, odd starts and
    lengths: the sums over all positions, forward and backward, for every way of expanding a matrix."""
    rng = np.random.default_rng(m + k)
    rows = []
    for r in range(m):
        cols = np.sort(rng.choice(k, size=int(rng.integers(0, min(k, 200))), replace=False))
        if r % 4 == 1:
            cols = cols[::-1]
        elif r % 4 == 2 and len(cols) > 2:
            cols = np.concatenate([cols, cols[-1:]])
        elif r % 4 == 3 and len(cols) > 2:
            cols = np.concatenate([cols[:1], cols, cols[:1]])
        rows.append(cols)
    counts = [len(c) for c in rows]
    ro = torch.tensor(np.concatenate([[0], np.cumsum(counts)]), dtype=torch.int32, device=DEV)
    ci = torch.tensor(np.concatenate(rows).astype(np.int32), device=DEV).to(index)
    values = torch.randint(1, 4, (ci.numel(),), device=DEV).half()
    ri = torch.arange(m, dtype=torch.int32, device=DEV)
    info = get_transpose_info(m, k, ri, ro, ci)
    where = torch.repeat_interleave(torch.arange(m, device=DEV), (ro[1:] - ro[:-1]).long())
    dense = torch.zeros(m, k, dtype=torch.float64, device=DEV).index_put((where, ci.long()), values.double(), accumulate=True)
    n = 72 if m > 100 else 300
    x = torch.randint(-1, 2, (k, n), device=DEV).half().requires_grad_(True)
    grad = torch.randint(-1, 2, (m, n), device=DEV).half()
    for auto in ("auto", True):
        out = MySpMM.run(x, ri, values, ro, ci, m, info, fwd_kwargs_1=default_fwd_kwargs(use_tensor_cores=auto))
        assert torch.equal(out.detach().double(), dense @ x.detach().double())
        (gx,) = torch.autograd.grad(out, x, grad)
        assert torch.equal(gx.double(), dense.t() @ grad.double())
    assert _lib.lib.iex_last_device_status(1) == 0
