"""GPU: the CTA-pair GEMM, the block decoder, the few-token SpMM and the CSR expansion at the sizes where
they can go wrong (edges of tiles and blocks, remainders, odd counts), exact on small integers."""
import numpy as np
import pytest
import torch

from intrasm_engine_b200 import _lib, ops
from intrasm_engine_b200.pytorch.horizontal_rewriter import SparseDenseLayer
from intrasm_engine_b200.pytorch.utils import DenseCopy, dense_to_sparse_cuda

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _ints(shape, seed, low=-2, high=3, density=1.0):
    rng = np.random.default_rng(seed)
    a = rng.integers(low, high, size=shape).astype(np.float16)
    if density < 1.0:
        a *= rng.random(shape) < density
    return a


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a)).to(DEV)


def _exact(a, b):
    ref = a.astype(np.float32) @ b.astype(np.float32)
    assert np.abs(ref).max(initial=0) < 2048
    return ref.astype(np.float16)


def _stream():
    return torch.cuda.current_stream().cuda_stream


@pytest.mark.parametrize("m,n,k", [(1, 8, 8), (256, 256, 64), (257, 264, 72), (1000, 136, 320), (40, 1024, 200)])
@pytest.mark.parametrize("a_mn,b_mn,out_t", [(0, 0, 0), (0, 0, 1), (1, 0, 1), (0, 1, 0), (1, 1, 0)])
def test_gemm_layouts(m, n, k, a_mn, b_mn, out_t):
    m, n = (m + 7) // 8 * 8 if a_mn or out_t else m, (n + 7) // 8 * 8
    a, b = _ints((m, k), m + n), _ints((n, k), m + k)
    ref = _exact(a, b.T)
    da, db = _dev(a.T if a_mn else a), _dev(b.T if b_mn else b)
    for tile_n, parts in ((0, 0), (64, 1), (192, 1), (256, 1), (128, 2), (256, 3), (64, 4)):
        if parts > (k + 63) // 64:
            continue
        out = torch.full((n, m) if out_t else (m, n), 9.0, dtype=torch.float16, device=DEV)
        _lib.call("iex_gemm_f16", m, n, k, da.data_ptr(), a_mn, da.stride(0), db.data_ptr(), b_mn, db.stride(0),
                  out.data_ptr(), out_t, out.stride(0), tile_n, parts, _stream())
        np.testing.assert_array_equal(out.cpu().numpy(), ref.T if out_t else ref)
    assert _lib.lib.iex_last_device_status(1) == 0


@pytest.mark.parametrize("n", [1, 3, 10, 77])
def test_gemm_unaligned_output_rows(n):
    """Output rows that are no multiple of 16 bytes, in a wider buffer that must stay untouched."""
    m, k = 130, 256
    a, b = _ints((m, k), n), _ints((n, k), n + 1)
    out = torch.full((m, n + 2), 9.0, dtype=torch.float16, device=DEV)
    da, db = _dev(a), _dev(b)
    for parts in (1, 2):
        _lib.call("iex_gemm_f16", m, n, k, da.data_ptr(), 0, k, db.data_ptr(), 0, k, out.data_ptr(), 0, n + 2, 64,
                  parts, _stream())
        got = out.cpu().numpy()
        np.testing.assert_array_equal(got[:, :n], _exact(a, b.T))
        assert (got[:, n:] == 9.0).all()


@pytest.mark.parametrize("m,k,n,density", [(1, 64, 1, 1.0), (8, 72, 3, 0.9), (300, 520, 64, 0.5), (301, 1016, 65, 0.1),
                                           (1000, 2048, 128, 0.95), (2500, 512, 129, 0.3), (20000, 136, 256, 0.4),
                                           (640, 4096, 17, 0.02)])
@pytest.mark.parametrize("index", [torch.int16, torch.int32])
def test_block_decoder(m, k, n, density, index):
    """Uneven rows (one full, one empty), odd nonzero counts, both layouts of x and of the output, alone and
    beside a dense matrix."""
    a = _ints((m, k), m + k, density=density)
    a[0] = 1
    if m > 2:
        a[1] = 0
    md = 200
    w, x = _ints((md, k), 1), _ints((n, k), 2, -1, 2)
    ref_s, ref_d = _exact(a, x.T), _exact(w, x.T)
    values, _ri, ro, ci = dense_to_sparse_cuda(_dev(a), index_dtype=index)
    if values.numel() < 64:
        pytest.skip("fewer nonzeros than the decoder takes")
    dw, bits = _dev(w), 16 if index == torch.int16 else 32
    for tokens_major in (1, 0):
        if not tokens_major and n % 8:
            continue
        dx = _dev(x if tokens_major else x.T)
        for rows_d in (0, md):
            os_ = torch.full((n, m) if tokens_major else (m, n), 9.0, dtype=torch.float16, device=DEV)
            od = torch.full((n, md), 9.0, dtype=torch.float16, device=DEV)
            _lib.call("iex_spmm_linear_f16_tile", m, rows_d, k, n, values.numel(), ro.data_ptr(), ci.data_ptr(), bits,
                      values.data_ptr(), dw.data_ptr(), dx.data_ptr(), tokens_major, None, os_.data_ptr(), tokens_major,
                      od.data_ptr(), 1, _stream())
            np.testing.assert_array_equal(os_.cpu().numpy(), ref_s.T if tokens_major else ref_s)
            if rows_d:
                np.testing.assert_array_equal(od.cpu().numpy(), ref_d.T)
    assert _lib.lib.iex_last_device_status(1) == 0


@pytest.mark.parametrize("m0,m1,k,n", [(8, 8, 8, 8), (200, 1000, 264, 64), (5000, 37, 512, 136), (37, 40000, 64, 256)])
def test_linear_pair(m0, m1, k, n):
    w0, w1, x = _ints((m0, k), 1), _ints((m1, k), 2), _ints((k, n), 3, -1, 2)
    o0, o1 = ops.native.linear_pair(_dev(x), _dev(w0), _dev(w1))
    np.testing.assert_array_equal(o0.cpu().numpy(), _exact(w0, x))
    np.testing.assert_array_equal(o1.cpu().numpy(), _exact(w1, x).T)


@pytest.mark.parametrize("n", [64, 128, 256])
@pytest.mark.parametrize("m0,m1,k,index", [(8, 40, 64, torch.int16), (203, 1000, 264, torch.int16), (2500, 37, 512, torch.int32)])
@pytest.mark.parametrize("what", ["a column twice", "descending", "inputs that are not finite"])
def test_sparse_dense_layer_multiplies_what_is_stored(m0, m1, k, n, index, what):
    """The dense copy it keeps has marks for columns that a row stores twice, and zeros that the CSR matrix has not."""
    a, w, x = _ints((m0, k), 1, density=0.6), _ints((m1, k), 2), _ints((k, n), 3, -1, 2)
    values, ri, ro, ci = dense_to_sparse_cuda(_dev(a), index_dtype=index)
    rows = np.repeat(np.arange(m0), np.diff(ro.cpu().numpy()))
    cols = ci.cpu().numpy().astype(np.int64)
    v = values.cpu().numpy().astype(np.float64)
    if what == "a column twice":
        again = np.flatnonzero((np.diff(rows) == 0) & (rows[1:] % 3 == 1))[::5] + 1
        cols[again] = cols[again - 1]
    elif what == "descending":
        order = np.lexsort((-cols, rows))
        cols, v = cols[order], v[order]
    xs = x.astype(np.float64)
    if what == "inputs that are not finite":
        xs[3, 5], xs[k - 1, n - 1], xs[7, 0] = np.inf, np.nan, -np.inf
    ref = np.zeros((m0, n))
    with np.errstate(invalid="ignore"):
        np.add.at(ref, rows, v[:, None] * xs[cols])
        ref_d = (w.astype(np.float64) @ xs).T
    values.copy_(torch.as_tensor(v).half())
    ci.copy_(torch.as_tensor(cols).to(index))
    layer = SparseDenseLayer(values, ri, ro, ci, m0, _dev(w))
    assert layer._dense.current(layer.values, layer.row_offsets, layer.column_indices) is not None
    out, dense = layer(torch.as_tensor(xs).half().to(DEV))
    np.testing.assert_array_equal(out.cpu().numpy().astype(np.float64), ref)  # whole numbers below 2048
    np.testing.assert_array_equal(dense.cpu().numpy().astype(np.float64), ref_d)
    assert _lib.lib.iex_last_device_status(1) == 0


@pytest.mark.parametrize("n", [1, 2, 3, 8, 16])
@pytest.mark.parametrize("m,k,density,index", [(1, 8, 1.0, torch.int16), (300, 1000, 0.3, torch.int16),
                                               (67, 2050, 0.9, torch.int32), (5000, 64, 0.05, torch.int16)])
def test_spmm_few_tokens(n, m, k, density, index):
    a, x = _ints((m, k), m + n, density=density), _ints((k, n), n, -1, 2)
    ref = _exact(a, x)
    values, _ri, ro, ci = dense_to_sparse_cuda(_dev(a), index_dtype=index)
    bits = 16 if index == torch.int16 else 32
    for dx, xr, xc in ((_dev(x), n, 1), (_dev(x.T), 1, k)):
        out = torch.full((m, n), 9.0, dtype=torch.float16, device=DEV)
        _lib.call("iex_spmm_f16_skinny", m, k, n, values.numel(), ro.data_ptr(), ci.data_ptr(), bits, values.data_ptr(),
                  dx.data_ptr(), xr, xc, out.data_ptr(), n, 1, _stream())
        np.testing.assert_array_equal(out.cpu().numpy(), ref)


@pytest.mark.parametrize("m,k,density", [(592, 8, 0.5), (700, 1600, 0.5), (700, 4608, 0.1), (600, 4616, 0.9),
                                         (1500, 33, 0.3), (3, 100, 1.0), (1, 8, 1.0), (200, 6144, 0.05), (200, 6152, 0.05)])
@pytest.mark.parametrize("index", [torch.int16, torch.int32])
def test_csr_expansion_and_sampling(m, k, density, index):
    a = _ints((m, k), m + k, density=density)
    da = _dev(a)
    values, _ri, ro, ci = dense_to_sparse_cuda(da, index_dtype=index)
    bits, ld = 16 if index == torch.int16 else 32, (k + 7) // 8 * 8
    out = torch.full((m, ld), 9.0, dtype=torch.float16, device=DEV)
    _lib.call("iex_csr_to_dense_f16_ld", m, k, ld, ro.data_ptr(), ci.data_ptr(), bits, values.data_ptr(), out.data_ptr(),
              _stream())
    assert torch.equal(out[:, :k], da) and not bool(out[:, k:].any())
    back = torch.empty_like(values)
    _lib.call("iex_csr_sample_f16", m, k, ld, ro.data_ptr(), ci.data_ptr(), bits, out.data_ptr(), back.data_ptr(),
              _stream())
    assert torch.equal(back, values)


def test_dense_copy_follows_the_values():
    a = _ints((64, 64), 5, 1, 3, density=0.5)
    values, _ri, ro, ci = dense_to_sparse_cuda(_dev(a))
    copy = DenseCopy(64, 64)
    assert torch.equal(copy.current(values, ro, ci), _dev(a))
    values.mul_(2)
    assert torch.equal(copy.current(values, ro, ci), _dev(a) * 2)
    sparse = _ints((64, 64), 6, 1, 3, density=0.1)
    values, _ri, ro, ci = dense_to_sparse_cuda(_dev(sparse))
    assert copy.current(values, ro, ci) is None


@pytest.mark.parametrize("count", [1, 255, 1024, 1025, 70001])
@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
def test_gather_values(count, dtype):
    v = torch.randn(count, device=DEV).to(dtype)
    perm = torch.randperm(count, device=DEV)
    out = torch.full((count + 1,), 9.0, dtype=dtype, device=DEV)
    _lib.call("iex_gather_values", count, v.element_size(), v.data_ptr(), perm.data_ptr(), out.data_ptr(), _stream())
    assert torch.equal(out[:-1], v[perm]) and float(out[-1]) == 9.0


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 8, 9])
@pytest.mark.parametrize("m,k,density", [(300, 1000, 0.3), (300, 1000, 0.09), (67, 2050, 0.45), (40, 14001, 0.03), (30, 60000, 0.05),
                                         (900, 192, 0.5), (64, 640, 0.6)])
@pytest.mark.parametrize("index", [torch.int16, torch.int32])
def test_few_columns_take_the_same_sum(n, m, k, density, index):
    """use_tensor_cores="auto" on both sides of the rule for few columns (row length, share stored, shared
    memory), with uneven rows, an empty one and arrays off the alignment of pair loads, against the sums of the
    CUDA cores: one fp16 rounding of fp32 sums in another order."""
    if index == torch.int16 and k > 32767:
        index = torch.int32
    rng = np.random.default_rng(m + k + n)
    a = (rng.standard_normal((m, k)) * 0.1).astype(np.float16) * (rng.random((m, k)) < density)
    a[1], a[2, : k // 2] = 0, 1
    values, ri, ro, ci = dense_to_sparse_cuda(_dev(a), index_dtype=index)
    b = torch.randn(k, n, device=DEV).half()
    terms = torch.as_tensor(np.abs(a.astype(np.float64))).to(DEV) @ b.double().abs()
    ref = torch.ops.iex_ops.spmm_sputnik_reuse_weight_half(b[None], ri, values, ro, ci, m)[0].double()
    shifted = torch.empty(values.numel() + 1, dtype=values.dtype, device=DEV)[1:]
    shifted.copy_(values)
    for v in (values, shifted):
        out = ops.native.myspmm(b, ri, v, ro, ci, m, [], 2)
        assert bool(((out.double() - ref).abs() <= 2.0 ** -10 * ref.abs() + 2e-5 * terms + 2.0 ** -24).all())
