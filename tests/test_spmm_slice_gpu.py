"""GPU: CSR SpMM with the dense operand in shared memory (long rows), bit for bit against the oracle at
the edges of its slices, windows and shared-memory limits."""
import numpy as np
import pytest
import torch

from intrasm_engine_b200 import _lib, ops, synthetic as syn  # noqa: F401  (ops registers torch.ops.iex_ops)
from . import gpu_util as G

pytestmark = pytest.mark.gpu

# k: around a TMA box of 64 rows and where 128-, 64- and 32-byte slices stop fitting; n: a column, the widths
# of the slices and one more, rows that are no multiple of 16 bytes
SHAPES = [(1, 3000, 8), (3, 63, 1000), (17, 1537, 1), (64, 64, 33), (65, 65, 32), (96, 1600, 36), (97, 2700, 17),
          (130, 5400, 16), (260, 1280, 128), (300, 700, 137), (640, 400, 64), (1100, 512, 24)]


@pytest.mark.parametrize("m,k,n", SHAPES)
@pytest.mark.parametrize("dtype,idx", [(np.float32, np.int32), (np.float16, np.int16), (np.float16, np.int32)])
def test_slices(oracle, m, k, n, dtype, idx):
    rng = np.random.default_rng(m + k + n)
    # empty, short, full and uneven rows
    row_density = rng.choice([0.0, 0.03, 0.4, 1.0], size=m, p=[0.1, 0.1, 0.7, 0.1])
    row_density[0] = 0.5
    a = syn.csr_from_mask(rng.random((m, k)) < row_density[:, None], rng=rng, std=0.1, dtype=dtype, index_dtype=idx)
    da = G.DevCSR(a)
    run = G.spmm_f32 if dtype == np.float32 else G.spmm_f16
    bias = rng.standard_normal(m).astype(np.float32)
    dense = rng.standard_normal((2, k, n)).astype(dtype)
    for b in (None, bias):
        got = run(da, G.dev(dense), bias=None if b is None else G.dev(b)).cpu().numpy()
        ref = oracle.spmm(a.row_indices, a.values, a.row_offsets, a.column_indices, dense, m, bias=b)
        np.testing.assert_array_equal(got, ref.astype(dtype))
    assert _lib.lib.iex_last_device_status(1) == 0


def test_slices_accumulate_batch_values(oracle):
    """Values of their own for each batch item, added to what is there."""
    rng = np.random.default_rng(3)
    m, k, n, batch = 200, 600, 72, 3
    while True:
        a = syn.csr_from_mask(rng.random((m, k)) < 0.5, rng=rng)
        if a.nnz % 4 == 0:
            break
    vals = rng.standard_normal((batch, a.nnz)).astype(np.float32)
    dense = rng.standard_normal((batch, k, n)).astype(np.float32)
    start = np.ones((batch, m, n), np.float32)
    got = G.spmm_f32(G.DevCSR(a), G.dev(dense), out=G.dev(start), accumulate=True, values=G.dev(vals)).cpu().numpy()
    ref = oracle.spmm(a.row_indices, vals, a.row_offsets, a.column_indices, dense, m, out=start)
    np.testing.assert_array_equal(got, ref)


def test_slices_leave_out_other_rows(oracle):
    """Infinities in rows of the dense operand that a row of A has no nonzero for stay out of its sums."""
    rng = np.random.default_rng(4)
    mask = rng.random((150, 512)) < 0.4
    mask[:, 7] = False
    mask[3, 7] = True
    a = syn.csr_from_mask(mask, rng=rng)
    b = rng.standard_normal((512, 64)).astype(np.float32)
    b[7] = np.inf
    b[0, 5] = np.nan
    got = G.spmm_f32(G.DevCSR(a), G.dev(b)[None])[0].cpu().numpy()
    ref = oracle.spmm(a.row_indices, a.values, a.row_offsets, a.column_indices, b, 150)[0]
    np.testing.assert_array_equal(got, ref)


@pytest.mark.parametrize("dtype,idx,log2_nnz", [(torch.float32, torch.int32, 29), (torch.float16, torch.int16, 30)])
def test_slices_of_two_gigabytes_of_values(dtype, idx, log2_nnz):
    """A little more than 2^31 bytes of values: the bytes behind a nonzero do not fit an int.  Every row is
    full of ones, so that every row of the result is the sum of the dense operand's rows, exactly."""
    k, n = 1024, 3
    m = (1 << log2_nnz) // k + 5
    values = torch.ones(m * k, dtype=dtype, device=G.DEV)
    cols = torch.arange(k, device=G.DEV, dtype=idx).repeat(m)
    offsets = torch.arange(m + 1, device=G.DEV, dtype=torch.int32) * k
    order = torch.arange(m, device=G.DEV, dtype=torch.int32)
    dense = torch.randint(0, 3, (1, k, n), device=G.DEV).to(dtype)
    ref = dense[0].float().sum(0)
    assert float(ref.max()) < 2048
    op = torch.ops.iex_ops.spmm_sputnik_reuse_weight if dtype == torch.float32 else torch.ops.iex_ops.spmm_sputnik_reuse_weight_half
    out = op(dense, order, values, offsets, cols, m)
    assert out.shape == (1, m, n) and torch.equal(out[0].float(), ref.expand(m, n))
    assert _lib.lib.iex_last_device_status(1) == 0
