"""GPU: the fp16 head / tail planes of masked attention: every width class at tile and band edges, scales far from one,
tiles that do not suit the planes (summed position by position), rows and columns that are zero or not finite."""
import numpy as np
import pytest
import torch

from intrasm_engine_b200 import _lib, ops
from intrasm_engine_b200.pytorch.attention import SparseAttentionChain
from intrasm_engine_b200.pytorch.utils import dense_to_sparse_cuda

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _case(heads, m, n, d, dv, seed=0, density=0.1):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    mask = torch.rand((m, n), generator=g, device=DEV) < density
    _values, _ri, ro, ci = dense_to_sparse_cuda(mask.to(torch.float16))
    q, k, v = (torch.randn(s, generator=g, device=DEV) for s in ((heads, m, d), (heads, n, d), (heads, n, dv)))
    return mask, SparseAttentionChain(ro, ci, m, n), q, k, v, g


def _run(chain, q, k, v):
    out = ops.native.attention(q, k, v, chain.bits, chain.row_offsets, chain.column_indices)
    torch.cuda.synchronize()
    assert _lib.lib.iex_last_device_status(1) == 0
    return out


def _check(out, mask, q, k, v, bound=2e-6):
    """Per element against fp64.  Heads and tails leave 2^-22 of each of the three factors, a tile's 24 accumulations
    in the tensor core 2^-23 each at most: 2e-6 of the sum of the terms' magnitudes is twice that."""
    zero = torch.zeros((), dtype=torch.float64, device=DEV)
    q, k, v = q.double(), k.double(), v.double()
    ref = torch.where(mask, q @ k.transpose(1, 2), zero) @ v
    terms = torch.where(mask, q.abs() @ k.abs().transpose(1, 2), zero) @ v.abs()
    assert bool(((out.double() - ref).abs() <= bound * terms + 1e-44).all())


@pytest.mark.parametrize("d,dv", [(4, 4), (32, 64), (64, 32), (64, 68), (60, 128), (68, 32), (128, 64), (80, 80), (128, 128)])
@pytest.mark.parametrize("m,n", [(1, 1), (129, 65), (255, 129), (300, 640)])
def test_width_classes_at_tile_edges(d, dv, m, n):
    mask, chain, q, k, v, _g = _case(3, m, n, d, dv, d + dv + m, density=0.3 if m > 1 else 2.0)
    _check(_run(chain, q, k, v), mask, q, k, v)


@pytest.mark.parametrize("d", [64, 96])
@pytest.mark.parametrize("scale", [1e-30, 1e-12, 1e12, 1e18])
def test_scales_far_from_one(d, scale):
    mask, chain, q, k, v, g = _case(2, 200, 300, d, d, 5)
    _check(_run(chain, q * scale, k / scale, v), mask, q * scale, k / scale, v)
    if scale > 1:
        _check(_run(chain, q / scale, k, v * scale), mask, q / scale, k, v * scale)
    rows = torch.exp2(torch.randint(-6, 7, (300, 1), generator=g, device=DEV).float())
    columns = torch.exp2(torch.randint(-6, 7, (d,), generator=g, device=DEV).float())
    q2, k2, v2 = q * columns, k * rows, v * columns / rows
    _check(_run(chain, q2, k2, v2), mask, q2, k2, v2)


@pytest.mark.parametrize("d", [4, 64, 96])
@pytest.mark.parametrize("exponent", [-36, -42, -45, -48])
def test_all_operands_small(d, exponent):
    """The factor of a tile's sums is below fp32's range, the sums are not."""
    mask, chain, q, k, v, _g = _case(2, 200, 300, d, d, 5)
    q, k, v = q * 2.0 ** exponent, k * 2.0 ** exponent, v * 2.0 ** exponent
    out = _run(chain, q, k, v)
    assert bool(out.any())
    _check(out, mask, q, k, v)


@pytest.mark.parametrize("d", [4, 64, 96])
@pytest.mark.parametrize("exponent", [16, 20])
def test_large_sums_beside_a_larger_key(d, exponent):
    """The factor is above fp32's range because of a key that no row stores: rows store one of the others, four features."""
    _mask, _chain, q, k, v, _g = _case(2, 300, 200, d, d, 11)
    rows, keys = (torch.arange(n, device=DEV) for n in (300, 200))
    mask = (keys[None, :] == (7 * rows % 200)[:, None]) & (keys[None, :] != 70)
    _values, _ri, ro, ci = dense_to_sparse_cuda(mask.to(torch.float16))
    chain = SparseAttentionChain(ro, ci, 300, 200)
    q, k, v = (torch.sign(x) * (1 + torch.frac(x.abs())) for x in (q, k, v))
    q[..., 4:], k[..., 4:] = 0, 0
    q, k, v = q * 2.0 ** exponent, k * 2.0 ** exponent, v * 2.0 ** (82 + 40 - 2 * exponent)
    v[:, 70] *= 2.0 ** 28
    out = _run(chain, q, k, v)
    assert bool(torch.isfinite(out).all())
    _check(out, mask, q, k, v)


@pytest.mark.parametrize("d", [64, 96])
@pytest.mark.parametrize("what", ["key of k", "key of v", "column of v"])
def test_tiles_that_do_not_suit_the_planes(d, what):
    mask, chain, q, k, v, _g = _case(2, 300, 200, d, d, 7)
    for exponent in (-20, -32, 40):
        k2, v2 = k.clone(), v.clone()
        if what == "key of k":
            k2[1, 70] *= 2.0 ** exponent
        elif what == "key of v":
            v2[1, 70] *= 2.0 ** exponent
        else:
            v2[1, :, 3] *= 2.0 ** exponent
        out = _run(chain, q, k2, v2)
        _check(out, mask, q, k2, v2)
        assert torch.equal(out[0], _run(chain, q, k, v)[0])


@pytest.mark.parametrize("d", [64, 96])
@pytest.mark.parametrize("what", ["elements", "keys"])
@pytest.mark.parametrize("exponent", [8, 14, 20, 26, 27, 30, 34, 40, 60])
def test_small_elements_of_a_tile_of_v(d, what, exponent):
    """Every other element, or key, of v 2^-exponent times as large, under rows that store one key: nothing else in the sum
    hides what it loses."""
    _mask, _chain, q, k, v, _g = _case(2, 300, 200, d, d, 11)
    rows, keys, columns = (torch.arange(n, device=DEV) for n in (300, 200, d))
    mask = keys[None, :] == (7 * rows % 200)[:, None]
    _values, _ri, ro, ci = dense_to_sparse_cuda(mask.to(torch.float16))
    chain = SparseAttentionChain(ro, ci, 300, 200)
    small = (keys[:, None] + (columns[None, :] if what == "elements" else 0)) % 2 == 1
    v = torch.where(small, v * 2.0 ** -exponent, v)
    _check(_run(chain, q, k, v), mask, q, k, v)


def _unlike(q, k, what, c, column):
    """Features that are large on one side and small on the other, in all rows or some."""
    q, k = q.clone(), k.clone()
    if what == "feature of q":
        q[..., column] *= 2.0 ** c
        k[..., column] *= 2.0 ** -c
    elif what == "feature of k":
        q[..., column] *= 2.0 ** -c
        k[..., column] *= 2.0 ** c
    elif what == "feature off":
        q[..., column] *= 2.0 ** c
        k[..., column] = 0
    elif what == "one row":
        q[1, 77, column] *= 2.0 ** c
        k[..., column] *= 2.0 ** -c
    elif what == "one key":
        q[..., column] *= 2.0 ** -c
        k[0, 33, column] *= 2.0 ** c
    elif what == "every element":  # also disjoint features whose common ones are small on both sides
        g = torch.Generator(device=DEV)
        g.manual_seed(c)
        for x in (q, k):
            x *= torch.exp2(-torch.randint(0, c + 1, x.shape, generator=g, device=DEV).float())
            x *= torch.rand(x.shape, generator=g, device=DEV) < 0.3
    return q, k


@pytest.mark.parametrize("d,column", [(64, 0), (64, 37), (96, 80), (32, 3)])
@pytest.mark.parametrize("what", ["feature of q", "feature of k", "feature off", "one row", "one key", "every element"])
@pytest.mark.parametrize("c", [8, 12, 16, 20, 24, 28, 32, 40, 60])
def test_small_elements_of_a_row_of_q_or_k(d, column, what, c):
    """Rows that are summed by position add up to d / 4 products and 2 sums a score and 45 or so positions of the row:
    2^-24 each, 4e-6 of the terms."""
    mask, chain, q, k, v, _g = _case(2, 300, 200, d, d, 13)
    q, k = _unlike(q, k, what, c, column)
    _check(_run(chain, q, k, v), mask, q, k, v, 4e-6)


@pytest.mark.parametrize("d", [64, 96])
def test_small_elements_with_more_keys_than_are_held_at_a_time(d):
    mask, chain, q, k, v, _g = _case(2, 140, 17000, d, d, 15, density=0.002)
    q[0, :, 9] *= 2.0 ** 30
    k[0, 8000:8400, 9] *= 2.0 ** -30
    k[0, 16990:, 9] = 0
    v[1, 16500, 3] = float("inf")
    out = _run(chain, q, k, v)
    rows = ~mask[:, 16500]
    v[1, 16500] = 0
    _check(out[:1], mask, q[:1], k[:1], v[:1], 4e-6)
    _check(out[1:, rows], mask[rows], q[1:, rows], k[1:], v[1:], 4e-6)
    assert bool(torch.isinf(out[1, ~rows, 3]).all())


@pytest.mark.parametrize("d", [36, 64, 96])
@pytest.mark.parametrize("m,n,density", [(140, 17000, 0.002), (300, 200, 0.1), (1300, 450, 0.1)])
def test_features_that_are_off_in_half_of_the_rows(d, m, n, density):
    """No tile of keys has a column that is large in all of them: their words come with the planes."""
    mask, chain, q, k, v, _g = _case(2, m, n, d, d, 17, density=density)
    q, k = q.relu(), k.relu()
    _check(_run(chain, q, k, v), mask, q, k, v, 4e-6)
    k[0, ::7] = 0
    k[0, 3::7] *= torch.arange(d, device=DEV) % 9 == 0  # little in common
    q[0, 5::11] *= torch.arange(d, device=DEV) % 9 != 0
    q[0, 5::11, 9] = 1e-7  # all that they have
    k[1, n // 2:] = k[1, n // 2:].clamp(min=0.5)  # tiles that are not described beside ones that are
    _check(_run(chain, q, k, v), mask, q, k, v, 4e-6)


def test_small_elements_in_a_band_cut_between_blocks():
    mask, chain, q, k, v, _g = _case(1, 130, 3000, 64, 64, 14, density=0.01)
    q[0, 40, 9] *= 2.0 ** 40
    k[0, 2000:, 9] = 0
    k[0, 2100] = 0
    _check(_run(chain, q, k, v), mask, q, k, v, 4e-6)
    assert torch.equal(_run(chain, q, k, v), _run(chain, q, k, v))


def test_band_cut_between_blocks_that_does_not_suit():
    mask, chain, q, k, v, _g = _case(1, 130, 3000, 64, 64, 8, density=0.05)
    v[0, 2900] = 0
    v[0, 2900, 5] = 1e-30
    v[0, 17] *= 1e20
    _check(_run(chain, q, k, v), mask, q, k, v)


def test_zero_rows_and_values_that_are_not_finite():
    mask, chain, q, k, v, _g = _case(2, 260, 200, 64, 64, 9)
    k[0, 11] = 0
    v[0, 11] = 3e38  # a key that gives nothing
    v[1, 64:128] = 0
    q[1, 5] = 0
    q[0, 9] = 1e-41
    _check(_run(chain, q, k, v), mask, q, k, v)
    clean = _run(chain, q, k, v)
    for value in (float("inf"), float("nan"), torch.finfo(torch.float32).min):
        k2 = k.clone()
        k2[0, 20, 7] = value
        out = _run(chain, q, k2, v)
        seen = mask[:, 20]
        assert torch.allclose(out[0, ~seen], clean[0, ~seen], rtol=1e-5, atol=1e-4) and torch.equal(out[1], clean[1])
        if not np.isfinite(value):
            assert bool((~torch.isfinite(out[0, seen & (q[0, :, 7] != 0)])).all())
    q2 = q.clone()
    q2[0, 33, 1] = float("nan")
    out = _run(chain, q2, k, v)
    others = torch.arange(260, device=DEV) != 33
    assert torch.equal(out[0, others], clean[0, others]) and bool(torch.isnan(out[0, 33]).all() == mask[33].any())
