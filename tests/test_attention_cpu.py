"""CPU: operands of ``SparseAttentionChain`` that do not belong together are refused on the host before
either way of computing the chain is taken."""
import pytest
import torch

from intrasm_engine_b200 import _lib, ops
from intrasm_engine_b200.pytorch.attention import SparseAttentionChain


class _Reached(Exception):
    pass


def _reached(*_args, **_kwargs):
    raise _Reached


def _chain(bits):
    chain = SparseAttentionChain.__new__(SparseAttentionChain)
    chain.m, chain.n, chain.nnz, chain.plan = 8, 12, 4, None
    chain.row_offsets = torch.zeros(9, dtype=torch.int32)
    chain.column_indices = torch.zeros(4, dtype=torch.int32)
    chain.bits = torch.zeros(256, dtype=torch.uint8) if bits else None
    return chain


@pytest.mark.parametrize("bits", [True, False])
@pytest.mark.parametrize("k,v,dtypes", [
    ((3, 12, 16), (1, 12, 16), "fff"),   # one v for three heads
    ((1, 12, 16), (3, 12, 16), "fff"),
    ((3, 12, 8), (3, 12, 16), "fff"),    # k narrower and wider than q
    ((3, 12, 32), (3, 12, 16), "fff"),
    ((3, 11, 16), (3, 12, 16), "fff"),
    ((3, 12, 16), (3, 11, 16), "fff"),
    ((3, 12, 16), (3, 12, 16), "fhf"),   # half the bytes that would be read
    ((3, 12, 16), (3, 12, 16), "ffh")])
def test_mismatched_operands(monkeypatch, bits, k, v, dtypes):
    monkeypatch.setattr(ops.native, "attention", _reached)
    monkeypatch.setattr(_lib, "call", _reached)
    monkeypatch.setattr(torch.cuda, "current_stream", _reached)
    types = [torch.float32 if t == "f" else torch.float16 for t in dtypes]
    q, k, v = (torch.zeros(s, dtype=t) for s, t in zip(((3, 8, 16), k, v), types))
    with pytest.raises(AssertionError):
        _chain(bits)(q, k, v)


def test_matching_operands_pass(monkeypatch):
    monkeypatch.setattr(ops, "native", type("N", (), {"attention": staticmethod(lambda q, *_: q)}))
    q, k, v = torch.zeros(2, 8, 16), torch.zeros(2, 12, 16), torch.zeros(3, 12, 4)
    assert _chain(True)(q, k, v) is q
