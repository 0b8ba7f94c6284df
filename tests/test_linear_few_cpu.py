"""CPU: what the linear layer for any number of tokens refuses, and which way one or two tokens take where there are two."""
import pytest

from intrasm_engine_b200 import _lib, ops


@pytest.mark.parametrize("tokens", [1, 16, 17])
@pytest.mark.parametrize("missing", ["input", "weight", "out", "all"])
def test_operands_that_are_missing(tokens, missing):
    """An error before anything is launched, whichever kernel the sizes would take."""
    at = {name: 0 if missing in (name, "all") else 1 << 20 for name in ("input", "weight", "out")}
    assert _lib.lib.iex_linear_f16_any(tokens, 4096, 4096, at["input"], at["weight"], at["out"], 0) == -1


# tokens, rows, columns, stored share, kernel with the CSR arrays, with the dense copy (us, B200); host time 7.8 and 8.2 us a call
MEASURED = [(1, 512, 512, 0.5, 4.1, 4.0), (1, 1024, 1024, 0.5, 4.2, 4.2), (1, 2048, 1024, 0.5, 4.1, 4.0), (2, 1024, 1024, 0.5, 4.2, 4.1),
            (2, 2048, 1024, 0.3, 4.1, 4.5), (2, 1024, 4096, 0.3, 6.9, 4.7), (1, 4096, 1024, 0.5, 4.2, 4.5), (1, 1024, 4096, 0.5, 5.9, 4.6),
            (1, 4096, 2048, 0.5, 6.7, 4.5), (2, 4096, 2048, 0.3, 9.4, 4.5), (2, 1024, 4096, 0.5, 8.5, 4.6), (1, 4096, 4096, 0.5, 10.3, 5.9),
            (2, 4096, 4096, 0.3, 15.8, 5.6), (1, 11008, 2048, 0.3, 8.8, 6.1), (1, 11008, 4096, 0.5, 23.4, 16.1), (2, 11008, 4096, 0.5, 35.1, 16.3)]


@pytest.mark.parametrize("tokens,rows,columns,stored,csr,copy", MEASURED)
def test_the_faster_way_counts_what_the_host_takes(tokens, rows, columns, stored, csr, copy):
    copy_us = min(_lib.lib.iex_linear_f16_few_estimate_us(tokens, columns, rows, 1), _lib.lib.iex_gemm_f16_estimate_us(rows, tokens, columns, 0, 1))
    assert ops.native.skinny_first(tokens, int(rows * columns * stored), copy_us) == (max(7.8, csr) < max(8.2, copy))
