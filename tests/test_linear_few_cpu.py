"""CPU: what the linear layer for any number of tokens refuses."""
import pytest

from intrasm_engine_b200 import _lib


@pytest.mark.parametrize("tokens", [1, 16, 17])
@pytest.mark.parametrize("missing", ["input", "weight", "out", "all"])
def test_operands_that_are_missing(tokens, missing):
    """An error before anything is launched, whichever kernel the sizes would take."""
    at = {name: 0 if missing in (name, "all") else 1 << 20 for name in ("input", "weight", "out")}
    assert _lib.lib.iex_linear_f16_any(tokens, 4096, 4096, at["input"], at["weight"], at["out"], 0) == -1
