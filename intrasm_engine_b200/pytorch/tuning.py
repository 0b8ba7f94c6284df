"""Kernel selection for the fp16 CSR SpMM on B200: CUDA cores or tensor cores.

The reference sketches a tuner that is meant to pick a kernel configuration per layer shape
(intrasm_engine/tuning/my_autograd_func_tuner.py; its build_and_test returns nothing).  Here
the choice is made from estimates fitted to measurements, which stand beside the kernels
(``iex_spmm_f16_estimate_us`` and ``spmm_half_way`` in torch_ext/iex_autograd.cpp); no search at
run time, nothing read back from the device (nnz is the length of the values tensor).

``use_tensor_cores="auto"`` has one model with two sets of ways.  An eager call may also expand
the matrix or take the kernel for few columns.  A call that is recorded into a graph constructor
chooses between the two kernels that need no scratch, with ``choose_spmm_kernel``.
"""
from __future__ import annotations

from .. import ops

TENSOR_CORES = 1  # Way in torch_ext/iex_autograd.cpp


def tensor_core_supported(k: int, n: int, value_bits: int, index_bits: int) -> bool:
    """Shape limits of iex_spmm_f16_tc (column indices must also ascend inside each row, which
    every converter in this package guarantees)."""
    return (value_bits == 16 and index_bits in (16, 32) and n % 64 == 0 and 0 < n <= 256
            and k % 8 == 0 and k > 0 and (index_bits == 32 or k <= 65280))


def choose_spmm_kernel(m: int, k: int, n: int, nnz: int, value_bits: int = 16,
                       index_bits: int = 16) -> str:
    """``"tensor_core"`` or ``"cuda_core"`` for A [m, k] (CSR, nnz stored) times B [k, n]."""
    if not tensor_core_supported(k, n, value_bits, index_bits) or m <= 0:
        return "cuda_core"
    return "tensor_core" if ops.native.spmm_half_way(m, k, n, nnz, index_bits, False) == TENSOR_CORES else "cuda_core"
