"""CPU: the kernel-selection cost model reproduces the measured winners and respects the
tensor-core kernel's shape limits."""
from intrasm_engine_b200 import ops
from intrasm_engine_b200.pytorch import tuning


def test_measured_cases():
    # (m, k, n, sparsity) -> winner measured on B200
    cases = [((2048, 512, 128, 0.70), "tensor_core"), ((512, 2048, 128, 0.95), "cuda_core"),
             ((11008, 4096, 64, 0.50), "tensor_core"), ((512, 512, 256, 0.98), "cuda_core")]
    for (m, k, n, sp), want in cases:
        nnz = int(m * k * (1 - sp))
        assert tuning.choose_spmm_kernel(m, k, n, nnz) == want, (m, k, n, sp)


def test_eager_and_recorded_calls_share_the_model():
    """Where an eager call takes one of the two kernels that a recorded one has, both take the same."""
    ways = set()
    for m, k in ((256, 512), (2048, 512), (512, 2048), (1024, 1024), (4096, 4096), (11008, 4096)):
        for n in (64, 128, 256, 48, 100):
            for sp in (0.5, 0.7, 0.8, 0.9, 0.95, 0.98):
                nnz = int(m * k * (1 - sp))
                eager = ops.native.spmm_half_way(m, k, n, nnz, 16, True)
                recorded = ops.native.spmm_half_way(m, k, n, nnz, 16, False)
                ways.add(eager)
                assert recorded in (0, 1)
                if eager != 2:  # not expanded
                    assert eager == recorded
                assert tuning.choose_spmm_kernel(m, k, n, nnz) == ("tensor_core" if recorded == 1 else "cuda_core")
    assert ways == {0, 1, 2}


def test_few_columns_are_an_eager_way():
    assert ops.native.spmm_half_way(4096, 4096, 4, 1677721, 16, True) == 3
    assert ops.native.spmm_half_way(4096, 4096, 4, 1677721, 16, False) == 0
    assert ops.native.spmm_half_way(4096, 4096, 9, 1677721, 16, True) != 3


def test_shape_limits():
    assert not tuning.tensor_core_supported(512, 48, 16, 16)     # n not a multiple of 64
    assert not tuning.tensor_core_supported(512, 320, 16, 16)    # n too large
    assert not tuning.tensor_core_supported(70000, 64, 16, 16)   # 16-bit indices cannot reach
    assert tuning.tensor_core_supported(70000 - 70000 % 8, 64, 16, 32)
    assert tuning.choose_spmm_kernel(512, 512, 48, 100000) == "cuda_core"
    assert tuning.choose_spmm_kernel(512, 512, 64, 100000, value_bits=32) == "cuda_core"


def test_monotone_in_density():
    prev = "cuda_core"
    for sp in (0.99, 0.95, 0.9, 0.8, 0.5, 0.2):
        nnz = int(4096 * 4096 * (1 - sp))
        cur = tuning.choose_spmm_kernel(4096, 4096, 128, nnz)
        assert not (prev == "tensor_core" and cur == "cuda_core")  # once dense enough, stays
        prev = cur
    assert prev == "tensor_core"
