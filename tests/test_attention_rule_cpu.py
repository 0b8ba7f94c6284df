"""CPU: the choice between one launch over all heads and SDDMM -> SpMM head by head, at masks where both
were measured on B200 (us: one launch, head by head)."""
import pytest

from intrasm_engine_b200 import _lib

# heads, m, n, d, stored share or width of a band, one launch, head by head
MEASURED = [
    (1, 256, 256, 64, 0.002, 15, 47), (32, 1024, 1024, 128, 0.0005, 169, 613), (12, 1000, 3000, 80, 0.002, 121, 257),
    (12, 4096, 4096, 64, 0.02, 211, 265), (24, 4096, 4096, 64, 0.05, 550, 723), (12, 4096, 4096, 80, 0.002, 368, 256),
    (12, 4096, 4096, 80, 0.05, 371, 712), (32, 4096, 4096, 128, 0.02, 2162, 1075), (32, 4096, 4096, 128, 0.1, 2213, 4330),
    (4, 4096, 4096, 128, 0.0005, 249, 112), (1, 8192, 8192, 64, 0.0005, 84, 48), (32, 8192, 8192, 64, 0.002, 2504, 640),
    (12, 8192, 8192, 64, 0.05, 863, 1686), (12, 8192, 8192, 32, 0.0201, 536, 614), (1, 16384, 16384, 64, 32, 275, 49),
    (8, 16384, 16384, 64, 256, 2260, 1425), (8, 16384, 16384, 64, 1024, 2236, 5026), (8, 16384, 16384, 128, 128, 8492, 1308),
    (8, 4096, 4096, 128, 32, 481, 184), (8, 4096, 4096, 64, 1024, 145, 1513)]


@pytest.mark.parametrize("heads,m,n,d,stored,one_launch,head_by_head", MEASURED)
def test_measured_masks(heads, m, n, d, stored, one_launch, head_by_head):
    nnz = int(m * n * stored) if stored < 1 else m * (stored + 1)
    assert bool(_lib.lib.iex_attention_f32_prefers(heads, m, n, d, d, nnz)) == (one_launch < head_by_head)


def test_shapes_the_kernel_does_not_take():
    for shape in ((0, 64, 64, 64, 64), (1, 64, 64, 132, 64), (1, 64, 64, 64, 132), (1, 64, 64, 62, 64)):
        assert not _lib.lib.iex_attention_f32_supported(*shape)
        assert not _lib.lib.iex_attention_f32_prefers(*shape, 1000)


def test_rows_of_q_stay_below_what_a_tma_coordinate_holds():
    """64 x 40 M rows of q would wrap into negative rows, which read as zeros."""
    last = 2 ** 31 - 129
    for heads, m, taken in ((64, 40_000_000, 0), (54, 40_000_000, 0), (53, 40_000_000, 1), (1, last, 1), (1, last + 1, 0), (3, last // 3, 1),
                            (3, last // 3 + 1, 0)):
        assert _lib.lib.iex_attention_f32_supported(heads, m, 128, 4, 4) == taken, (heads, m)
        if not taken:
            assert not _lib.lib.iex_attention_f32_prefers(heads, m, 128, 4, 4, 2 ** 31 - 1)
            assert _lib.lib.iex_attention_workspace_bytes(heads, m, 128, 4, 4) == 0
