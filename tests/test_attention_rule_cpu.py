"""CPU: the choice between one launch over all heads and SDDMM -> SpMM head by head, at masks where both
were measured on B200 (us: one launch, head by head)."""
import random

import pytest

from intrasm_engine_b200 import _lib

# heads, m, n, d, stored share or width of a band, one launch, head by head
MEASURED = [
    (1, 256, 256, 64, 0.002, 17, 51), (32, 1024, 1024, 128, 0.0005, 80, 614), (12, 1000, 3000, 80, 0.002, 62, 258),
    (12, 4096, 4096, 64, 0.02, 139, 269), (24, 4096, 4096, 64, 0.05, 278, 723), (12, 4096, 4096, 80, 0.002, 213, 258),
    (12, 4096, 4096, 80, 0.05, 222, 698), (32, 4096, 4096, 128, 0.02, 785, 780), (32, 4096, 4096, 128, 0.1, 772, 3514),
    (4, 4096, 4096, 128, 0.0005, 88, 113), (1, 8192, 8192, 64, 0.0005, 51, 49), (32, 8192, 8192, 64, 0.002, 1517, 635),
    (12, 8192, 8192, 64, 0.05, 510, 1369), (12, 8192, 8192, 32, 0.0201, 393, 632), (1, 16384, 16384, 64, 32, 162, 50),
    (8, 16384, 16384, 64, 256, 1266, 1056), (8, 16384, 16384, 64, 1024, 1257, 4942), (8, 16384, 16384, 128, 128, 2954, 1175),
    (8, 4096, 4096, 128, 32, 186, 186), (8, 4096, 4096, 64, 1024, 85, 1535), (7, 7176, 7176, 64, 0.0203, 240, 406),
    (1, 6314, 6314, 32, 0.01, 41, 50), (1, 6314, 6314, 32, 0.02, 40, 50), (1, 6314, 6314, 32, 0.04, 40, 64),
    (1, 4096, 4096, 64, 0.002, 27, 48), (1, 4096, 4096, 64, 0.01, 27, 48), (1, 4096, 4096, 128, 0.01, 39, 48),
    (2, 4096, 4096, 128, 0.005, 55, 77), (4, 8192, 8192, 64, 0.002, 166, 118), (4, 8192, 8192, 64, 0.01, 170, 121),
    (4, 8192, 8192, 128, 0.005, 342, 121), (4, 8192, 8192, 128, 0.01, 344, 205), (16, 4096, 4096, 32, 0.002, 143, 341),
    (16, 4096, 4096, 128, 0.005, 371, 329), (16, 4096, 4096, 128, 0.01, 374, 329), (24, 4096, 4096, 128, 0.01, 614, 474),
    (32, 8192, 8192, 64, 0.01, 1590, 829), (32, 8192, 8192, 64, 0.005, 1534, 638), (16, 8192, 8192, 128, 0.01, 1534, 852),
    (2, 16384, 16384, 64, 256, 313, 287), (2, 16384, 16384, 64, 512, 314, 782), (1, 16384, 16384, 64, 512, 164, 452),
    (1, 16384, 16384, 64, 0.01, 172, 102), (1, 12000, 12000, 96, 0.005, 191, 66), (3, 10000, 5000, 48, 0.004, 92, 96),
    (2, 2048, 16384, 64, 0.004, 54, 80), (2, 16384, 2048, 64, 0.004, 53, 80), (1, 2048, 2048, 128, 0.001, 26, 47),
    (1, 3000, 3000, 128, 0.002, 31, 47), (1, 3000, 3000, 32, 0.002, 21, 49)]


@pytest.mark.parametrize("heads,m,n,d,stored,one_launch,head_by_head", MEASURED)
def test_measured_masks(heads, m, n, d, stored, one_launch, head_by_head):
    nnz = int(m * n * stored) if stored < 1 else m * (stored + 1)
    one = bool(_lib.lib.iex_attention_f32_prefers(heads, m, n, d, d, nnz))
    assert one == (one_launch < head_by_head) or max(one_launch, head_by_head) <= 1.03 * min(one_launch, head_by_head)


def test_bits_are_built_for_every_mask_that_some_call_prefers():
    assert _lib.lib.iex_attention_f32_prefers(7, 7176, 7176, 64, 64, int(7176 * 7176 * 0.0203))
    assert _lib.lib.iex_attention_f32_may_prefer(7176, 7176, int(7176 * 7176 * 0.0203))
    rng, missed, preferred, refused = random.Random(5), [], 0, 0
    for _ in range(20000):
        m, n = (int(2 ** rng.uniform(7, 15)) for _ in range(2))
        d, dv = (rng.choice([4, 20, 32, 36, 48, 64, 68, 80, 96, 128]) for _ in range(2))
        heads, nnz = rng.randint(1, 64), int(m * n * 2 ** rng.uniform(-14, -1)) + 1
        one, may = (bool(f) for f in (_lib.lib.iex_attention_f32_prefers(heads, m, n, d, dv, nnz),
                                      _lib.lib.iex_attention_f32_may_prefer(m, n, nnz)))
        preferred, refused = preferred + one, refused + (not may)
        if one and not may:
            missed.append((heads, m, n, d, dv, nnz))
    assert not missed and preferred > 1000 and refused > 1000


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
