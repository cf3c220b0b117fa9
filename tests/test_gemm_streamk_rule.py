"""Over how many CTAs a decode GEMM with few tiles cuts its rows: about four contributors per tile, more where the rows are long
and that would leave most of the CTAs idle, not where it would only add partial sums."""
import pytest

from semi_pd_b200._lib import lib


@pytest.mark.parametrize("tiles,kblocks,slots,ctas", [
    (16, 448, 74, 64), (12, 448, 74, 48), (8, 512, 74, 32), (8, 640, 74, 32), (4, 272, 74, 16), (16, 64, 148, 64),  # four per tile
    (16, 224, 148, 64), (28, 64, 148, 112), (1, 20, 148, 4),
    (8, 1408, 74, 74), (8, 1024, 74, 74), (4, 1408, 74, 74), (4, 512, 74, 32), (1, 448, 74, 7), (1, 1408, 74, 22),  # more
    (4, 320, 74, 20), (16, 1408, 148, 148),
    (8, 1408, 36, 32), (4, 1408, 20, 16), (4, 1408, 37, 37), (1, 4, 74, 1), (50, 64, 40, 40), (3, 1, 1, 1),  # partitions, the least
])
def test_rule(tiles, kblocks, slots, ctas):
    assert lib.spd_gemm_streamk_ctas(tiles, kblocks, 4, slots) == ctas


def test_bounds():
    for tiles in range(1, 80, 3):
        for kblocks in list(range(1, 40)) + [64, 100, 255, 256, 257, 384, 448, 512, 1000, 1408, 5000]:
            for slots in (1, 2, 37, 74, 148):
                n = lib.spd_gemm_streamk_ctas(tiles, kblocks, 4, slots)
                assert 1 <= n <= slots
                # a share is 4 k-blocks at least, unless the tiles are fewer than that long
                assert n == 1 or tiles * kblocks // n >= 4
    assert lib.spd_gemm_streamk_ctas(0, 4, 4, 74) < 0 and lib.spd_gemm_streamk_ctas(4, 4, 4, 0) < 0
