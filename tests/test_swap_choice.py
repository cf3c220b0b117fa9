"""Which prefill GEMMs take tiles of 256 weight rows: where they need fewer or shorter waves, on the whole GPU and on partitions."""
import pytest

from semi_pd_b200._lib import SPD_EPI_GELU, SPD_EPI_NONE, SPD_EPI_SILU_MUL, lib


@pytest.mark.parametrize("M,N,K,epilogue,sms,rows", [
    (1300, 14336, 4096, SPD_EPI_SILU_MUL, 148, 192), (1300, 4096, 14336, SPD_EPI_NONE, 148, 160),
    (700, 4096, 14336, SPD_EPI_NONE, 148, 0),        # as many waves of as many columns
    (1600, 14336, 4096, SPD_EPI_SILU_MUL, 148, 256),  # likewise, but 11 % fewer rows over several waves
    (2500, 4096, 14336, SPD_EPI_NONE, 148, 0),       # more waves
    (4096, 4096, 4096, SPD_EPI_NONE, 148, 0), (256, 4096, 4096, SPD_EPI_NONE, 148, 0), (257, 4096, 4096, SPD_EPI_NONE, 148, 96),
    (1300, 4096, 4096, SPD_EPI_GELU, 148, 0), (1300, 4096, 4096, SPD_EPI_NONE, 1, 0), (300, 4096, 4096, SPD_EPI_NONE, 2, 160),
    (1 << 20, 128, 64, SPD_EPI_NONE, 148, 0)])       # more token tiles than a call's list holds
def test_swap_rows(M, N, K, epilogue, sms, rows):
    assert lib.spd_gemm_swap_rows(M, N, K, epilogue, sms) == rows


def test_swap_rows_refuses_bad_sizes():
    assert lib.spd_gemm_swap_rows(0, 128, 64, SPD_EPI_NONE, 148) < 0


@pytest.mark.parametrize("M,N,K,sms", [(1300, 64, 2048, 148), (640, 64, 2048, 72), (640, 3648, 2048, 148), (384, 3648, 2048, 108),
                                       (513, 264, 1024, 148), (800, 1000, 192, 148), (257, 6144, 4096, 72)])
def test_few_tiles_of_128_columns_are_faster(M, N, K, sms):
    assert lib.spd_gemm_swap_rows(M, N, K, SPD_EPI_NONE, sms) == 0
