"""Which kernel a call's sizes choose, at the sizes that the GPU tests of those kernels run: the width of a prefill GEMM's tiles
on CTA pairs, and tcgen05 or mma.sync for the windowed prefill attention, on the whole GPU and on a partition."""
import pytest

from semi_pd_b200._lib import SPD_EPI_GELU, SPD_EPI_NONE, SPD_EPI_SILU_MUL, lib


@pytest.mark.parametrize("M,N,cols", [(768, 4096, 192), (768, 4104, 192), (700, 4000, 192), (768, 4224, 192), (4096, 3648, 224),
                                      (4000, 3592, 224), (2048, 6144, 256), (2048, 6080, 256)])
@pytest.mark.parametrize("K", [64, 200, 1024])
def test_pair_tile_columns(M, N, K, cols):
    assert lib.spd_gemm_pair_cols(M, N, K, SPD_EPI_NONE, 148) == cols
    for epilogue in (SPD_EPI_SILU_MUL, SPD_EPI_GELU):
        assert lib.spd_gemm_pair_cols(M, N, K, epilogue, 148) in (0, 256)


def test_single_cta_tiles():
    assert lib.spd_gemm_pair_cols(256, 4096, 4096, SPD_EPI_NONE, 148) == 0   # decode
    assert lib.spd_gemm_pair_cols(600, 3648, 2048, SPD_EPI_NONE, 148) == 0   # a call too short for the rows a pair pads
    assert lib.spd_gemm_pair_cols(4096, 4096, 4096, SPD_EPI_NONE, 1) == 0    # no pair of SMs
    assert lib.spd_gemm_pair_cols(4096, 4096, 4096, SPD_EPI_NONE, 2) == 256


def _tcgen05(ext, window, sms, heads=8, groups=2):
    return lib.spd_attn_general_tcgen05(len(ext), sum(ext), max(ext), heads, groups, window, sms) == 1


# 148 SMs and 40 (the prefixes do not enter)
@pytest.mark.parametrize("ext,window,whole,part", [
    ([128] * 10, 512, False, False), ([129] * 10, 512, True, True),                  # portions of one tile
    ([770, 770, 667], 128, False, True), ([770, 770, 733], 128, True, True),         # two blocks of 64 queries an SM
    ([192, 927], 300, False, True), ([192, 930], 300, True, True),                   # one, from windows of 256 on
    ([192, 930], 255, False, True), ([300, 200], 255, False, False), ([400, 200], 255, False, True),
    ([192, 88], 256, False, True), ([184, 60], 256, False, False),
    ([255], 1024, False, False), ([256], 1024, True, True), ([256], -1, True, True),  # a request alone
    ([1023], 600, False, True), ([1024], 600, True, True), ([5, 191], 600, False, False), ([5, 192], 600, True, True),
    ([580] + [1] * 58 + [0] * 21, 256, False, False), ([580] + [1] * 60 + [0] * 19, 256, True, True)])  # 8 tokens a request
def test_windowed_prefill(ext, window, whole, part):
    assert _tcgen05(ext, window, 148) is whole
    assert _tcgen05(ext, window, 40) is part
