"""Which GEMMs of few weight tiles a cluster of pairs cuts along K, on the whole GPU and on partitions, and where SiLU * mul goes
into the GEMM."""
import ctypes

import pytest

from semi_pd_b200._lib import SPD_EPI_GELU, SPD_EPI_NONE, SPD_EPI_SILU_MUL, lib


def _form(M, N, K, epilogue=SPD_EPI_NONE, out_f32=0, sms=148):
    split = ctypes.c_int(-1)
    tiles = lib.spd_gemm_split_tiles(M, N, K, epilogue, out_f32, sms, ctypes.addressof(split))
    return tiles, split.value


@pytest.mark.parametrize("M,N,K,form", [
    (32, 4096, 4096, (1, 3)), (1, 4096, 4096, (0, 0)), (16, 4096, 14336, (0, 0)),  # up to 16 tokens: more SMs by single CTAs
    (17, 4096, 14336, (1, 3)), (64, 6144, 4096, (1, 2)), (40, 64, 2048, (2, 4)), (256, 3648, 2048, (2, 0)),
    (64, 28672, 4096, (0, 0)),                                                     # more weight tiles than pairs
    (448, 4096, 14336, (2, 2)), (640, 4096, 4096, (0, 0)), (1024, 4096, 14336, (0, 0))])
def test_form(M, N, K, form):
    assert _form(M, N, K) == form


@pytest.mark.parametrize("sms", [2, 40, 72, 76, 148])
@pytest.mark.parametrize("M", [1, 33, 256, 511])
@pytest.mark.parametrize("N,K", [(64, 64), (2048, 512), (4096, 14336), (16384, 1024)])
def test_clusters_fit(M, N, K, sms):
    tiles, split = _form(M, N, K, sms=sms)
    w_tiles = (N + 255) // 256
    assert 0 <= tiles <= (M + 31) // 32 and 0 <= split <= 4
    if tiles:
        assert (M + tiles - 1) // tiles <= 256 and w_tiles * tiles * max(split, 1) <= sms // 2
        assert split == 0 or 8 * (split - 1) <= K // 64


def test_not_taken():
    assert _form(64, 4096, 4096, sms=1) == (0, 0) and _form(64, 4096, 4096, SPD_EPI_GELU) == (0, 0)
    assert _form(64, 4096, 16448) == (0, 0) and _form(64, 4096, 4096, out_f32=2) == (0, 0)
    assert _form(256, 3648, 2048, out_f32=1)[1] > 0  # the uncut tiles have 16-bit results only
    assert lib.spd_gemm_split_tiles(0, 64, 64, SPD_EPI_NONE, 0, 148, ctypes.addressof(ctypes.c_int(0))) < 0


def test_silu_in_the_gemm():
    assert lib.spd_gemm_silu_fused(300, 14336, 4096, 148) == 1 and lib.spd_gemm_silu_fused(64, 14336, 4096, 148) == 1
    assert lib.spd_gemm_silu_fused(64, 14336, 4096, 72) == 0  # 112 tiles on 36 pairs: four waves, the last nearly empty
    assert lib.spd_gemm_silu_fused(64, 14336, 4096, 76) == 1 and lib.spd_gemm_silu_fused(64, 2816, 2048, 148) == 1
    assert lib.spd_gemm_silu_fused(64, 2816, 2048, 1) == 0 and lib.spd_gemm_silu_fused(0, 8, 8, 148) < 0


def test_room():
    whole = [lib.spd_gemm_split_room(s, -1, 148) for s in (1, 2, 3, 4)]
    assert whole == [74, 33, 22, 15]
    assert [lib.spd_gemm_split_room(s, f, 76) for s, f in ((2, 15), (3, 9), (4, 6))] == [15, 9, 6]  # as the driver says
    assert lib.spd_gemm_split_room(4, 0, 76) == 0 and lib.spd_gemm_split_room(2, 0, 148) == 0       # none fits: none
    assert lib.spd_gemm_split_room(2, 33, 40) == 10                                                 # a budget of fewer SMs
    assert lib.spd_gemm_split_room(0, 5, 148) == 0 and lib.spd_gemm_split_room(5, 5, 148) == 0
    for sms in range(2, 148, 6):
        for s in (1, 2, 3, 4):
            assert 0 <= lib.spd_gemm_split_room(s, -1, sms) <= min(sms // (2 * s), whole[s - 1])


@pytest.mark.parametrize("M,N,K,sms,taken", [
    (1, 4096, 14336, 40, False), (64, 4096, 14336, 40, False), (1, 4096, 14336, 72, False), (256, 4096, 14336, 72, True),
    (1, 6144, 4096, 72, False), (1, 4096, 4096, 40, False), (64, 4096, 4096, 40, True), (64, 2048, 2048, 72, True),
    (64, 64, 2048, 40, True), (512, 4096, 14336, 108, False), (448, 4096, 14336, 148, True)])
def test_partitions_that_stream_k_uses_better(M, N, K, sms, taken):
    assert (_form(M, N, K, sms=sms)[0] > 0) is taken
