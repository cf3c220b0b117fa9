"""Which GEMMs of few tokens a cluster of single CTAs cuts along K: up to 16 tokens, up to 32 on rows of at most 1024."""
import pytest

from semi_pd_b200._lib import lib


@pytest.mark.parametrize("M,N,K,sms,ctas", [
    (16, 4096, 4096, 148, 128), (17, 4096, 4096, 148, 0), (17, 4096, 1024, 148, 64), (32, 2048, 1024, 76, 32),
    (33, 2048, 1024, 148, 0), (32, 2048, 1032, 148, 0), (32, 6144, 1024, 72, 0), (32, 64, 512, 148, 0), (1, 14336, 4096, 148, 0)])
def test_cluster_ctas(M, N, K, sms, ctas):
    assert lib.spd_gemm_cluster_ctas(M, N, K, sms) == ctas


def test_refuses_bad_sizes():
    assert lib.spd_gemm_cluster_ctas(0, 128, 64, 148) < 0
