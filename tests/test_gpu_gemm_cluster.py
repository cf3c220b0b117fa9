"""GEMMs of 17 to 32 tokens on short rows, K cut over a cluster of single CTAs: batches and weights that end inside a tile, uneven
shares of k-blocks, results in 32 bits unrounded (their only form there is not the one of gemm_pair_split.cu)."""
import ctypes

import pytest
import torch

from semi_pd_b200._lib import SPD_EPI_NONE, lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K", [(17, 64, 1024), (32, 4096, 1024), (29, 1000, 1000), (31, 136, 968), (16, 2048, 1024), (33, 2048, 1024)])
def test_exact_results(dtype, M, N, K):
    from semi_pd_b200 import ops
    assert lib.spd_gemm_split_tiles(M, N, K, SPD_EPI_NONE, 2, 0, ctypes.addressof(ctypes.c_int(0))) == 0
    assert (lib.spd_gemm_cluster_ctas(M, N, K, 0) > 0) is (M <= 32)
    g = torch.Generator("cuda").manual_seed(M + N + K)
    x = torch.randn(M, K + 8, generator=g, device="cuda").to(dtype)[:, :K]
    w = (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).to(dtype)
    out = torch.full((M + 1, N + 8), 7.0, device="cuda")
    ops.linear(x, w, out=out[:M, :N], out_f32=True, exact_f32=True)
    y = x.double() @ w.double().t()
    # K exact products summed in fp32 in any order, every sum at most a unit (2^-23) off
    bound = K * 2.0 ** -23 * (x.double().abs() @ w.double().abs().t())
    assert ((out[:M, :N].double() - y).abs() <= bound).all()
    assert (out[M:] == 7).all() and (out[:, N:] == 7).all()
    again = torch.empty(M, N, device="cuda")
    ops.linear(x, w, out=again, out_f32=True, exact_f32=True)
    assert torch.equal(again, out[:M, :N])
