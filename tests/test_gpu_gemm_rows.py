"""Prefill GEMMs around the choice between pair tiles of 256 rows and single tiles of 128: row counts that pad differently,
short and long K, with and without the SiLU * mul epilogue."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [257, 384, 385, 600, 897, 1281, 1300])
@pytest.mark.parametrize("N,K", [(512, 4096), (4096, 1024), (2304, 4096)])
def test_rows(M, N, K):
    from semi_pd_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    w = (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).bfloat16()
    want = x.double() @ w.double().T
    # outputs N(0, 1), at most about 6: one rounding to bf16 (half an ulp of values below 8 is 2^-6) of fp32 sums (1e-4)
    assert (ops.linear(x, w).double() - want).abs().max().item() < 2 ** -6 + 2e-3
    gate, up = want[:, : N // 2].bfloat16().double(), want[:, N // 2:].bfloat16().double()
    got = ops.linear(x, w, epilogue=ops.SPD_EPI_SILU_MUL).double()
    # gate and up are rounded before the product (a sum next to a rounding boundary may fall to the other side: an ulp, 2^-7
    # of it, each) and the product after it (2^-8): of values up to 6 x 6
    assert (got - torch.nn.functional.silu(gate) * up).abs().max().item() < (2 * 2 ** -7 + 2 ** -8) * 36
