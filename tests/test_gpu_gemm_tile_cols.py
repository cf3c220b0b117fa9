"""Prefill GEMMs on pair tiles of 256, 224 and 192 columns: shapes for which the rule takes each, with last tiles of all kinds
(a whole one, a few columns, one half of the pair empty), short and long K, 16-bit and 32-bit outputs."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# 148 SMs: 768 x 4096 takes 192 columns (66 tiles in one wave of 74 pairs), 4096 x 3648 takes 224, 2048 x 6144 takes 256
@pytest.mark.parametrize("M,N", [(768, 4096), (768, 4104), (700, 4000), (768, 4224), (4096, 3648), (4000, 3592), (2048, 6144),
                                 (2048, 6080)])
@pytest.mark.parametrize("K", [64, 200, 1024])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_tile_columns(M, N, K, dtype):
    from semi_pd_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    x = torch.randn(M, K, generator=g, device="cuda").to(dtype)
    w = (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).to(dtype)
    want = x.double() @ w.double().T
    # fp32 sums of K products of values up to 5 x 5 K^-0.5; outputs N(0, 1), below 8: half an ulp is 2^-6 (bf16), 2^-9 (fp16)
    assert (ops.linear(x, w, out_f32=True, exact_f32=True).double() - want).abs().max().item() < 1e-4
    assert (ops.linear(x, w).double() - want).abs().max().item() < (2 ** -6 if dtype == torch.bfloat16 else 2 ** -9) + 1e-4
    try:
        ops.set_sm_budget(20)
        assert torch.equal(ops.linear(x, w), ops.linear(x, w))
        assert (ops.linear(x, w).double() - want).abs().max().item() < (2 ** -6 if dtype == torch.bfloat16 else 2 ** -9) + 1e-4
    finally:
        ops.set_sm_budget(0)
