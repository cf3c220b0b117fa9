"""Decode GEMMs whose weight rows are long (the down projection over all experts at once): few tiles, each cut along K over
many CTAs or pairs; one workspace for all of them, call after call."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [16384, 16448, 32768, 90112])
@pytest.mark.parametrize("N", [256, 1024, 2048, 4104])
def test_long_rows(N, K):
    from semi_pd_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(N + K)
    w = (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).bfloat16()
    other = torch.randn(512, 8192, generator=g, device="cuda").bfloat16()
    # fp32 sums of K products in steps of 16 that round by 2^-23 of a sum of about 1; four CTAs or more share them
    tol = 2e-5 + K / 64 * 2 ** -23
    for M in (1, 20, 40, 64, 100, 256):
        x = torch.randn(M, K, generator=g, device="cuda").bfloat16()
        want = x.double() @ w.double().T
        first = ops.linear(x, w, out_f32=True, exact_f32=True)
        assert (first.double() - want).abs().max().item() < tol
        half = ops.linear(x, w)
        assert (half.double() - want).abs().max().item() < 2 ** -6 + tol  # half an ulp below 8
        for _ in range(3):  # the flags and partial sums that the calls leave behind
            ops.linear(torch.ones(33, 8192, device="cuda").bfloat16(), other)
            assert torch.equal(ops.linear(x, w, out_f32=True, exact_f32=True), first)
        try:
            for budget in (2, 40, 75):
                ops.set_sm_budget(budget)
                assert (ops.linear(x, w, out_f32=True, exact_f32=True).double() - want).abs().max().item() < 4 * tol  # whole tiles
        finally:
            ops.set_sm_budget(0)
