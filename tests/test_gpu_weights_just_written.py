"""A weight matrix that the kernel right before the GEMM has written, one that lets the GEMM in while it still runs: beyond 256
tokens and with SiLU * mul every form waits for it."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("M,N,K,silu,form", [
    (300, 4096, 4096, False, "swap"), (1300, 6144, 4096, False, "swap"), (400, 4096, 2048, True, "swap"), (448, 4096, 14336, False, "split"),
    (300, 256, 4096, False, "split"), (64, 14336, 512, True, "swap"), (1, 2816, 2048, True, "split"), (200, 2816, 2048, True, "any")])
def test_gemm(M, N, K, silu, form):
    from semi_pd_b200 import ops
    from semi_pd_b200._lib import lib
    epilogue = ops.SPD_EPI_SILU_MUL if silu else ops.SPD_EPI_NONE
    split = ctypes.c_int(0)
    tiles = lib.spd_gemm_split_tiles(M, N, K, epilogue, 0, 0, ctypes.addressof(split))
    assert form == "any" or (form == "split") == (tiles > 0 and split.value > 0)
    assert form != "swap" or M <= 256 or lib.spd_gemm_swap_rows(M, N, K, epilogue, 0) > 0
    g = torch.Generator(device=DEV).manual_seed(M + N)
    rows = N * (1 + silu)
    x = torch.randn(M, K, generator=g, device=DEV).bfloat16()
    src = [(torch.randn(rows, K, generator=g, device=DEV) * K ** -0.5).bfloat16() for _ in range(2)]
    order = torch.randperm(rows, generator=g, device=DEV).int()
    want = [ops.linear(x, s[order.long()].contiguous(), epilogue=epilogue) for s in src]
    for i in range(20):
        w = ops.moe_gather(src[i % 2], order)  # (from the allocator: where the other one was)
        got = ops.linear(x, w, epilogue=epilogue)
        del w
        assert torch.equal(got, want[i % 2])
