"""GEMMs on few weight tiles whose K a cluster of pairs cuts: one to four pairs, one and several token tiles, batches that end
inside a token tile, weights that end inside a tile, uneven shares of k-blocks, rings that wrap and rings that hold a whole
share, 16-bit results and those in 32 bits, SiLU * mul, and the uncut tiles beside one another."""
import ctypes

import pytest
import torch

from semi_pd_b200._lib import SPD_EPI_NONE, SPD_EPI_SILU_MUL, lib

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _form(M, N, K, epilogue, out_f32=0):
    split = ctypes.c_int(0)
    tiles = lib.spd_gemm_split_tiles(M, N, K, epilogue, out_f32, 0, ctypes.addressof(split))
    return tiles, split.value


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K,silu,form", [
    (1, 2048, 2816, False, (1, 4)), (33, 4096, 1032, False, (1, 3)), (64, 64, 2048, False, (2, 4)), (255, 64, 2048, False, (8, 4)),
    (200, 6080, 4096, False, (1, 2)), (40, 12288, 2048, False, (1, 1)), (256, 3648, 2048, False, (2, 0)), (70, 1000, 448, False, None),
    (17, 264, 72, False, None), (300, 256, 4096, False, (10, 4)), (448, 4096, 8192, False, None), (96, 5632, 2048, False, None),
    (1, 2816, 2048, True, (1, 2)), (40, 1000, 4096, True, None), (129, 264, 1032, True, None), (256, 2816, 2048, True, (2, 0)),
    (64, 14336, 512, True, (0, 0)), (8, 136, 8, True, None)])
def test_against_64_bits(dtype, M, N, K, silu, form):
    from semi_pd_b200 import ops
    epilogue = SPD_EPI_SILU_MUL if silu else SPD_EPI_NONE
    if form is not None:
        assert _form(M, N, K, epilogue) == form
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    x = torch.randn(M, K + 8, generator=g, device=DEV).to(dtype)[:, :K]
    w = (torch.randn(N * (1 + silu), K, generator=g, device=DEV) * K ** -0.5).to(dtype)
    out = torch.full((M + 1, N + 8), 7.0, device=DEV, dtype=dtype)
    ops.linear(x, w, out=out[:M, :N], epilogue=epilogue)
    y, halves, mean = x.double() @ w.double().t(), 1.0, 0.5
    if silu:
        # of gate and up as 16-bit numbers, which a sum in another order may round the other way: an ulp (two halves) of up
        # moves the product by as much, one of the gate by up to 1 + |gate| times as much
        gate, up = y.to(dtype).double().chunk(2, 1)
        y, halves, mean = torch.nn.functional.silu(gate) * up, 1 + 2 + 2 * (1 + gate.abs()), 1.0
    # fp32 sums of K products of N(0, 1) x N(0, 1 / K); one rounding to 16 bits: 2^-9 (2^-12) of the value at most
    unit, got = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11, out[:M, :N].double()
    assert ((got - y).norm() / y.norm()).item() < unit * mean
    assert ((got - y).abs() <= unit * halves * y.abs() + 1e-4).all()
    assert (out[M:] == 7).all() and (out[:, N:] == 7).all()  # nothing beside the result
    again = ops.linear(x, w, epilogue=epilogue)
    assert torch.equal(again, out[:M, :N])  # the same sums in the same order
    if not silu and _form(M, N, K, epilogue, 1)[1] == _form(M, N, K, epilogue)[1]:
        assert torch.equal(ops.linear(x, w, out_f32=True), again.float())


def test_a_row_does_not_hang_on_the_others():
    """Infinite and not-a-number tokens stay in their own rows."""
    from semi_pd_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(3)
    for N, K in ((2048, 2816), (64, 2048), (6144, 4096)):
        x = torch.randn(50, K, generator=g, device=DEV).bfloat16()
        w = (torch.randn(N, K, generator=g, device=DEV) * K ** -0.5).bfloat16()
        y = ops.linear(x, w)
        x[7, 3], x[49, K - 1] = float("nan"), float("inf")
        z = ops.linear(x, w)
        keep = [i for i in range(50) if i not in (7, 49)]
        assert torch.equal(y[keep], z[keep]) and torch.isnan(z[7]).all() and not torch.isfinite(z[49]).any()


@pytest.mark.parametrize("M,N,K", [(1, 4096, 14336), (64, 4096, 4096), (256, 1280, 4096), (448, 4096, 2048)])
def test_on_a_partition(M, N, K):
    """Clusters are those that fit the stream's SMs, launched and captured."""
    from semi_pd_b200 import ops
    part = ops.get_partition(0, 76, 72)
    g = torch.Generator(device=DEV).manual_seed(M)
    x = torch.randn(M, K, generator=g, device=DEV).bfloat16()
    w = (torch.randn(N, K, generator=g, device=DEV) * K ** -0.5).bfloat16()
    y = x.double() @ w.double().t()
    torch.cuda.synchronize()
    for stream, sms in ((part.prefill_stream, part.prefill_sms), (part.decode_stream, part.decode_sms)):
        ops.set_sm_budget(sms)
        try:
            with torch.cuda.stream(stream):
                got = ops.linear(x, w)
                stream.synchronize()
                graph, again = torch.cuda.CUDAGraph(), torch.empty_like(got)
                with torch.cuda.graph(graph, stream=stream):
                    ops.linear(x, w, out=again)
                graph.replay()
                stream.synchronize()
        finally:
            ops.set_sm_budget(0)
        assert ((got.double() - y).norm() / y.norm()).item() < 2.0 ** -9  # one rounding to 16 bits
        assert torch.equal(got, again)
