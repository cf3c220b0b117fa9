"""Grouped expert GEMMs over sorted rows: enough row tiles for 128 x 256 tiles beside too few, experts stacked along the rows
and concatenated along K, column counts that end inside a tile, several panels of column tiles with a short last one,
experts of one and of several row tiles, unused row tiles at the end."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _groups(E, tiles, unused):
    """Expert of each row tile, ascending: unequal shares of `tiles`, then unused tiles."""
    cut = sorted((i * i * tiles) // (E * E) for i in range(1, E))
    edges = [0] + cut + [tiles]
    ids = [e for e in range(E) for _ in range(edges[e + 1] - edges[e])]
    return torch.tensor(ids + [-1] * unused, dtype=torch.int32)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("layout", ["stacked", "k_concat", "silu"])
@pytest.mark.parametrize("E,tiles,N,K", [
    (4, 19, 2048, 512),    # 19 x 8 tiles of 256 columns: just enough
    (4, 18, 2048, 512),    # just too few
    (5, 40, 1152, 256),    # the last tile of 256 columns half empty
    (3, 40, 1160, 128),    # and with 8 columns more
    (2, 14, 2816, 8192),   # two panels, the second of one tile
    (2, 8, 1032, 16384),   # K of 256 blocks
])
def test_rows_by_expert(dtype, layout, E, tiles, N, K):
    from semi_pd_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(N + K + tiles)
    ids = _groups(E, tiles, 3)
    wide = 2 * N if layout == "silu" else N
    x = torch.randn(ids.numel() * 128, K, generator=g, device=DEV).to(dtype)
    w = (torch.randn(E, wide, K, generator=g, device=DEV) * K ** -0.5).to(dtype)
    flat = w.permute(1, 0, 2).reshape(wide, E * K).contiguous() if layout == "k_concat" else w.view(E * wide, K)
    out = ops.linear_grouped_rows(x, flat, ids.to(DEV), E, N, k_concat=layout == "k_concat",
                                  epilogue=ops.SPD_EPI_SILU_MUL if layout == "silu" else 0)
    for e in range(E):
        rows = (ids == e).nonzero().view(-1)
        if not rows.numel():
            continue
        lo, hi = int(rows[0]) * 128, (int(rows[-1]) + 1) * 128
        y = x[lo:hi].double() @ w[e].double().t()
        halves, mean = 1.0, 0.5  # half ulps that an element and the norm may be off
        if layout == "silu":
            # of gate and up as 16-bit numbers, which a sum in another order may round the other way: an ulp (two halves) of
            # up moves the product by as much, one of the gate by up to 1 + |gate| times as much
            gate, up = y.to(dtype).double().split(N, 1)
            y = torch.nn.functional.silu(gate) * up
            halves, mean = 1 + 2 + 2 * (1 + gate.abs()), 1.0
        got = out[lo:hi].double()
        # fp32 sums of K products of N(0, 1) x N(0, 1 / K); one rounding to 16 bits: 2^-9 (2^-12) of the value at most
        unit = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
        assert ((got - y).norm() / y.norm()).item() < unit * mean
        assert ((got - y).abs() <= unit * halves * y.abs() + 1e-4).all()
