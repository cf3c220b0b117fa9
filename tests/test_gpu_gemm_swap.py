"""GEMMs whose tiles have 256 weight rows and token rows of any multiple of 32: batches that end inside a 32-row unit and
inside an MMA tile, unequal token tiles, weights that end inside a tile, K that ends inside a block; by expert with counts of
0, 1, one unit, 256 and more, not-a-number in the rows between the experts, buffers that end at the last row."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _check(got, y, dtype, halves=1.0, mean=0.5):
    # fp32 sums of K products of N(0, 1) x N(0, 1 / K); one rounding to 16 bits: 2^-9 (2^-12) of the value at most
    unit = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    assert ((got - y).norm() / y.norm()).item() < unit * mean
    assert ((got - y).abs() <= unit * halves * y.abs() + 1e-4).all()


def _silu_mul(y, dtype):
    # of gate and up as 16-bit numbers, which a sum in another order may round the other way: an ulp (two halves) of up moves
    # the product by as much, one of the gate by up to 1 + |gate| times as much
    gate, up = y.to(dtype).double().chunk(2, 1)
    return torch.nn.functional.silu(gate) * up, 1 + 2 + 2 * (1 + gate.abs())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("silu", [False, True])
@pytest.mark.parametrize("M,N,K", [(257, 2048, 256), (289, 136, 72), (513, 264, 1024), (800, 1000, 192), (1300, 6144, 1096),
                                   (1601, 4096, 1032), (1801, 4360, 1088)])
def test_plain(dtype, silu, M, N, K):
    from semi_pd_b200 import ops
    from semi_pd_b200._lib import lib
    epilogue = ops.SPD_EPI_SILU_MUL if silu else ops.SPD_EPI_NONE
    # (a plain GEMM of few columns has tiles of 128 by single CTAs, which are faster there)
    assert (lib.spd_gemm_swap_rows(M, N, K, epilogue, 148) > 0) is (silu or N not in (136, 264, 1000))
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    x = torch.randn(M, K + 8, generator=g, device=DEV).to(dtype)[:, :K]
    w = (torch.randn(N * (1 + silu), K, generator=g, device=DEV) * K ** -0.5).to(dtype)
    out = torch.full((M + 1, N + 8), 7.0, device=DEV, dtype=dtype)
    ops.linear(x, w, out=out[:M, :N], epilogue=epilogue)
    y, halves, mean = x.double() @ w.double().t(), 1.0, 0.5
    if silu:
        y, halves = _silu_mul(y, dtype)
        mean = 1.0
    _check(out[:M, :N].double(), y, dtype, halves, mean)
    assert (out[M:] == 7).all() and (out[:, N:] == 7).all()  # nothing beside the result


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("layout", ["stacked", "k_concat", "silu"])
@pytest.mark.parametrize("counts,N,K", [([1, 0, 31, 33, 256, 257], 256, 128), ([700], 264, 64), ([0, 0, 5], 136, 448),
                                        ([90] * 40 + [513, 0], 1408, 192), ([0, 0], 128, 64), ([3] * 256, 128, 64)])
def test_by_expert(dtype, layout, counts, N, K):
    from semi_pd_b200 import ops
    E, wide = len(counts), 2 * N if layout == "silu" else N
    starts, rows = [], 0
    for c in counts:
        starts.append(rows)
        rows += (c + 127) // 128 * 128
    last = max((s + c for s, c in zip(starts, counts)), default=0)
    rows = max(last, 1)  # the buffers end with the last expert's rows, not with its tile
    g = torch.Generator(device=DEV).manual_seed(N + K + E)
    x = torch.full((rows, K), float("nan"), device=DEV, dtype=dtype)
    for s, c in zip(starts, counts):
        x[s: s + c] = torch.randn(c, K, generator=g, device=DEV).to(dtype)
    w = (torch.randn(E, wide, K, generator=g, device=DEV) * K ** -0.5).to(dtype)
    flat = w.permute(1, 0, 2).reshape(wide, E * K).contiguous() if layout == "k_concat" else w.view(E * wide, K)
    group_rows = torch.tensor([list(p) for p in zip(starts, counts)], dtype=torch.int32, device=DEV)
    tiles = torch.zeros(1, dtype=torch.int32, device=DEV)
    out = ops.linear_grouped_rows(x, flat, tiles, E, N, k_concat=layout == "k_concat", group_rows=group_rows,
                                  epilogue=ops.SPD_EPI_SILU_MUL if layout == "silu" else 0)
    for e, (s, c) in enumerate(zip(starts, counts)):
        if c == 0:
            continue
        y, halves, mean = x[s: s + c].double() @ w[e].double().t(), 1.0, 0.5
        if layout == "silu":
            y, halves = _silu_mul(y, dtype)
            mean = 1.0
        _check(out[s: s + c].double(), y, dtype, halves, mean)


def test_align_gives_the_rows():
    from semi_pd_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(1)
    for T, E, k in ((40, 64, 6), (600, 7, 4)):  # one CTA, a cluster
        ids = torch.randint(0, E + 1, (T, k), generator=g, device=DEV).int()  # E: a choice outside the experts
        row_token, inv_pos, tile_group, rows = ops.moe_align_groups(ids, E)
        for a, b in zip((inv_pos >= 0, tile_group), (ops.moe_align(ids, E)[1] >= 0, ops.moe_align(ids, E)[2])):
            assert torch.equal(a, b)
        assert torch.equal(rows[:, 1].cpu(), torch.bincount(ids.view(-1), minlength=E + 1)[:E].int().cpu())
        for e, (s, c) in enumerate(rows.cpu().tolist()):
            assert s % 128 == 0 and (row_token[s: s + c] >= 0).all()
            assert c % 128 == 0 or row_token[s + c] == -1
            assert c == 0 or tile_group[s // 128] == e


@pytest.mark.parametrize("sms", [1, 2])
def test_by_expert_on_few_sms(sms):
    from semi_pd_b200 import ops
    E, T, N, K = 5, 150, 136, 64
    g = torch.Generator(device=DEV).manual_seed(2)
    ids = torch.randint(0, E, (T, 2), generator=g, device=DEV).int()
    x = torch.randn(T, K, generator=g, device=DEV).bfloat16()
    w = (torch.randn(E, N, K, generator=g, device=DEV) * K ** -0.5).bfloat16()
    row_token, inv_pos, tile_group, rows = ops.moe_align_groups(ids, E)
    xs = ops.moe_gather(x, row_token)
    ops.set_sm_budget(sms)
    try:
        y = ops.linear_grouped_rows(xs, w.view(E * N, K), tile_group, E, N, group_rows=rows)
    finally:
        ops.set_sm_budget(0)
    got = y[inv_pos.long()].view(T, 2, N).double()
    _check(got, torch.einsum("tjnk,tk->tjn", w[ids.long()].double(), x.double()), torch.bfloat16)
