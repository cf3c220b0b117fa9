"""moe_align on one CTA and on a cluster of four (more than 2048 entries), shares of one round of reads and of several, experts
without entries, choices outside the experts; moe_dense_act with a token's row cut over blocks."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("T,E,k", [(341, 64, 6), (342, 64, 6), (1366, 7, 3), (5461, 64, 6), (5462, 160, 6), (9000, 33, 8), (2049, 1, 1)])
@pytest.mark.parametrize("outside", [False, True])
def test_rows_by_expert(T, E, k, outside):
    from semi_pd_b200 import ops
    g = torch.Generator().manual_seed(T + E)
    ids = torch.randint(0, max(1, E - E // 4), (T, k), generator=g, dtype=torch.int32)  # the last quarter has no entries
    if outside:
        ids[torch.rand(T, k, generator=g) < 0.1] = E + 3
    row_token, inv_pos, tile_group = (t.cpu().long() for t in ops.moe_align(ids.to(DEV), E))
    flat = ids.view(-1).long()
    inside = flat < E
    assert (inv_pos[~inside] == -1).all()
    pos, expert = inv_pos[inside], flat[inside]
    assert pos.unique().numel() == pos.numel()
    assert torch.equal(row_token[pos], torch.arange(T * k)[inside] // k)
    assert torch.equal(tile_group[pos // 128], expert)
    assert int((row_token >= 0).sum()) == int(inside.sum())
    tiles = -(-torch.bincount(expert, minlength=E) // 128)
    want = torch.repeat_interleave(torch.arange(E), tiles)
    assert torch.equal(tile_group[: want.numel()], want) and (tile_group[want.numel():] == -1).all()


@pytest.mark.parametrize("T,E,k,inter", [(1, 5, 2, 8), (3, 64, 6, 1408), (40, 16, 4, 200), (256, 64, 6, 64), (700, 4, 2, 24)])
def test_dense_act(T, E, k, inter):
    from semi_pd_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(T + inter)
    gu = torch.randn(T, E * 2 * inter, generator=g, device=DEV).bfloat16()
    ids = torch.stack([torch.randperm(E, generator=torch.Generator().manual_seed(t))[:k] for t in range(T)]).int().to(DEV)
    w = torch.rand(T, k, generator=g, device=DEV) + 0.1
    got = ops.moe_dense_act(gu, ids, w, E, inter).view(T, E, inter).float()
    x = gu.view(T, E, 2, inter).float()
    want = torch.nn.functional.silu(x[:, :, 0]) * x[:, :, 1]
    dense = torch.zeros(T, E, device=DEV).scatter_(1, ids.long(), w)
    # the product is rounded to bf16 before and after the weight: 2^-9 each of values up to 5 x 5 x 1.1
    assert (got - want * dense[..., None]).abs().max().item() < 2 * 2 ** -9 * 28
    assert (got[dense == 0] == 0).all()


@pytest.mark.parametrize("T,E,k", [(1, 1, 1), (1, 256, 8), (40, 64, 6), (256, 256, 8), (257, 256, 8), (2048, 3, 1)])
def test_one_cta_keeps_every_entry_in_its_experts_rows(T, E, k):
    """Up to 2048 entries one CTA does it alone, without a cluster (257 x 8: four)."""
    from semi_pd_b200 import ops
    g = torch.Generator().manual_seed(T + E)
    ids = torch.randint(0, E, (T, k), generator=g, dtype=torch.int32)
    for _ in range(3):  # its places come from atomics: any order inside an expert
        row_token, inv_pos, tile_group = (t.cpu().long() for t in ops.moe_align(ids.to(DEV), E))
        assert inv_pos.unique().numel() == T * k
        assert torch.equal(row_token[inv_pos], torch.arange(T * k) // k)
        assert torch.equal(tile_group[inv_pos // 128], ids.view(-1).long())
        assert int((row_token >= 0).sum()) == T * k
