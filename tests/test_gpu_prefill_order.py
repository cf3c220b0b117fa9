"""Prefill attention where CTAs get several items: the row tiles are sorted by weight on the device, up to a number of tiles
that shared memory holds; past it they come in the order of their position.  Requests of very unequal length, empty ones
and as many as the list takes, against the kernel on CUDA cores (fp32 sums)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
D = 128


def _args(pre, ext, H, G, dtype):
    g = torch.Generator(device=DEV).manual_seed(sum(ext) + len(ext))
    lens = [p + e for p, e in zip(pre, ext)]
    rtt = torch.zeros(len(ext), max(lens) + 4, dtype=torch.int32)
    at = 1
    for b, n in enumerate(lens):
        rtt[b, :n] = torch.arange(at, at + n)
        at += n
    k, v = (torch.randn(at, G, D, generator=g, device=DEV).to(dtype) for _ in range(2))
    q = torch.randn(sum(ext), H * D, generator=g, device=DEV).to(dtype)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    starts = [sum(ext[:b]) for b in range(len(ext))]
    return (q, k, v, rtt.to(DEV), torch.arange(len(ext), device=DEV), i32(pre), i32(ext), i32(starts), max(ext), H, G, D,
            D ** -0.5)


def _unequal(n, most):
    return [(37 * b * b + 11 * b) % most + 1 for b in range(n)]


# (H, G) = (4, 2): two heads per item; (3, 3): two token tiles per item.  The list holds 768 tiles: tokens / 128 + requests
# (tokens / 256 for two token tiles) decide on the host, so 640 - 900 requests lie on both sides of it.
@pytest.mark.parametrize("H,G", [(4, 2), (3, 3)])
@pytest.mark.parametrize("n,most,prefix", [(3, 2000, 700), (8, 1500, 0), (40, 400, 130), (640, 12, 9), (767, 2, 0), (768, 2, 3),
                                           (900, 5, 1)])
def test_sorted_and_unsorted_items(H, G, n, most, prefix):
    from semi_pd_b200 import ops
    ext = _unequal(n, most)
    if n == 40:
        ext[3] = ext[17] = 0
    pre = [prefix + b if b % 2 else 0 for b in range(n)]
    args = _args(pre, ext, H, G, torch.bfloat16)
    want = ops.attn_prefill(*args, impl="simt").float()
    out = ops.attn_prefill(*args)
    # both round the output to 16 bits (2^-9 of |o| < 5), the tensor-core kernel its probabilities as well
    assert (out.float() - want).abs().max().item() < 3e-2
    try:  # few CTAs: every one walks many items
        ops.set_sm_budget(6)
        assert torch.equal(ops.attn_prefill(*args), out)
    finally:
        ops.set_sm_budget(0)


# up to 384 row tiles the list is made with a tile per thread, past that by compaction; portions of exactly one K / V tile and
# of whole tiles (both warpgroups begin every item together), CTAs with many items of one tile
@pytest.mark.parametrize("H,G", [(4, 2), (3, 3)])
@pytest.mark.parametrize("pre,ext", [([0] * 384, [1, 2, 3] * 128), ([7] * 385, [2] * 385), ([0] * 128, [300] + [0] * 126 + [257]),
                                     ([0] * 130, [260] + [0] * 128 + [1]), ([0] * 64, [128] * 64), ([128, 0] * 20, [128] * 40),
                                     ([0, 256, 0], [384] * 3)])
def test_list_of_tiles(H, G, pre, ext):
    from semi_pd_b200 import ops
    args = _args(pre, ext, H, G, torch.float16)
    want = ops.attn_prefill(*args, impl="simt").float()
    out = ops.attn_prefill(*args)
    # both round the output to 16 bits (2^-12 of |o| < 5), the tensor-core kernel its probabilities as well
    assert (out.float() - want).abs().max().item() < 4e-3
    try:
        ops.set_sm_budget(3)
        assert torch.equal(ops.attn_prefill(*args), out)
    finally:
        ops.set_sm_budget(0)
