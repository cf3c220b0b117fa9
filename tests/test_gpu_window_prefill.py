"""attn_general's tcgen05 prefill (head size 128, window / sinks / query temperature): portions around the 128-query and
128-key tiles, windows that end inside, at and past a tile, rows whose window leaves the tiles of their item, groups of one
head (two token tiles per item) and of several, scattered slots, a sink and scores far from zero."""
import pytest
import torch

from tests.helpers import assert_requests_close

pytestmark = pytest.mark.gpu
DEV = "cuda"
D = 128


def _run(pre, ext, H, G, window, dtype, sinks=None, qtemp=(0.0, 0), scattered=False, shift=0.0, scale=D ** -0.5,
         odd=()):
    from semi_pd_b200 import ops
    g = torch.Generator().manual_seed(sum(ext) + 31 * H + window)
    lens = [p + e for p, e in zip(pre, ext)]
    room = sum(-(-n // 128) * 128 for n in lens) + 129
    k = torch.randn(room, G, D, generator=g)
    k[..., 0] += shift  # with q's first channel at a constant: every score moves by the same large amount
    k, v = k.to(dtype), torch.randn(room, G, D, generator=g).to(dtype)
    rtt = torch.zeros(len(ext), max(lens) + 4, dtype=torch.int32)
    perm, at = torch.randperm(room - 1, generator=g) + 1, 0
    for b, n in enumerate(lens):
        rtt[b, :n] = (perm[at:at + n] if scattered else torch.arange(at, at + n) + 1).int()
        at += n if scattered else -(-n // 128) * 128
    q = torch.randn(sum(ext), H, D, generator=g)
    if shift:
        q[..., 0] = 1.0
    q = q.to(dtype)
    sk = None if sinks is None else torch.linspace(-sinks, sinks, H)
    want, o = [], 0
    for b, (p, e) in enumerate(zip(pre, ext)):
        rows = rtt[b, :p + e].long()
        kk, vv = (x[rows].double().repeat_interleave(H // G, 1) for x in (k, v))
        i = p + torch.arange(e)
        j = torch.arange(p + e)
        s = torch.einsum("qhd,khd->hqk", q[o:o + e].double(), kk) * scale
        if qtemp[1]:
            s = s * (1 + qtemp[0] * torch.log(torch.floor((i.double() + 1) / qtemp[1]) + 1))[None, :, None]
        gone = (j[None] > i[:, None]) | ((i[:, None] - j[None] >= window) if window > 0 else False)
        s = s.masked_fill(gone[None], float("-inf"))
        if sk is not None:
            s = torch.cat((s, sk.double()[:, None, None].expand(-1, e, 1)), -1)
        want.append(torch.einsum("hqk,khd->qhd", torch.softmax(s, -1)[..., : p + e], vv))
        o += e
    want = torch.cat(want).flatten(1)
    blind = torch.ones(want.shape, dtype=torch.bool)  # outputs that meet none of the infinite or NaN values put in below
    for b, pos, head, channel, value in odd:
        v[rtt[b, pos].long(), head, channel] = value
        at, first = sum(ext[:b]), max(0, pos - pre[b])
        last = min(ext[b], pos - pre[b] + window) if window > 0 else ext[b]
        blind.view(-1, H, D)[at + first: at + max(first, last), head * (H // G): (head + 1) * (H // G), channel] = False
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    out = ops.attn_general(q.flatten(1).to(DEV), k.to(DEV), v.to(DEV), rtt.to(DEV), torch.arange(len(ext), device=DEV), H, G,
                           D, D, scale, window=window, sinks=None if sk is None else sk.to(DEV), qtemp_coef=qtemp[0],
                           qtemp_every=qtemp[1], prefix_lens=i32(pre), extend_lens=i32(ext),
                           extend_start_loc=i32([sum(ext[:b]) for b in range(len(ext))]), max_extend_len=max(ext))
    # P and the output are rounded to 16 bits: relative 2^-9 (2^-12) each of values up to |v| ~ 5
    tol = 3e-2 if dtype == torch.bfloat16 else 4e-3
    out = out.cpu().double()
    err = (out - want)[blind].abs().max().item()
    assert err < tol, err
    assert_requests_close(out, want, ext, dtype, blind)
    assert not out[~blind].isfinite().any()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("H,G", [(4, 2), (3, 3), (6, 2), (1, 1)])
@pytest.mark.parametrize("window", [512, 640, 1000, -1])
def test_portions_and_windows(dtype, H, G, window):
    _run([0, 700, 5, 128], [192, 257, 1, 128], H, G, window, dtype, sinks=1.0, qtemp=(0.3, 128))


@pytest.mark.parametrize("window", [1, 2, 63, 64, 65, 127, 128, 129, 300])
@pytest.mark.parametrize("H,G", [(2, 1), (3, 3)])
def test_small_windows(window, H, G):
    _run([3, 0], [1030, 200], H, G, window, torch.bfloat16, sinks=2.0)


@pytest.mark.parametrize("window", [512, 600])
def test_scattered_slots_and_no_options(window):
    _run([333, 0, 1200], [200, 140, 3], 8, 2, window, torch.float16, scattered=True)


@pytest.mark.parametrize("shift", [-60.0, 60.0])
def test_scores_far_from_zero(shift):
    # every score is moved by +-60: rows that see nothing in their item's first units must not start from zero
    _run([700, 0], [260, 9], 4, 2, 512, torch.bfloat16, shift=shift, scale=1.0 / 8)
    _run([0, 4], [1100, 9], 4, 2, 70, torch.bfloat16, shift=shift, scale=1.0 / 8)


def test_large_sinks_and_empty_requests():
    _run([100, 50, 0], [256, 0, 200], 4, 2, 512, torch.bfloat16, sinks=150.0)


@pytest.mark.parametrize("H,G,window", [(4, 2, 512), (3, 3, 130), (4, 2, -1), (2, 1, 1)])
@pytest.mark.parametrize("scattered", [False, True])
def test_values_that_are_not_finite_reach_only_the_rows_that_see_them(H, G, window, scattered):
    # a later token of the same tile, a token that the window has left within it and before it, cached ones
    nan, inf = float("nan"), float("inf")
    odd = [(0, 700, 0, 5, nan), (0, 1024, 0, 100, inf), (1, 333, G - 1, 64, -inf), (1, 1600, G - 1, 0, nan)]
    for dtype in (torch.bfloat16, torch.float16):
        _run([0, 600], [1030, 1100], H, G, window, dtype, sinks=1.0, qtemp=(0.3, 128), scattered=scattered, odd=odd)


def test_negative_scale_and_temperature_keep_their_results():
    # a reference maximum of raw scores does not serve negative factors: these stay on the other kernel
    _run([10, 0], [250, 9], 2, 1, 512, torch.float16, scale=-D ** -0.5)
    _run([10, 0], [250, 9], 2, 1, 512, torch.float16, qtemp=(-0.1, 64))


@pytest.mark.parametrize("ext,window", [(1023, 512), (1024, 512), (1499, 128), (1500, 128)])
def test_a_request_alone(ext, window):
    _run([77], [ext], 4, 2, window, torch.bfloat16, sinks=1.0)


def test_the_sm_budget_bounds_the_grid():
    """With a budget of 4 SMs a call occupies 4: it takes many times as long as on the whole device."""
    from semi_pd_b200 import ops
    H, G, n = 8, 2, 2048
    k, v = (torch.randn(2 * n + 1, G, D, device=DEV).bfloat16() for _ in range(2))
    q = torch.randn(2 * n, H * D, device=DEV).bfloat16()
    rtt = (torch.arange(2 * n, device=DEV, dtype=torch.int32) + 1).view(2, n)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    args = (q, k, v, rtt, torch.arange(2, device=DEV), H, G, D, D, D ** -0.5)
    more = dict(window=1024, prefix_lens=i32([0, 0]), extend_lens=i32([n, n]), extend_start_loc=i32([0, n]), max_extend_len=n)

    def run(budget):
        ops.set_sm_budget(budget)
        try:
            out = ops.attn_general(*args, **more)
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            a.record()
            for _ in range(3):
                ops.attn_general(*args, **more)
            b.record()
            torch.cuda.synchronize()
        finally:
            ops.set_sm_budget(0)
        return out, a.elapsed_time(b)

    (whole, t_whole), (few, t_few) = run(0), run(4)
    assert torch.equal(whole, few)
    assert t_few > 8 * t_whole  # 64 items on 64 CTAs, or 16 rounds on 4


# the three lines of the choice between this kernel and the mma.sync one, a case on each side: portions of 128 tokens, two
# (window below 256) and one block of 64 queries an SM, portions alone that fill less (148 SMs, 8 heads), and 8 tokens a
# request on average
@pytest.mark.parametrize("pre,ext,window", [([900] + [0] * 9, [128] * 10, 512), ([900] + [0] * 9, [129] * 10, 512),
                                            ([40, 0, 0], [770, 770, 667], 128), ([40, 0, 0], [770, 770, 733], 128),
                                            ([300, 0], [192, 927], 300), ([300, 0], [192, 930], 300),
                                            ([300, 0], [192, 930], 255),
                                            ([700], [255], 1024), ([700], [256], 1024), ([700], [256], -1), ([0], [1023], 600),
                                            ([0], [1024], 600), ([0, 9], [5, 191], 600), ([0, 9], [5, 192], 600),
                                            ([0] * 80, [580] + [1] * 58 + [0] * 21, 256),
                                            ([0] * 80, [580] + [1] * 60 + [0] * 19, 256)])
def test_both_sides_of_the_choice_of_kernel(pre, ext, window):
    _run(pre, ext, 8, 2, window, torch.bfloat16, sinks=1.0, qtemp=(0.3, 128))
