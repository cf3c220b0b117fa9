"""MLA prefill with expanded heads (mla_gather + attn_mla_prefill): portions and prefixes around the 64-key, 128-query and
256-query tiles, head counts, consecutive and scattered slots, sorted and unsorted items, scores far from zero, infinite and
NaN keys and values, the rotated queries in place, and the rule that sends a batch here."""
import pytest
import torch

from tests.helpers import assert_requests_close

pytestmark = pytest.mark.gpu
DEV = "cuda"
R, DR, NOPE, DV = 512, 64, 128, 128
# P and the output are rounded to 16 bits (2^-9 / 2^-12 relative); values are N(0, 1), the largest |v| about 5
TOL = {torch.float16: 4e-3, torch.bfloat16: 3e-2}


def _run(pre, ext, H, dtype, scattered=False, budget=0, odd=(), shift=0.0):
    from semi_pd_b200 import ops
    g = torch.Generator().manual_seed(sum(ext) + 7 * sum(pre) + H)
    lens = [p + e for p, e in zip(pre, ext)]
    total = sum(lens)
    rtt = torch.zeros(len(lens) + 1, max(lens) + 3, dtype=torch.int32)
    perm, at = (torch.randperm(total, generator=g) if scattered else torch.arange(total)) + 1, 0
    rpi = torch.randperm(len(lens) + 1, generator=g)[: len(lens)]
    for b, n in enumerate(lens):
        rtt[rpi[b], :n] = perm[at:at + n].int()
        at += n
    pool = torch.randn(total + 1, 1, R + DR, generator=g).to(dtype)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    rows, start = ops.mla_gather(pool.to(DEV), rtt.to(DEV), rpi.to(DEV), i32(pre), i32(ext), total, max(lens), R, DR)
    assert torch.equal(rows.cpu(), pool[perm.long(), 0])
    assert start.tolist() == [sum(lens[:b]) for b in range(len(lens))]
    kv = torch.randn(total, H, NOPE + DV, generator=g)
    kv[..., 0] += shift  # with q's first channel at a constant: every score moves by the same large amount
    q = torch.randn(sum(ext), H * (NOPE + DR) + 40, generator=g)[:, : H * (NOPE + DR)].to(dtype)  # rows of a wider tensor
    if shift:
        q = q.clone()
        q.view(sum(ext), H, NOPE + DR)[..., 0] = 4.0
    kv = kv.to(dtype)
    scale = (NOPE + DR) ** -0.5
    want, at = [], 0
    for b, (p, e) in enumerate(zip(pre, ext)):
        s0 = sum(lens[:b])
        k = torch.cat((kv[s0:s0 + p + e, :, :NOPE], rows.cpu()[s0:s0 + p + e, None, R:].expand(-1, H, -1)), -1).double()
        sc = torch.einsum("qhd,khd->hqk", q.view(-1, H, NOPE + DR)[at:at + e].double(), k) * scale
        sc = sc + torch.full((e, p + e), float("-inf"), dtype=torch.float64).triu(p + 1)
        want.append(torch.einsum("hqk,khd->qhd", sc.softmax(-1), kv[s0:s0 + p + e, :, NOPE:].double()))
        at += e
    want = torch.cat(want)
    blind = torch.ones(want.shape, dtype=torch.bool)  # outputs that meet none of the infinite or NaN values put in below
    for b, pos, head, channel, value in odd:
        kv[sum(lens[:b]) + pos, head, channel] = value
        first = sum(ext[:b]) + max(0, pos - pre[b])
        blind[first: sum(ext[: b + 1]), head, slice(None) if channel < NOPE else channel - NOPE] = False
    dq = torch.zeros(q.shape[0], q.shape[1] + 64, dtype=dtype, device=DEV)
    dq[:, : q.shape[1]] = q.to(DEV)
    ops.set_sm_budget(budget)
    try:
        out = ops.attn_mla_prefill(dq[:, : q.shape[1]], kv.flatten(1).to(DEV), rows, start, i32(pre), i32(ext),
                                   i32([sum(ext[:b]) for b in range(len(ext))]), max(ext), max(lens), H, NOPE, DR, DV, scale)
    finally:
        ops.set_sm_budget(0)
    out = out.cpu().double().view(want.shape)
    err = (out - want)[blind].abs().max().item()
    assert err < TOL[dtype], err
    assert_requests_close(out.flatten(1), want.flatten(1), ext, dtype, blind.flatten(1))
    assert not out[~blind].isfinite().any()
    return out


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("H,scattered", [(16, False), (3, True)])
@pytest.mark.parametrize("pre,ext", [([0], [1]), ([0], [64]), ([0], [65]), ([63], [128]), ([64], [129]), ([1], [256]),
                                     ([0, 127, 0], [257, 1, 384]), ([1000, 0], [3, 700]), ([5, 0, 300, 64], [0, 513, 190, 64])])
def test_tiles(pre, ext, H, scattered, dtype):
    _run(pre, ext, H, dtype, scattered)


@pytest.mark.parametrize("n,most", [(30, 400), (300, 70), (766, 3), (900, 2)])
def test_many_requests(n, most):
    ext = [(37 * b * b + 11 * b) % most + 1 for b in range(n)]
    pre = [9 * (b % 5) for b in range(n)]
    out = _run(pre, ext, 4, torch.bfloat16)
    assert torch.equal(_run(pre, ext, 4, torch.bfloat16, budget=6), out)


@pytest.mark.parametrize("shift", [-60.0, 60.0])
def test_scores_far_from_zero(shift):
    _run([300, 0], [260, 9], 2, torch.bfloat16, shift=shift)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_values_that_are_not_finite_reach_only_the_rows_that_see_them(dtype):
    # a later token of the same tile, one of the next request behind a request's ragged end, a key, cached ones
    nan, inf = float("nan"), float("inf")
    odd = [(0, 700, 0, 5 + NOPE, nan), (0, 1024, 1, 100 + NOPE, inf), (1, 0, 2, 64 + NOPE, -inf), (1, 640, 0, NOPE, nan),
           (1, 900, 1, 7, nan)]
    _run([0, 600], [1030, 500], 3, dtype, odd=odd)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_rotated_queries_in_place(dtype):
    from semi_pd_b200 import ops
    T, H = 77, 5
    g = torch.Generator(device=DEV).manual_seed(3)
    qa = torch.randn(T, H * (NOPE + DR) + R + DR, generator=g, device=DEV).to(dtype)
    w = torch.randn(R, generator=g, device=DEV).to(dtype)
    cs = torch.randn(500, DR, generator=g, device=DEV)
    pos, loc = torch.arange(T, device=DEV) * 3, torch.randperm(T, generator=g, device=DEV) + 1
    pools = [torch.zeros(T + 1, 1, R + DR, device=DEV, dtype=dtype) for _ in range(2)]
    q_lat = torch.zeros(T, H * (R + DR), device=DEV, dtype=dtype)
    ops.mla_rotary_store(qa, q_lat, pools[0], pos, loc, w, cs, H, NOPE, R, DR, 1e-6)
    inplace = qa.clone()
    ops.mla_rotary_store_inplace(inplace, pools[1], pos, loc, w, cs, H, NOPE, R, DR, 1e-6)
    assert torch.equal(pools[0], pools[1])
    heads = lambda t: t[:, : H * (NOPE + DR)].reshape(T, H, NOPE + DR)  # noqa: E731
    assert torch.equal(heads(inplace)[..., NOPE:], q_lat.view(T, H, R + DR)[..., R:])
    assert torch.equal(heads(inplace)[..., :NOPE], heads(qa)[..., :NOPE])
    assert torch.equal(inplace[:, H * (NOPE + DR):], qa[:, H * (NOPE + DR):])


def test_gather_refuses_what_it_would_read_wrongly():
    from semi_pd_b200 import ops
    pool = torch.randn(65, 1, R + DR, device=DEV).bfloat16()
    rtt, idx = torch.arange(64, dtype=torch.int32, device=DEV).view(2, 32), torch.tensor([1, 0], device=DEV)
    lens = torch.tensor([3, 5], dtype=torch.int32, device=DEV)

    def call(rtt=rtt, idx=idx, pre=lens, ext=lens):
        return ops.mla_gather(pool, rtt, idx, pre, ext, 16, 10, R, DR)

    rows, start = call()
    assert start.tolist() == [0, 6] and torch.equal(rows, pool[torch.cat((rtt[1, :6], rtt[0, :10])).long(), 0])
    for wrong in (dict(idx=idx.int()), dict(idx=torch.tensor([[1, 5], [0, 5]], device=DEV)[:, 0]), dict(rtt=rtt.long()),
                  dict(rtt=rtt.T), dict(rtt=rtt.flatten()), dict(pre=lens.long()), dict(ext=lens[:1])):
        with pytest.raises(RuntimeError, match="mla_gather"):
            call(**wrong)
