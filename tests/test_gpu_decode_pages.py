"""Decode attention over page tables that are runs but for single entries: the copy of a whole tile or the gather of its rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("stray", [(), (0,), (31,), (32,), (95,), (127,), (128,), (255, 256), (511,), tuple(range(0, 640, 97))])
@pytest.mark.parametrize("lens", [[640, 127, 128, 129, 1], [640] * 40])
def test_runs_with_stray_entries(dtype, stray, lens):
    from semi_pd_b200 import ops
    g = torch.Generator().manual_seed(len(lens) + sum(stray))
    B, Hq, Hk, D = len(lens), 8, 2, 128
    room = sum(lens) + 700
    k = torch.randn(room, Hk, D, generator=g).to(dtype)
    v = torch.randn(room, Hk, D, generator=g).to(dtype)
    q = torch.randn(B, Hq * D, generator=g).to(dtype)
    rtt = torch.zeros(B, 648, dtype=torch.int32)
    at = 1
    for b, n in enumerate(lens):
        rtt[b, :n] = torch.arange(at, at + n)
        at += n
        for i in stray:
            if i < n:
                rtt[b, i] = room - 1 - i
    want = torch.empty(B, Hq, D, dtype=torch.float64)
    for b, n in enumerate(lens):
        rows = rtt[b, :n].long()
        kk, vv = (t[rows].double().repeat_interleave(Hq // Hk, 1) for t in (k, v))
        p = torch.einsum("hd,nhd->hn", q[b].double().view(Hq, D), kk).mul(D ** -0.5).softmax(-1)
        want[b] = torch.einsum("hn,nhd->hd", p, vv)
    out = ops.attn_decode(q.to(DEV), k.to(DEV), v.to(DEV), rtt.to(DEV), torch.arange(B, device=DEV),
                          torch.tensor(lens, device=DEV), Hq, Hk, D, D ** -0.5)
    # P and the output are rounded to 16 bits, values are at most about 4.5 (one key): half an ulp of each
    tol = 4.5 * (2 ** -8 if dtype == torch.bfloat16 else 2 ** -11)
    assert (out.cpu().double().view_as(want) - want).abs().max().item() < tol
