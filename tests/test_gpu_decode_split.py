"""attn_decode's work split: requests cut over several SMs, several requests per SM, one SM for all, ranges that start and
end on and beside tiles, an empty request, more items than the split takes (whole items), a call without a workspace."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
D = 128


def _run(lens, Hq, Hk, dtype=torch.bfloat16, sms=0, workspace="full", repeat=1):
    from semi_pd_b200 import _lib, ops
    g = torch.Generator().manual_seed(sum(lens) + Hq)
    B = len(lens)
    room = sum(-(-max(n, 1) // 128) * 128 for n in lens) + 1
    k, v = (torch.randn(room, Hk, D, generator=g).to(dtype) for _ in range(2))
    q = torch.randn(B, Hq * D, generator=g).to(dtype)
    rtt = torch.zeros(B, max(lens) + 8, dtype=torch.int32)
    at = 1
    for b, n in enumerate(lens):
        rtt[b, :n] = torch.arange(n) + at
        at += -(-max(n, 1) // 128) * 128
    want = torch.zeros(B, Hq, D, dtype=torch.float64)
    for b, n in enumerate(lens):
        if n:
            rows = rtt[b, :n].long()
            kk, vv = (x[rows].double().repeat_interleave(Hq // Hk, 1) for x in (k, v))
            p = torch.softmax(torch.einsum("hd,khd->hk", q[b].double().view(Hq, D), kk) * D ** -0.5, -1)
            want[b] = torch.einsum("hk,khd->hd", p, vv)
    need = ops.lib.spd_attn_decode_workspace_bytes(B, Hq, D)
    ws = torch.zeros(max(need, 1), dtype=torch.uint8, device=DEV)
    kd, vd, qd, rd = k.to(DEV), v.to(DEV), q.to(DEV), rtt.to(DEV)
    idx, ld = torch.arange(B, device=DEV), torch.tensor(lens, dtype=torch.int64, device=DEV)
    outs = []
    for _ in range(repeat):
        out = torch.empty_like(qd)
        rc = _lib.lib.spd_attn_decode_paged(out.data_ptr(), qd.data_ptr(), kd.data_ptr(), vd.data_ptr(), rd.data_ptr(),
                                            idx.data_ptr(), ld.data_ptr(), B, Hq, Hk, D, Hq * D, Hq * D, rd.stride(0),
                                            float(D ** -0.5), 0 if dtype == torch.bfloat16 else 1,
                                            ws.data_ptr() if workspace == "full" else None,
                                            ws.numel() if workspace == "full" else 0, sms, ops._stream())
        assert rc == 0, rc
        outs.append(out.cpu())
    # values N(0, 1): the largest output is that of a request of one token; P and the output are rounded to 16 bits
    err = (outs[0].double().view(B, Hq, D) - want).abs().max().item()
    assert err < (3e-2 if dtype == torch.bfloat16 else 4e-3), err
    assert all(torch.equal(outs[0], o) for o in outs[1:])  # the parts are merged in a fixed order; counters are re-armed


@pytest.mark.parametrize("Hq,Hk", [(32, 8), (8, 8), (8, 1), (4, 2)])
@pytest.mark.parametrize("lens", [[1], [5000], [127, 128, 129], [0, 300, 0], [2000, 3, 70, 1], [400 + 37 * i for i in range(12)]])
def test_cuts(Hq, Hk, lens):
    _run(lens, Hq, Hk, repeat=3)


@pytest.mark.parametrize("sms", [1, 2, 7, 40])
def test_partitions(sms):
    _run([900, 64, 1300, 256, 5], 16, 4, torch.float16, sms=sms, repeat=2)


def test_many_requests():
    _run([1 + (53 * i) % 700 for i in range(70)], 32, 8)      # 560 items: cut
    _run([1 + (53 * i) % 90 for i in range(300)], 32, 8)      # 2400 items: whole ones


def test_without_a_workspace():
    _run([1 + (53 * i) % 500 for i in range(30)], 32, 8, workspace="none")  # 240 items, whole ones
    _run([300] * 40, 16, 4, workspace="none")
