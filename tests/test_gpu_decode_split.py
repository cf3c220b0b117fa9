"""attn_decode's work split: requests cut over several SMs, several requests per SM, one SM for all, ranges that start and
end on and beside tiles, an empty request, more items than the split takes (whole items), a call without a workspace."""
import pytest
import torch

from tests.helpers import assert_requests_close

pytestmark = pytest.mark.gpu
DEV = "cuda"
D = 128


def _run(lens, Hq, Hk, dtype=torch.bfloat16, sms=0, workspace="own", repeat=1):
    """workspace: "own" (zeroed, this stream's alone at every batch size), "shared" (spd_attn_decode_paged, filled with
    something else where the call may not touch it), "none"."""
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
    untouched = workspace == "shared" and B * Hk >= (sms or ops.device_sm_count(0))
    if untouched:
        ws.fill_(255)
    call = _lib.lib.spd_attn_decode_paged_own if workspace == "own" else _lib.lib.spd_attn_decode_paged
    kd, vd, qd, rd = k.to(DEV), v.to(DEV), q.to(DEV), rtt.to(DEV)
    idx, ld = torch.arange(B, device=DEV), torch.tensor(lens, dtype=torch.int64, device=DEV)
    outs = []
    for _ in range(repeat):
        out = torch.zeros_like(qd)
        rc = call(out.data_ptr(), qd.data_ptr(), kd.data_ptr(), vd.data_ptr(), rd.data_ptr(), idx.data_ptr(), ld.data_ptr(),
                  B, Hq, Hk, D, Hq * D, Hq * D, rd.stride(0), float(D ** -0.5), 0 if dtype == torch.bfloat16 else 1,
                  ws.data_ptr() if workspace != "none" else None, ws.numel() if workspace != "none" else 0, sms,
                  ops._stream())
        assert rc == 0, rc
        outs.append(out.cpu())
    # values N(0, 1): the largest output is that of a request of one token; P and the output are rounded to 16 bits
    err = (outs[0].double().view(B, Hq, D) - want).abs().max().item()
    assert err < (3e-2 if dtype == torch.bfloat16 else 4e-3), err
    assert_requests_close(outs[0].view(B, Hq, D), want, [1] * B, dtype)
    if untouched:
        assert bool((ws == 255).all())
    assert all(torch.equal(outs[0], o) for o in outs[1:])  # the parts are merged in a fixed order; counters are re-armed


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("Hq,Hk", [(32, 8), (8, 8), (8, 1), (4, 2)])
@pytest.mark.parametrize("lens", [[1], [5000], [127, 128, 129], [0, 300, 0], [2000, 3, 70, 1], [400 + 37 * i for i in range(12)]])
def test_cuts(Hq, Hk, lens, dtype):
    _run(lens, Hq, Hk, dtype, repeat=3)


@pytest.mark.parametrize("sms", [1, 2, 7, 40])
def test_partitions(sms):
    _run([900, 64, 1300, 256, 5], 16, 4, torch.float16, sms=sms, repeat=2)


def test_many_requests():
    _run([1 + (53 * i) % 700 for i in range(70)], 32, 8)      # 560 items: whole ones
    _run([4000 - 53 * i for i in range(20)], 32, 8)           # 160 items: cut
    _run([1 + (53 * i) % 90 for i in range(300)], 32, 8)      # 2400 items: whole ones


def test_without_a_workspace():
    _run([1 + (53 * i) % 500 for i in range(30)], 32, 8, workspace="none")  # 240 items, whole ones
    _run([300] * 40, 16, 4, workspace="none")


@pytest.mark.parametrize("lens,Hq,Hk,sms", [([1 + (53 * i) % 500 for i in range(30)], 32, 8, 0), ([3000] * 20, 32, 8, 0),
                                            ([900, 64, 1300, 256, 5], 16, 4, 7), ([300, 5000], 16, 4, 0)])
def test_a_shared_workspace(lens, Hq, Hk, sms):
    # as many items as SMs: the workspace may hold anything and belong to another stream; fewer: it is used
    _run(lens, Hq, Hk, workspace="shared", sms=sms, repeat=2)


def test_a_captured_call_keeps_its_results():
    """A call captured without a workspace replays right after a larger batch has replaced the operator's own one, and the
    same graph serves lengths that are cut and lengths that are not."""
    from semi_pd_b200 import ops
    Hq, Hk, B, L = 32, 8, 20, 3000
    g = torch.Generator(device=DEV).manual_seed(5)
    k, v = (torch.randn(B * L + 1, Hk, D, generator=g, device=DEV).bfloat16() for _ in range(2))
    q = torch.randn(B, Hq * D, generator=g, device=DEV).bfloat16()
    rtt = (torch.arange(B * L, device=DEV, dtype=torch.int32) + 1).view(B, L)
    idx, lens = torch.arange(B, device=DEV), torch.full((B,), L, dtype=torch.int64, device=DEV)
    own = torch.zeros(ops.lib.spd_attn_decode_workspace_bytes(B, Hq, D), dtype=torch.uint8, device=DEV)
    args = (k, v, rtt, idx, lens, Hq, Hk, D, D ** -0.5)
    side = torch.cuda.Stream()
    for more in (dict(), dict(workspace=own, own_workspace=True)):
        graph, out = torch.cuda.CUDAGraph(), torch.empty_like(q)
        with torch.cuda.stream(side):
            ops.attn_decode(q, *args, out=out, **more)
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=side):
            ops.attn_decode(q, *args, out=out, **more)
        with torch.cuda.stream(side):  # a larger batch than any before
            many = 40
            ops.attn_decode(q.repeat(many, 1), k, v, rtt.repeat(many, 1), torch.arange(B * many, device=DEV),
                            torch.full((B * many,), 9, dtype=torch.int64, device=DEV), Hq, Hk, D, D ** -0.5)
        torch.cuda.synchronize()
        for n in (L, 40, L, 700):
            lens.fill_(n)
            graph.replay()
            torch.cuda.synchronize()
            want = torch.empty(B, Hq, D, dtype=torch.float64, device=DEV)
            for b in range(B):
                kk, vv = (x[1 + b * L: 1 + b * L + n].double().repeat_interleave(Hq // Hk, 1) for x in (k, v))
                p = torch.softmax(torch.einsum("hd,khd->hk", q[b].double().view(Hq, D), kk) * D ** -0.5, -1)
                want[b] = torch.einsum("hk,khd->hd", p, vv)
            err = ((out.double().view(want.shape) - want).norm() / want.norm()).item()
            assert err < 4e-3, (n, err)
