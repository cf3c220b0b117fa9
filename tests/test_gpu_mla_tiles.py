"""attn_mla on its tile and split edges: consecutive slots (one copy per pair of column blocks) beside scattered ones and
both in one request, lengths around the 64-key tile, requests cut over several SMs or sharing one, head counts that fill
no group of 16, a workspace of the least size a call has to bring, a batch large enough to be cut at request starts."""
import pytest
import torch

from tests.helpers import assert_requests_close

pytestmark = pytest.mark.gpu
DEV = "cuda"
R, DR = 512, 64


def _pool(lens, dtype, layout, g):
    """Latent rows and a page table: "runs" of 128 consecutive slots (the pool's allocator), "scattered", or runs with a
    stray slot in every third tile."""
    room = sum(-(-n // 128) * 128 for n in lens) + 200
    pool = (torch.randn(room, R + DR, generator=g) * 0.5).to(dtype)
    rtt = torch.zeros(len(lens), max(max(lens), 1) + 8, dtype=torch.int32)
    if layout == "scattered":
        perm, at = torch.randperm(room - 1, generator=g) + 1, 0
        for b, n in enumerate(lens):
            rtt[b, :n] = perm[at:at + n].int()
            at += n
        return pool, rtt
    order = torch.randperm(sum(-(-n // 128) for n in lens), generator=g).tolist()
    for b, n in enumerate(lens):
        for i in range(0, n, 128):
            k = min(128, n - i)
            rtt[b, i:i + k] = torch.arange(k, dtype=torch.int32) + 1 + 128 * order.pop()
        if layout == "stray":
            for i in range(70, n, 192):
                rtt[b, i] = room - 1 - (i % 50)
    return pool, rtt


def _reference(q, pool, rtt, pre, ext, scale):
    out, at = [], 0
    for b, (p, e) in enumerate(zip(pre, ext)):
        rows = pool[rtt[b, :p + e].long()].double()
        sc = torch.einsum("qhl,kl->hqk", q[at:at + e].double(), rows) * scale
        sc = sc + torch.full((e, p + e), float("-inf"), dtype=torch.float64).triu(p + 1)
        out.append(torch.einsum("hqk,kr->qhr", sc.softmax(-1), rows[:, :R]))
        at += e
    return torch.cat(out)


# probabilities and outputs are rounded to 16 bits (2^-9 / 2^-12 relative); values are N(0, 0.25) averaged over the keys, so
# the largest of them is that of a request of one key, |v| <= 2.5: half an ulp of the output plus the same for P
TOL = {torch.float16: 2e-3, torch.bfloat16: 1.6e-2}


def _run(pre, ext, H, dtype, layout, decode, ws_bytes=None, sms=0, odd=(), own=True):
    from semi_pd_b200 import ops
    g = torch.Generator().manual_seed(sum(ext) + 7 * sum(pre) + H)
    lens = [p + e for p, e in zip(pre, ext)]
    pool, rtt = _pool(lens, dtype, layout, g)
    q = (torch.randn(sum(ext), H, R + DR, generator=g) * 0.5).to(dtype)
    scale = 192 ** -0.5
    want = _reference(q, pool, rtt, pre, ext, scale)
    blind = torch.ones(len(q), dtype=torch.bool)  # query rows that see none of the infinite or NaN values put in below
    for b, pos, channel, value in odd:
        pool[rtt[b, pos].long(), channel] = value
        at = sum(ext[:b])
        blind[at + max(0, pos - pre[b]): at + ext[b]] = False
    need = ops.lib.spd_attn_mla_workspace_bytes(H, R) if ws_bytes is None else ws_bytes
    ws = torch.full((need,), 255, dtype=torch.uint8, device=DEV)  # (not zeroed: NaN patterns)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    if decode:
        more = dict(seq_lens=torch.tensor(lens, dtype=torch.int64, device=DEV))
    else:
        starts = [sum(ext[:i]) for i in range(len(ext))]
        more = dict(prefix_lens=i32(pre), extend_start_loc=i32(starts))
    ops.set_sm_budget(sms)
    try:
        out = ops.attn_mla(q.to(DEV).view(q.shape[0], -1), pool.to(DEV), rtt.to(DEV), torch.arange(len(ext), device=DEV), H,
                           R, DR, scale, ws, own_workspace=own, **more)
    finally:
        ops.set_sm_budget(0)
    if not own and q.shape[0] * -(-H // 16) >= 2 * (sms or ops.device_sm_count(0)):
        assert bool((ws == 255).all())  # another stream may be using it
    out = out.cpu().double().view(want.shape)
    err = (out - want)[blind].abs().max().item()
    assert err < TOL[dtype], err
    assert_requests_close(out, want, ext, dtype, blind)
    for b, pos, channel, value in odd:
        at = sum(ext[:b])
        assert not out[at + max(0, pos - pre[b]): at + ext[b], :, channel].isfinite().any()


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("layout", ["runs", "scattered", "stray"])
@pytest.mark.parametrize("lens", [[63], [64], [65], [128, 129, 1, 191, 640], [5000], [2000] * 3 + [3] * 40])
def test_decode_tiles(dtype, layout, lens):
    _run([n - 1 for n in lens], [1] * len(lens), 16, dtype, layout, True)


@pytest.mark.parametrize("H", [1, 5, 20, 48])
@pytest.mark.parametrize("decode", [True, False])
def test_head_counts(H, decode):
    ext = [1, 1, 1] if decode else [9, 1, 70]
    _run([300, 64, 700], ext, H, torch.bfloat16, "runs", decode)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("layout", ["runs", "scattered", "stray"])
@pytest.mark.parametrize("pre,ext", [([0], [3]), ([0], [64]), ([61], [7]), ([0, 130, 5], [1, 65, 4]), ([2000], [2]),
                                     ([0, 640], [700, 259])])
def test_extend_tiles(layout, pre, ext, dtype):
    _run(pre, ext, 16, dtype, layout, False)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("layout", ["runs", "scattered"])
@pytest.mark.parametrize("pre,ext,odd", [
    ([0], [64], [(0, 63, 5, float("nan"))]),                       # the last row of a full tile
    ([100], [130], [(0, 150, 511, float("inf")), (0, 229, 0, float("-inf"))]),
    ([0, 500], [70, 66], [(0, 2, 17, float("inf")), (1, 502, 3, float("nan"))]),   # inside a group of four tokens
    ([1500], [6], [(0, 1504, 100, float("nan"))]),                 # items cut over several SMs
    ([0, 3], [700, 300], [(0, 640, 1, float("inf")), (1, 200, 2, float("nan"))]),  # whole items
])
def test_values_that_are_not_finite_reach_no_earlier_token(dtype, layout, pre, ext, odd):
    _run(pre, ext, 16, dtype, layout, False, odd=odd)
    _run(pre, ext, 5, dtype, layout, False, odd=odd, sms=2)


def test_empty_requests_in_an_extend_batch():
    _run([0, 40, 0, 10, 3], [0, 9, 0, 70, 0], 16, torch.float16, "runs", False)


def test_small_partition_and_request_starts():
    # 40 requests on 2 SMs: 20 per SM, cut at request starts; on 8 SMs the ranges cut requests
    for sms in (2, 8):
        _run([50 + 9 * i for i in range(40)], [1] * 40, 16, torch.bfloat16, "runs", True, sms=sms)


def test_a_shared_workspace():
    _run([0, 640], [700, 259], 16, torch.float16, "runs", False, own=False)
    _run([50 + 9 * i for i in range(40)], [1] * 40, 16, torch.bfloat16, "runs", True, sms=8, own=False)
    _run([300, 64], [40, 5], 16, torch.bfloat16, "runs", False, own=False)  # too small to go without it


@pytest.mark.parametrize("decode", [True, False])
def test_least_workspace(decode):
    # items x heads x splits x 514 floats is what a call has to bring; nothing is split over SMs then
    H, ext = 16, [1, 1] if decode else [5, 2]
    least = sum(ext) * H * 8 * 514 * 4
    _run([200, 100], ext, H, torch.bfloat16, "runs", decode, ws_bytes=least)
    with pytest.raises(RuntimeError):
        _run([200, 100], ext, H, torch.bfloat16, "runs", decode, ws_bytes=least - 4)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("T,H", [(1, 16), (3, 1), (130, 5), (7, 32)])
def test_rotary_store(dtype, T, H):
    from semi_pd_b200 import ops
    g = torch.Generator().manual_seed(T + H)
    nope = 128
    qa = torch.randn(T, H * (nope + DR) + R + DR + 8, generator=g).to(dtype)[:, : H * (nope + DR) + R + DR]
    w = (1 + 0.1 * torch.randn(R, generator=g)).to(dtype)
    ang = torch.rand(500, DR // 2, generator=g) * 6
    table = torch.cat((ang.cos(), ang.sin()), 1)
    pos, loc = torch.randint(0, 500, (T,), generator=g), torch.randperm(T + 20, generator=g)[:T]
    q_lat = torch.zeros(T, H * (R + DR), dtype=dtype, device=DEV)
    pool = torch.zeros(T + 20, 1, R + DR, dtype=dtype, device=DEV)
    whole = torch.empty(T, qa.shape[1] + 8, dtype=dtype, device=DEV)
    d_qa = whole[:, : qa.shape[1]]
    d_qa.copy_(qa)
    ops.mla_rotary_store(d_qa, q_lat, pool, pos.to(DEV), loc.to(DEV), w.to(DEV), table.to(DEV), H, nope, R, DR, 1e-6)
    c, s = table[pos].double()[:, None, : DR // 2], table[pos].double()[:, None, DR // 2:]

    def rot(x):  # interleaved pairs
        a, b = x.double()[..., 0::2], x.double()[..., 1::2]
        return torch.stack((a * c - b * s, b * c + a * s), -1).flatten(-2)

    x = qa[:, H * (nope + DR): H * (nope + DR) + R].double()
    want = torch.zeros(T + 20, R + DR, dtype=torch.float64)
    want[loc, :R] = x / (x.square().mean(-1, keepdim=True) + 1e-6).sqrt() * w.double()
    want[loc, R:] = rot(qa[:, None, H * (nope + DR) + R:])[:, 0]
    q_want = torch.zeros(T, H, R + DR, dtype=torch.float64)
    q_want[..., R:] = rot(qa[:, : H * (nope + DR)].view(T, H, nope + DR)[..., nope:])
    # one rounding to 16 bits of fp32 results of at most about 8
    tol = 2 ** -11 * 8 + 1e-5 if dtype == torch.float16 else 2 ** -8 * 8 + 1e-5
    assert (pool.cpu().double()[:, 0] - want).abs().max().item() < tol
    assert (q_lat.cpu().double().view(T, H, -1) - q_want).abs().max().item() < tol


def test_rotary_store_refuses_what_it_would_read_past():
    from semi_pd_b200 import ops
    H, nope, T = 2, 128, 5
    good = dict(qa=torch.zeros(T, H * (nope + DR) + R + DR), q_lat=torch.zeros(T, H * (R + DR)), pool=torch.zeros(9, 1, R + DR),
                pos=torch.zeros(T, dtype=torch.int64), loc=torch.arange(T), w=torch.ones(R), table=torch.zeros(4, DR))
    bad = [dict(qa=torch.zeros(T, H * (nope + DR) + R)), dict(qa=torch.zeros(H * (nope + DR) + R + DR, T).t()),
           dict(q_lat=torch.zeros(T - 1, H * (R + DR))), dict(q_lat=torch.zeros(T, H * R)),
           dict(q_lat=torch.zeros(H * (R + DR), T).t()), dict(pool=torch.zeros(9, 1, R)),
           dict(pool=torch.zeros(9, 1, 2 * (R + DR))[..., : R + DR]), dict(pos=torch.zeros(T - 1, dtype=torch.int64)),
           dict(pos=torch.zeros(2 * T, dtype=torch.int64)[::2]), dict(loc=torch.arange(T + 1)),
           dict(loc=torch.arange(2 * T)[::2]), dict(w=torch.ones(R - 8)), dict(w=torch.ones(2 * R)[::2]),
           dict(table=torch.zeros(4, DR // 2)), dict(table=torch.zeros(4, 2 * DR)[:, :DR])]

    def call(a):
        d = {}
        for n, t in a.items():  # (the layout of the CPU tensor: .to keeps only dense strides)
            dt = t.dtype if t.dtype == torch.int64 or n == "table" else torch.float16
            d[n] = torch.empty(t.untyped_storage().nbytes() // t.element_size(), dtype=dt, device=DEV).as_strided(
                t.shape, t.stride()).copy_(t)
        ops.mla_rotary_store(d["qa"], d["q_lat"], d["pool"], d["pos"], d["loc"], d["w"], d["table"], H, nope, R, DR, 1e-6)

    call(good)
    for i, b in enumerate(bad):
        try:
            call({**good, **b})
        except RuntimeError as e:
            assert "mla_rotary_store" in str(e), (i, e)
        else:
            raise AssertionError(f"case {i} was accepted")
    torch.cuda.synchronize()


def test_a_wait_that_ran_out_is_reported():
    """A kernel whose bounded wait runs out ends, sets the status word, and the calls with such waits refuse from then on."""
    import ctypes

    from semi_pd_b200 import _lib, ops
    torch.cuda.synchronize()
    ops.check_waits()
    n = ctypes.c_int()
    try:
        assert _lib.lib.spd_wait_selftest(2, ops._stream()) == 0
        torch.cuda.synchronize()
        with pytest.raises(RuntimeError, match="ran out"):
            ops.check_waits()
        with pytest.raises(RuntimeError, match="ran out"):
            _run([63], [1], 16, torch.bfloat16, "runs", True)
    finally:
        torch.cuda.synchronize()
        assert _lib.lib.spd_wait_status(ctypes.byref(n), 1) == 0
    assert n.value == 1
    ops.check_waits()
    _run([63], [1], 16, torch.bfloat16, "runs", True)
