"""MLA decode: few items (their parts are merged by item), full tiles by copies of five lanes beside gathered ones, queries by
one copy per item for any row stride, and a running maximum that may lag."""
import pytest
import torch

from tests.test_gpu_mla_tiles import DEV, DR, R, TOL, _pool, _reference, _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [1, 2, 18, 36, 37, 38])  # up to a quarter of the SMs' number by item
@pytest.mark.parametrize("H", [6, 16, 18])
def test_few_items(batch, H):
    _run([0 if i == 1 else 63 + 131 * ((7 * i + 1) % 10) for i in range(batch)], [1] * batch, H, torch.bfloat16,
         "stray" if batch == 18 else "runs", True)


@pytest.mark.parametrize("keys", [64, 65, 128, 129, 8000, 19000])  # one tile to more parts than SMs take two tiles each
def test_one_long_request(keys):
    _run([keys - 1], [1], 16, torch.float16, "runs", True)


@pytest.mark.parametrize("sms", [1, 3])
def test_many_items_per_cta(sms):
    # full tiles, tails and scattered requests in turn in one CTA's list
    _run([(40, 63, 127, 200, 700)[i % 5] for i in range(60)], [1] * 60, 16, torch.bfloat16, "stray", True, sms=sms)


@pytest.mark.parametrize("step", [0.9, 7.9, 8.1, 40.0])
def test_rising_scores(step):
    # every tile's scores are `step` (log2) above the last one's: the reference lags, or moves with each tile
    from semi_pd_b200 import ops
    g = torch.Generator().manual_seed(5)
    H, n = 16, 64 * 12 + 5
    pool, rtt = _pool([n], torch.float16, "runs", g)
    q = (torch.randn(1, H, R + DR, generator=g) * 0.1).to(torch.float16)
    q[:, :, -1] = 1.0
    scale = 0.0625
    pool[:, -1] = 0
    pool[rtt[0, :n].long(), -1] = ((torch.arange(n) // 64 - 6) * step * 0.6931 / scale).to(torch.float16)
    want = _reference(q, pool, rtt, [n - 1], [1], scale)
    ws = torch.full((ops.lib.spd_attn_mla_workspace_bytes(H, R),), 255, dtype=torch.uint8, device=DEV)
    for sms in (0, 1):
        ops.set_sm_budget(sms)
        try:
            out = ops.attn_mla(q.to(DEV).view(1, -1), pool.to(DEV), rtt.to(DEV), torch.arange(1, device=DEV), H, R, DR, scale,
                               ws, seq_lens=torch.tensor([n], device=DEV), own_workspace=True)
        finally:
            ops.set_sm_budget(0)
        assert (out.cpu().double().view(want.shape) - want).abs().max().item() < TOL[torch.float16]


@pytest.mark.parametrize("stride", [0, 18 * 576, -9216])
def test_query_row_strides(stride):
    from semi_pd_b200 import ops
    from semi_pd_b200._lib import SPD_BF16, check, lib
    g = torch.Generator().manual_seed(6)
    H, lens = 16, [70, 200, 1, 64]
    pool, rtt = _pool(lens, torch.bfloat16, "runs", g)
    rows = (torch.randn(4, 18, R + DR, generator=g) * 0.5).to(torch.bfloat16)
    buf = rows.reshape(-1).to(DEV)
    first = {0: 0, 18 * 576: 0, -9216: 3 * 9216}[stride]
    q = torch.stack([buf.cpu()[first + i * stride: first + i * stride + H * 576] for i in range(4)]).view(4, H, 576)
    want = _reference(q, pool, rtt, [n - 1 for n in lens], [1] * 4, 0.07)
    out = torch.empty(4, H * R, dtype=torch.bfloat16, device=DEV)
    ws = torch.full((ops.lib.spd_attn_mla_workspace_bytes(H, R),), 255, dtype=torch.uint8, device=DEV)
    pool_d, rtt_d, idx, sl = pool.to(DEV), rtt.to(DEV), torch.arange(4, device=DEV), torch.tensor(lens, device=DEV)
    check(lib.spd_attn_mla_own(out.data_ptr(), buf.data_ptr() + 2 * first, pool_d.data_ptr(), rtt_d.data_ptr(), idx.data_ptr(),
                               sl.data_ptr(), None, None, 4, 4, H, R, DR, stride, out.stride(0), rtt_d.stride(0), 0.07,
                               SPD_BF16, ws.data_ptr(), ws.numel(), 0, torch.cuda.current_stream().cuda_stream), "mla")
    assert (out.cpu().double().view(want.shape) - want).abs().max().item() < TOL[torch.bfloat16]


@pytest.mark.parametrize("lens", [[100] * 20, [65, 128, 64, 129] * 9, [1] * 30, [64] * 40, [6080], [6081, 6200], [6150, 1, 12300]])
def test_least_units_per_cta(lens):
    # items of just three units are not cut, very long ones are cut into ranges of four
    _run([n - 1 for n in lens], [1] * len(lens), 16, torch.bfloat16, "runs", True)
