"""Rotation and cache write at the sizes where a block has a thread for each piece of a token, and where it has not."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens", [1, 3, 444, 445])
@pytest.mark.parametrize("heads", [(32, 8, 128, 128), (1, 1, 64, 32), (2, 1, 128, 64), (40, 40, 128, 128), (64, 8, 64, 64)])
@pytest.mark.parametrize("neox", [True, False])
def test_rope_kvwrite(tokens, heads, neox):
    from semi_pd_b200 import ops
    Hq, Hk, D, rot = heads
    g = torch.Generator().manual_seed(tokens + Hq)
    qkv = torch.randn(tokens, (Hq + 2 * Hk) * D, generator=g).bfloat16()
    cs = torch.randn(512, rot, generator=g)
    pos = torch.randint(0, 512, (tokens,), generator=g)
    loc = torch.randperm(tokens + 5, generator=g)[:tokens]
    q, k, v = qkv.double().split([Hq * D, Hk * D, Hk * D], -1)
    c, s = cs[pos].double().unsqueeze(1).split(rot // 2, -1)

    def turn(x, h):
        x = x.reshape(tokens, h, D).clone()
        a, b = (x[..., :rot // 2], x[..., rot // 2:rot]) if neox else (x[..., 0:rot:2], x[..., 1:rot:2])
        a, b = a * c - b * s, b * c + a * s
        x[..., :rot] = torch.cat([a, b], -1) if neox else torch.stack([a, b], -1).flatten(-2)
        return x
    dev = qkv.cuda()
    dq, dk, dv = dev.split([Hq * D, Hk * D, Hk * D], -1)
    kp = torch.zeros(tokens + 5, Hk, D, dtype=torch.bfloat16, device="cuda")
    vp = torch.zeros_like(kp)
    ops.rope_kvwrite(pos.cuda(), dq, dk, dv, kp, vp, loc.cuda(), D, cs.cuda(), neox)
    # one rounding to 16 bits of a value computed in fp32 (a product's and a sum's rounding, 2^-22 at most, beside it)
    for got, want in ((dq, turn(q, Hq)), (dk, turn(k, Hk)), (kp[loc.cuda()], turn(k, Hk))):
        want = want.reshape(tokens, -1)
        got = got.double().cpu().reshape(tokens, -1)
        assert ((got - want).abs() <= want.abs() * 2 ** -8 + 1e-5).all()
    assert torch.equal(vp[loc.cuda()].reshape(tokens, -1).cpu(), qkv[:, (Hq + Hk) * D:])


@pytest.mark.parametrize("sms,tokens", [(2, 1), (2, 2), (2, 6), (2, 7), (72, 47), (72, 48), (72, 216), (72, 217)])
@pytest.mark.parametrize("heads", [(32, 8, 128, 128), (64, 8, 128, 128)])
def test_lines_follow_the_callers_sms(sms, tokens, heads):
    from semi_pd_b200 import ops
    ops.set_sm_budget(sms)
    try:
        test_rope_kvwrite(tokens, heads, True)
    finally:
        ops.set_sm_budget(0)
