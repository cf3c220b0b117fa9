"""RMS norm with the weights read beside the row and behind its sum: on both sides of the lines between them, with and without
the sum of a residual, rows longer than the registers hold."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("tokens,dim", [(1, 8), (3, 4096), (444, 4104), (445, 4104), (445, 6144), (444, 6152), (445, 6152), (450, 8192),
                                        (75, 8200), (75, 12288), (74, 12296), (75, 12296), (5, 16384), (75, 16384), (9, 16400)])
def test_rows(dtype, tokens, dim):
    from semi_pd_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(tokens + dim)
    x, r = (torch.randn(tokens, dim, generator=g, device=DEV).to(dtype) for _ in range(2))
    w = torch.randn(dim, generator=g, device=DEV).to(dtype)
    unit = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11

    def want(v):
        return v * torch.rsqrt(v.square().mean(-1, keepdim=True) + 1e-6) * w.double()

    def near(got, v, roundings):  # of values computed in fp32 to 16 bits, each by at most half a unit in the last place
        assert ((got.double() - v).abs() <= 1.01 * roundings * unit * v.abs() + 1e-6).all()
    near(ops.rmsnorm(x, w, 1e-6), want(x.double()), 1)
    both = x.float() + r.float()
    total = both.to(dtype)
    y, s = x.clone(), r.clone()
    ops.fused_add_rmsnorm(y, s, w, 1e-6)
    assert torch.equal(s, total)
    near(y, want(both.double()), 1 if dim <= 16384 else 2)  # (what the registers do not hold is read back rounded)
