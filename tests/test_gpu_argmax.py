"""Greedy sampling over rows that a cluster of CTAs shares: rows of every length around a CTA's share, ties in one share and
over two, rows of nothing but infinities, not-a-number beside numbers, rows that are not 16-byte aligned; also as
(max, index) pairs."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("V", [16383, 16384, 16389, 65536, 128256, 50272])
@pytest.mark.parametrize("B", [1, 5, 37, 38])
@pytest.mark.parametrize("pad", [0, 3])
def test_rows(B, V, pad):
    from semi_pd_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(B + V)
    x = torch.randn(B, V + pad, generator=g, device=DEV)[:, :V]
    x[0, 7::1000] = 9.0                       # ties: the first
    if B > 1:
        x[1] = float("-inf")
        x[2, :-1], x[2, -1] = float("nan"), -3.0
        x[3, -1] = 20.0
    want = torch.where(x.isnan(), torch.full_like(x, float("-inf")), x)
    best = want.max(-1)[0]
    first = (want == best[:, None]).int().argmax(-1)
    assert torch.equal(ops.argmax(x).long(), first)
    assert torch.equal(ops.argmax_merge(ops.argmax_partial(x, 0)[None]).long().view(-1), first)


@pytest.mark.parametrize("V", [5, 8192, 8193, 16380, 16384, 49151, 49152, 98303, 98304, 128000, 196608])  # around the lines between the forms
@pytest.mark.parametrize("B", [1, 4, 5, 6, 7, 12, 13, 32, 33])
def test_forms(B, V):
    from semi_pd_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(B + V)
    x = torch.randint(-50, 50, (B, V), generator=g, device=DEV).float()  # ties everywhere
    x[0] = float("-inf")
    best = x.max(-1)[0]
    assert torch.equal(ops.argmax(x).long(), (x == best[:, None]).int().argmax(-1))
