"""The chunked retention prefill with its portions cut into segments that run side by side (long portions of few requests):
portions around a segment's end, short ones beside long ones, a continued state, every rotation, both 16-bit types, several
value slices; infinite and NaN values and states in each place that a segment can have."""
import pytest
import torch

from tests.test_gpu_retention_chunked import DK, _case, _rel, _run, _want

pytestmark = pytest.mark.gpu


def _cut(ext, H, dv, rot, dtype):
    from semi_pd_b200 import _lib
    dt = _lib.SPD_BF16 if dtype == torch.bfloat16 else _lib.SPD_F16
    return _lib.lib.spd_retention_workspace_bytes(len(ext), sum(ext), H, DK, dv, rot, 0, dt, 0) > 0


# few heads: segments are 128 tokens, the shortest
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rot,dv", [(64, 128), (0, 64), (128, 64), (48, 192)])
@pytest.mark.parametrize("pre,ext", [([0], [767]), ([9], [768]), ([0], [769]), ([0, 30, 4], [1000, 3, 769])])
def test_segments(dtype, rot, dv, pre, ext):
    H, scale, decay = 2, DK ** -0.5, [0.97, 0.9999]
    assert _cut(ext, H, dv, rot, dtype)
    case = _case(pre, ext, H, dv, rot, dtype, decay)
    want = _want(*case, pre, ext, H, dv, rot, scale)
    got = _run(*case, pre, ext, H, dv, rot, scale)
    for a, b in zip(got, want):  # sums of up to 1000 fp32 products: 2^-24 each, at random
        assert _rel(a, b) < 1e-6


@pytest.mark.parametrize("decay", [[0.0, 1.0], [1e-3, 0.5], [1e-30, 0.99999]])
def test_decays(decay):
    pre, ext, H, dv = [3, 0], [700, 900], 2, 64
    case = _case(pre, ext, H, dv, 64, torch.bfloat16, decay)
    assert _cut(ext, H, dv, 64, torch.bfloat16)
    for a, b in zip(_run(*case, pre, ext, H, dv, 64, 0.1), _want(*case, pre, ext, H, dv, 64, 0.1)):
        assert _rel(a, b) < 1e-6


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("what", ["q", "k", "v", "state"])
@pytest.mark.parametrize("at", [5, 127, 128, 300, 900, 1023])
def test_values_that_are_not_finite(dtype, what, at):
    """As one token after another: everything before them, and what does not meet them, is what it is without them."""
    pre, ext, H, dv, scale = [4, 0], [1024, 600], 2, 128, DK ** -0.5
    q, k, v, state, table, decay = _case(pre, ext, H, dv, 64, dtype, [0.97, 0.999])
    assert _cut(ext, H, dv, 64, dtype)
    nan, inf = float("nan"), float("inf")
    if what == "state":
        state[0, 1, 7, 70] = nan
        state[0, 0, 100, 3] = 2.0 ** 70  # too large to be split beside the others, but finite
    elif what == "q":
        q[at, 3], q[at, DK + 100] = nan, inf
    elif what == "k":
        k[at, 90] = inf
    else:
        v[at, dv + 66] = -inf
    case = (q, k, v, state, table, decay)
    want = _want(*case, pre, ext, H, dv, 64, scale)
    got = _run(*case, pre, ext, H, dv, 64, scale)
    for a, b in zip(got, want):
        fine = b.isfinite()
        assert torch.equal(a.isfinite(), fine)
        assert _rel(a[fine], b[fine]) < 1e-6
