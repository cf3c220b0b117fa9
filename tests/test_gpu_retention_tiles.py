"""The retention prefill in tiles of 128 tokens: portions around a tile's end and its middle, requests without new tokens among
others, a continued state, every rotation, both 16-bit types, one and several value blocks, more tiles than SMs, decays at both
ends; infinite and NaN values and states in every place that a tile can have; rows with strides; a partition of the SMs."""
import pytest
import torch

from tests.test_gpu_retention_chunked import DK, _case, _rel, _run, _want

pytestmark = pytest.mark.gpu


def _tiled(ext, H, dv, rot, dtype, sms=0):
    from semi_pd_b200 import _lib
    dt = _lib.SPD_BF16 if dtype == torch.bfloat16 else _lib.SPD_F16
    return _lib.lib.spd_retention_tiles_workspace_bytes(len(ext), sum(ext), H, DK, dv, rot, 0, dt, sms) > 0


# fp32 sums: each of some hundred rounded products and additions is off by up to 2^-24 of it, at random
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rot,dv", [(64, 128), (0, 64), (128, 64), (48, 192), (16, 256)])
@pytest.mark.parametrize("pre,ext", [([0], [384]), ([9], [385]), ([700, 0, 4, 30], [447, 0, 449, 511]), ([0, 5, 1], [1000, 1, 65])])
def test_portions(dtype, rot, dv, pre, ext):
    H, scale, decay = 2, DK ** -0.5, [0.97, 0.9999]
    assert _tiled(ext, H, dv, rot, dtype)
    case = _case(pre, ext, H, dv, rot, dtype, decay)
    for a, b in zip(_run(*case, pre, ext, H, dv, rot, scale), _want(*case, pre, ext, H, dv, rot, scale)):
        assert _rel(a, b) < 1e-6


@pytest.mark.parametrize("decay", [[0.0, 1.0], [1e-3, 0.5], [1e-30, 0.99999]])
def test_decays(decay):
    pre, ext, H, dv = [3, 0], [700, 900], 2, 128
    case = _case(pre, ext, H, dv, 64, torch.bfloat16, decay)
    assert _tiled(ext, H, dv, 64, torch.bfloat16)
    for a, b in zip(_run(*case, pre, ext, H, dv, 64, 0.1), _want(*case, pre, ext, H, dv, 64, 0.1)):
        assert _rel(a, b) < 1e-6


@pytest.mark.parametrize("budget", [0, 40])
def test_several_items_an_sm(budget):
    from semi_pd_b200 import ops
    H, dv, pre, ext = 24, 128, [0, 100, 0], [1500, 600, 900]
    case = _case(pre, ext, H, dv, 64, torch.bfloat16, [1 - 2.0 ** (-3 - 0.25 * h) for h in range(H)])
    assert _tiled(ext, H, dv, 64, torch.bfloat16, budget)
    ops.set_sm_budget(budget)
    try:
        got = _run(*case, pre, ext, H, dv, 64, 0.1)
    finally:
        ops.set_sm_budget(0)
    for a, b in zip(got, _want(*case, pre, ext, H, dv, 64, 0.1)):
        assert _rel(a, b) < 1e-6


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("what", ["q", "k", "v", "state", "large"])
@pytest.mark.parametrize("at", [0, 127, 128, 500, 767])
def test_values_that_are_not_finite(dtype, what, at):
    """As one token after another: everything before them, and what does not meet them, is what it is without them."""
    pre, ext, H, dv, scale = [4, 0], [768, 400], 2, 128, DK ** -0.5
    q, k, v, state, table, decay = _case(pre, ext, H, dv, 64, dtype, [0.97, 0.999])
    assert _tiled(ext, H, dv, 64, dtype)
    nan, inf = float("nan"), float("inf")
    if what == "state":
        state[0, 1, 7, 70], state[0, 0, 100, 3], state[0, 1, at % 128, 5] = nan, 2.0 ** 70, -inf
    elif what == "q":
        q[at, 3], q[at, DK + 100] = nan, inf
    elif what == "k":
        k[at, 90] = inf
    elif what == "v":
        v[at, dv + 66] = -inf
    elif dtype == torch.bfloat16:
        q[at], k[at] = q[at] * 2.0 ** 60, k[at] * 2.0 ** 60  # A would overflow beside values that do not
    case = (q, k, v, state, table, decay)
    want = _want(*case, pre, ext, H, dv, 64, scale)
    got = _run(*case, pre, ext, H, dv, 64, scale)
    for a, b in zip(got, want):
        fine = b.isfinite() & (b.abs() < 3e38)
        assert torch.equal(a.isfinite(), fine)
        assert torch.equal(a.isnan(), b.isnan())
        small = fine & (b.abs() < 1e30)
        assert _rel(a[small], b[small]) < 1e-6


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("what", ["q", "k", "v"])
@pytest.mark.parametrize("at", [130, 383, 700])
def test_a_large_state_before_a_tile_that_is_not_finite(dtype, what, at):
    """The state that one key of the first tile makes is above 2^64, and a later tile goes on from it token by token."""
    pre, ext, H, dv, scale = [4, 0], [768, 400], 2, 128, 2.0 ** 40
    q, k, v, state, table, decay = _case(pre, ext, H, dv, 64, dtype, [0.99, 0.9999])
    assert _tiled(ext, H, dv, 64, dtype)
    for h in range(H):
        k[10, h * DK + 100], v[10, h * dv: (h + 1) * dv: 3] = 2.0 ** 15, -2.0 ** 15
    {"q": q, "k": k, "v": v}[what][at, 70] = float("nan")
    case = (q, k, v, state, table, decay)
    for a, b in zip(_run(*case, pre, ext, H, dv, 64, scale), _want(*case, pre, ext, H, dv, 64, scale)):
        assert torch.equal(a.isnan(), b.isnan())
        # as above: sums of at most some hundred terms in fp32
        assert _rel(a[b.isfinite()], b[b.isfinite()]) < 1e-6
