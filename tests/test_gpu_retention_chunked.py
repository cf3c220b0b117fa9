"""The chunked tensor-core form of the retention prefill: portions around its 64-token chunk, rotations over none, some and
all channels, several value slices, both 16-bit types, a continued state, fast and slow decays, values that are not finite;
against the recurrence in 64 bits, with the error of 32-bit sums."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
DK = 128


def _case(pre, ext, H, dv, rot, dtype, decay, seed=0):
    g = torch.Generator().manual_seed(seed + sum(ext) + rot + dv)
    T = sum(ext)
    q, k = (torch.randn(T, H * DK, generator=g).to(dtype) for _ in range(2))
    v = torch.randn(T, H * dv, generator=g).to(dtype)
    state = torch.randn(len(ext) + 1, H, DK, dv, generator=g)
    pos = torch.arange(max(p + e for p, e in zip(pre, ext)) + 4, dtype=torch.float64)
    inv = 1e4 ** (-torch.arange(0, max(rot, 2), 2, dtype=torch.float64) / max(rot, 2))
    table = torch.cat(((pos[:, None] * inv).cos(), (pos[:, None] * inv).sin()), -1).float() if rot else None
    return q, k, v, state, table, torch.tensor(decay, dtype=torch.float32)


def _rotate(x, table, pos, rot):
    if not rot:
        return x
    c, s = table[pos, None, : rot // 2].double(), table[pos, None, rot // 2:].double()
    a, b = x[..., : rot // 2], x[..., rot // 2: rot]
    return torch.cat((a * c - b * s, b * c + a * s, x[..., rot:]), -1)


def _want(q, k, v, state, table, decay, pre, ext, H, dv, rot, scale):
    out, final, at = [], state.double().clone(), 0
    for r, (p, e) in enumerate(zip(pre, ext)):
        pos = p + torch.arange(e)
        qq = _rotate(q[at:at + e].double().view(e, H, DK), table, pos, rot)
        kk = _rotate(k[at:at + e].double().view(e, H, DK), table, pos, rot) * scale
        vv = v[at:at + e].double().view(e, H, dv)
        S = final[r] if p > 0 else torch.zeros_like(final[r])
        for t in range(e):
            S = decay.double()[:, None, None] * S + kk[t][:, :, None] * vv[t][:, None, :]
            out.append(torch.einsum("hkv,hk->hv", S, qq[t]).reshape(1, -1))
        if e:
            final[r] = S
        at += e
    return torch.cat(out), final


def _run(q, k, v, state, table, decay, pre, ext, H, dv, rot, scale):
    from semi_pd_b200 import ops
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    st = state.to(DEV)
    o = ops.retention(q.to(DEV), k.to(DEV), v.to(DEV), st, torch.arange(len(ext), device=DEV), H, DK, dv, decay.to(DEV),
                      None if table is None else table.to(DEV), rot, scale, prefix_lens=i32(pre), extend_lens=i32(ext),
                      extend_start_loc=i32([sum(ext[:i]) for i in range(len(ext))]))
    return o.cpu().double(), st.cpu().double()


def _rel(a, b):
    return ((a - b).norm() / b.norm()).item()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rot", [0, 16, 64, 128])
@pytest.mark.parametrize("pre,ext", [([0], [1]), ([7, 0, 30], [130, 1, 24]), ([0, 5], [63, 64]), ([9, 0, 0], [65, 0, 130]),
                                     ([200], [300])])
def test_portions(dtype, rot, pre, ext):
    H, dv = 3, 128
    a = _case(pre, ext, H, dv, rot, dtype, [0.97, 0.999, 0.875])
    o, s = _run(*a, pre, ext, H, dv, rot, DK ** -0.5)
    wo, ws = _want(*a, pre, ext, H, dv, rot, DK ** -0.5)
    # sums of at most some hundred terms in fp32 (2^-24 each, random signs) and one rounding per chunk of the state
    assert _rel(o, wo) < 1e-6 and _rel(s, ws) < 1e-6, (_rel(o, wo), _rel(s, ws))


@pytest.mark.parametrize("decay", [[0.0, 1.0], [1e-3, 0.5], [1e-30, 0.9999]])
def test_decays(decay):
    H, dv, pre, ext = 2, 64, [3, 0], [150, 70]
    a = _case(pre, ext, H, dv, 64, torch.bfloat16, decay)
    o, s = _run(*a, pre, ext, H, dv, 64, 1.0)
    wo, ws = _want(*a, pre, ext, H, dv, 64, 1.0)
    assert _rel(o, wo) < 1e-6 and _rel(s, ws) < 1e-6


def test_values_that_are_not_finite_leave_the_tokens_before_them_alone():
    H, dv, pre, ext = 1, 64, [0, 0], [100, 40]
    q, k, v, state, table, decay = _case(pre, ext, H, dv, 64, torch.bfloat16, [0.9])
    v[70, 5] = float("inf")
    v[90, 6] = float("nan")
    o, _ = _run(q, k, v, state, table, decay, pre, ext, H, dv, 64, 1.0)
    clean = v.clone()
    clean[70, 5] = clean[90, 6] = 0
    wo, _ = _want(q, k, clean, state, table, decay, pre, ext, H, dv, 64, 1.0)
    seen = torch.ones_like(wo, dtype=torch.bool)
    seen[70:100, 5] = seen[90:100, 6] = False
    assert torch.isfinite(o[seen]).all() and not torch.isfinite(o[70:100, 5]).any() and not torch.isfinite(o[90:100, 6]).any()
    assert _rel(o[seen], wo[seen]) < 1e-6


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("what", ["q", "k", "state", "v", "all"])
def test_values_that_are_not_finite_as_token_by_token(dtype, what):
    """Infinities and NaNs in q, k, v and the state: finite, infinite (with the sign) and NaN where the token-by-token kernel
    (taken by portions of one token) has them."""
    H, dv, pre, ext = 2, 64, [5, 0, 9], [200, 50, 64]
    q, k, v, state, table, decay = _case(pre, ext, H, dv, 64, dtype, [0.9, 0.5])
    inf, nan = float("inf"), float("nan")
    if what in ("q", "all"):  # a channel that is not rotated: 0.7 inf, then inf - inf
        q[70, 100], q[90, DK + 3], q[249, 100], q[249, 101] = inf, nan, -inf, inf
    if what in ("k", "all"):
        k[130, 99], k[220, 5] = -inf, nan
    if what in ("v", "all"):
        v[150, 3], v[263, dv + 1], v[300, 9] = inf, -inf, nan
    if what in ("state", "all"):
        state[0, 1, 100, 7], state[2, 0, 1, 2] = inf, -inf
    whole, ws = _run(q, k, v, state, table, decay, pre, ext, H, dv, 64, 1.0)
    st, rows = state, [[], [], []]
    starts = [0, 200, 250]
    for t in range(max(ext)):
        live = [r for r in range(3) if t < ext[r]]
        at = [starts[r] + t for r in live]
        o, s = _run(q[at], k[at], v[at], torch.cat((st[live], st[-1:])).float(), table, decay, [pre[r] + t for r in live],
                    [1] * len(live), H, dv, 64, 1.0)
        st = st.clone().double()
        st[live] = s[:-1]
        for i, r in enumerate(live):
            rows[r].append(o[i: i + 1])
    steps = torch.cat([torch.cat(r) for r in rows])
    for a, b in ((whole, steps), (ws[:3], st[:3])):
        fin = b.isfinite()
        assert torch.equal(a.isnan(), b.isnan()) and torch.equal(a.isinf(), b.isinf())
        assert torch.equal(a[b.isinf()], b[b.isinf()])
        assert _rel(a[fin], b[fin]) < 1e-6


def test_strided_rows_and_a_cut_prompt():
    """q, k, v as slices of one projection; a prompt in three portions against the prompt in one."""
    H, dv, n = 2, 128, 333
    q, k, v, state, table, decay = _case([0], [n], H, dv, 64, torch.float16, [0.95, 0.99])
    qkv = torch.cat((q, k, v), 1)
    parts = (qkv[:, : H * DK], qkv[:, H * DK: 2 * H * DK], qkv[:, 2 * H * DK:])
    whole, ws = _run(*parts, state, table, decay, [0], [n], H, dv, 64, DK ** -0.5)
    got, st, at = [], state, 0
    for m in (100, 1, n - 101):  # (the single token goes through the token-by-token kernel)
        o, s = _run(*(x[at:at + m].contiguous() for x in parts), st.float(), table, decay, [at], [m], H, dv, 64, DK ** -0.5)
        got.append(o)
        st, at = s, at + m
    assert _rel(torch.cat(got), whole) < 1e-6 and _rel(st[0], ws[0]) < 1e-6
