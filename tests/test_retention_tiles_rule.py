"""Which prefill batches of the retention mixer run in tiles: where their waves take less than the chunks of 64 tokens do."""
import pytest

from semi_pd_b200 import _lib


@pytest.mark.parametrize("batch,tokens,heads,dv,dtype,sms,tiled", [
    (1, 200, 16, 128, "bf16", 148, False), (1, 300, 16, 128, "bf16", 148, True), (4, 8192, 16, 128, "bf16", 148, True),
    (4, 8192, 16, 128, "f16", 148, False), (1, 1500, 16, 128, "f16", 148, True), (4, 1000, 16, 128, "bf16", 148, False),
    (8, 1024, 16, 128, "bf16", 148, False), (8, 8000, 16, 128, "bf16", 148, True), (1, 1500, 4, 64, "bf16", 148, True),
    (64, 2600, 4, 128, "bf16", 148, False), (1, 8000, 16, 128, "bf16", 72, True)])
def test_rule(batch, tokens, heads, dv, dtype, sms, tiled):
    dt = _lib.SPD_BF16 if dtype == "bf16" else _lib.SPD_F16
    room = _lib.lib.spd_retention_tiles_workspace_bytes(batch, tokens, heads, 128, dv, 64, 0, dt, sms)
    assert (room > 0) is tiled
    if tiled:  # two forms of the state, lists and marks of every tile that the batch may have
        assert room >= (tokens // 128 + batch) * heads * dv * 128 * 10


def test_not_for_other_sizes():
    f = _lib.lib.spd_retention_tiles_workspace_bytes
    assert f(1, 4000, 16, 128, 128, 64, 0, _lib.SPD_BF16, 148) > 0
    for args in ((1, 4000, 16, 64, 128, 64, 0, _lib.SPD_BF16, 148), (1, 4000, 16, 128, 96, 64, 0, _lib.SPD_BF16, 148),
                 (1, 4000, 16, 128, 128, 24, 0, _lib.SPD_BF16, 148), (1, 4000, 16, 128, 128, 64, 1, _lib.SPD_BF16, 148),
                 (1, 4000, 16, 128, 128, 64, 0, _lib.SPD_F32, 148), (0, 4000, 16, 128, 128, 64, 0, _lib.SPD_BF16, 148),
                 (100, 4000, 16, 128, 128, 64, 0, _lib.SPD_BF16, 148)):
        assert f(*args) == 0


@pytest.mark.parametrize("batch,tokens,heads,dv,sms", [(4, 1000, 4, 128, 72), (2, 500, 4, 128, 148), (8, 2000, 4, 128, 148), (2, 500, 16, 128, 148),
                                                       (8, 2400, 16, 128, 148), (4, 1200, 16, 128, 72), (1, 256, 16, 128, 148)])
def test_chunks_are_faster(batch, tokens, heads, dv, sms):
    assert _lib.lib.spd_retention_tiles_workspace_bytes(batch, tokens, heads, 128, dv, 64, 0, _lib.SPD_BF16, sms) == 0


@pytest.mark.parametrize("batch,tokens,heads,dv,dtype,sms", [(1, 400, 4, 128, "bf16", 148), (2, 900, 16, 128, "bf16", 148), (4, 2000, 16, 128, "bf16", 148),
                                                             (2, 1600, 4, 64, "f16", 72), (1, 8000, 8, 256, "bf16", 40)])
def test_tiles_are_faster(batch, tokens, heads, dv, dtype, sms):
    dt = _lib.SPD_BF16 if dtype == "bf16" else _lib.SPD_F16
    assert _lib.lib.spd_retention_tiles_workspace_bytes(batch, tokens, heads, 128, dv, 64, 0, dt, sms) > 0


def test_scratch_has_a_limit():
    """Long batches go to the chunks, which ran in little memory before there were tiles."""
    room = _lib.lib.spd_retention_tiles_workspace_bytes
    for batch, tokens, heads, dv in ((1, 131072, 16, 128), (1, 65536, 32, 256), (4, 65536, 64, 256), (8, 32768, 16, 128)):
        assert room(batch, tokens, heads, 128, dv, 64, 0, _lib.SPD_BF16, 148) == 0
        chunks = _lib.lib.spd_retention_workspace_bytes(batch, tokens, heads, 128, dv, 64, 0, _lib.SPD_BF16, 148)
        assert chunks <= 512 << 20
    assert 0 < room(4, 16384, 16, 128, 128, 64, 0, _lib.SPD_BF16, 148) <= 512 << 20
    for tokens in range(1000, 200000, 3717):
        assert room(1, tokens, 16, 128, 128, 64, 0, _lib.SPD_BF16, 148) <= 512 << 20
