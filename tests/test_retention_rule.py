"""Which prefill batches of the chunked retention are cut into segments, and into how many at most (bf16 rows of 128 channels):
where the waves that they run in, each with its start, take less than the longest portion."""
import pytest

from semi_pd_b200 import _lib


def _segments(batch, tokens, heads, dv, sms):
    room = _lib.lib.spd_retention_workspace_bytes(batch, tokens, heads, 128, dv, 64, 0, _lib.SPD_BF16, sms)
    per = heads * (2 * dv * 128 * 4 + dv // 64 * 4)  # two states a head and a flag per 64 columns
    assert room % per == 0
    return room // per


@pytest.mark.parametrize("batch,tokens,heads,dv,sms,segments", [
    (1, 300, 16, 128, 148, 0), (1, 500, 16, 128, 148, 4), (1, 1500, 16, 128, 148, 8), (1, 8000, 16, 128, 148, 18),
    (2, 1000, 16, 128, 148, 0), (2, 2000, 16, 128, 148, 9), (2, 6000, 16, 128, 148, 13), (3, 6000, 16, 128, 148, 0),
    (4, 8192, 16, 128, 148, 0), (3, 6000, 32, 128, 148, 10), (8, 8000, 4, 128, 148, 39), (4, 8000, 16, 64, 148, 29),
    (4, 8192, 64, 128, 148, 0), (1, 60, 16, 128, 148, 0), (2, 6000, 16, 128, 72, 0), (1, 8000, 4, 128, 40, 14)])
def test_rule(batch, tokens, heads, dv, sms, segments):
    assert _segments(batch, tokens, heads, dv, sms) == segments
