"""Which MLA prefill batches take the expanded form: those with many queries per key, within the keys whose K and V it keeps."""
import pytest

from semi_pd_b200.deepseek_v2 import _MLA_EXPANDED_MAX_KEYS, mla_expanded_pays


@pytest.mark.parametrize("ext,pre,heads,sms,pays", [
    ([1], [0], 16, 148, False), ([512], [0], 16, 148, False), ([1024], [0], 16, 148, True), ([4096], [0], 16, 148, True),
    ([128] * 4, [0, 515, 0, 521], 16, 148, False), ([1024] * 4, [0, 515, 0, 521], 16, 148, True),
    ([128], [4000], 16, 148, False), ([256], [4000], 16, 148, True), ([128], [16000], 16, 148, False),
    ([0, 2048], [700, 0], 16, 148, True), ([0], [5], 16, 148, False), ([2048], [0], 3, 40, True), ([2048], [0], 128, 148, True),
    ([2000], [_MLA_EXPANDED_MAX_KEYS - 2000], 16, 148, True), ([2000], [_MLA_EXPANDED_MAX_KEYS - 1999], 16, 148, False),
])
def test_rule(ext, pre, heads, sms, pays):
    assert mla_expanded_pays(ext, pre, heads, sms) is pays
