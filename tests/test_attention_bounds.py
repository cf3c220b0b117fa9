"""The bound that the attention tests hold a request to (tests.helpers.ATTN_REL) fails when one tile of its keys is left out or
counted twice: planted here in the 64-bit reference."""
import pytest
import torch

from tests.helpers import assert_requests_close


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("keys,tile", [(5000, 64), (5000, 128), (2000, 64), (700, 64), (65, 1)])
def test_a_lost_or_doubled_tile_is_seen(dtype, keys, tile):
    g = torch.Generator().manual_seed(keys + tile)
    q, k, v = torch.randn(8, 64, generator=g), torch.randn(keys, 64, generator=g), torch.randn(keys, 64, generator=g)
    s = (q.double() @ k.double().t()) * 64 ** -0.5
    p = torch.softmax(s, -1)
    want = p @ v.double()
    rounded = (p.to(dtype).double() @ v.double()).to(dtype)
    assert_requests_close(rounded[None], want[None], [1], dtype)
    for at in (0, keys // 2 // tile * tile, keys - tile):
        for times in (0.0, 2.0):
            w = s.exp()
            w[:, at: at + tile] *= times
            with pytest.raises(AssertionError):
                assert_requests_close((w @ v.double() / w.sum(-1, keepdim=True))[None], want[None], [1], dtype)
