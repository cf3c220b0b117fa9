"""Expert layers behind one another without a wait on the host: every pass ends, with the first one's bits."""
import pytest
import torch

from semi_pd_b200.configs import get_model_config
from semi_pd_b200.deepseek_v2 import DeepseekV2MoE

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens", [40, 400, 4096])
def test_passes_in_a_row(tokens):
    cfg = get_model_config("deepseek-v2-lite")
    g = torch.Generator("cuda").manual_seed(tokens)
    rnd = lambda r, c: torch.randn(r, c, generator=g, device="cuda").mul_(c ** -0.5).to(torch.bfloat16)
    H, E, inter = cfg.hidden_size, cfg.n_routed_experts, cfg.moe_intermediate_size
    shared = inter * cfg.n_shared_experts
    moe = DeepseekV2MoE(cfg)
    moe.gate.weight, moe.w_gate_up, moe.w_down_cat = rnd(E, H), rnd(E * 2 * inter, H), rnd(H, E * inter)
    moe.shared_experts.gate_up_proj.weight, moe.shared_experts.down_proj.weight = rnd(2 * shared, H), rnd(H, shared)
    x = rnd(tokens, H) * H ** 0.5
    first = moe.forward(x)
    done = torch.cuda.Event()
    wrong = torch.zeros((), dtype=torch.int64, device="cuda")
    for _ in range(4):  # (few passes in flight at a time)
        for _ in range(25):
            wrong += (moe.forward(x) != first).any()
        done.record()
        done.synchronize()
    assert wrong.item() == 0
