"""The MLA attention layer on prefill batches that take the expanded form (K and V of every head made from the cached latent
rows), through DeepseekV2AttentionMLA.forward: new prompts, a second chunk behind cached prefixes, scattered cache slots, with
and without YaRN, against the oracle's layer; the absorbed form on the same batch; the cache rows that both write."""
import pytest
import torch

from oracle import deepseek_oracle as D
from tests.test_gpu_deepseek import MINI, YARN, _weights

pytestmark = pytest.mark.gpu
DEV = "cuda"
SLOTS = 4096


def _layer(rope_scaling, dtype):
    from semi_pd_b200.configs import ModelConfig, ServerArgs
    from semi_pd_b200.model_runner import ModelRunner
    sizes = dict(MINI, num_hidden_layers=1)
    ocfg = D.DeepseekOracleConfig(**sizes, rope_scaling=rope_scaling)
    weights = _weights(ocfg, dtype)
    mcfg = ModelConfig(name="mini-deepseek", model_type="deepseek_v2", num_key_value_heads=16, head_dim=192,
                       rms_norm_eps=ocfg.rms_norm_eps, rope_theta=ocfg.rope_theta, rope_scaling=rope_scaling, **sizes)
    sa = ServerArgs(model_path="mini-deepseek", dtype="float16" if dtype == torch.float16 else "bfloat16",
                    load_format="external", max_total_tokens=SLOTS, max_running_requests=8, context_length=2000,
                    disable_cuda_graph=True, enable_semi_pd=True)
    mr = ModelRunner(mcfg, 0.5, 0, 0, 1, 0, sa)
    mr.model.load_weights(weights.items())
    mr.init_attention_backend()
    return mr, D.DeepseekOracle(ocfg, weights, kv_slots=SLOTS, max_reqs=8, max_ctx=2048)


def _batch(mr, idx, pre, ext, loc):
    from semi_pd_b200.forward_batch_info import ForwardBatch, ForwardMode, ModelWorkerBatch
    fb = ForwardBatch.init_new(ModelWorkerBatch(
        bid=0, forward_mode=ForwardMode.EXTEND, input_ids=torch.zeros(sum(ext), dtype=torch.int64, device=DEV),
        req_pool_indices=idx, seq_lens=torch.tensor([p + e for p, e in zip(pre, ext)], device=DEV), out_cache_loc=loc,
        seq_lens_sum=sum(pre) + sum(ext), extend_num_tokens=sum(ext), extend_seq_lens=list(ext), extend_prefix_lens=list(pre)), mr)
    mr.attn_backend.init_forward_metadata(fb)
    return fb


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("rope_scaling", [None, YARN], ids=["rope", "yarn"])
def test_layer_in_both_forms(rope_scaling, dtype):
    from semi_pd_b200 import deepseek_v2
    mr, oracle = _layer(rope_scaling, dtype)
    attn, pool = mr.model.model.layers[0].self_attn, mr.token_to_kv_pool.get_key_buffer(0)
    g = torch.Generator().manual_seed(4)
    slots, rows = torch.randperm(SLOTS - 1, generator=g) + 1, torch.randperm(mr.req_to_token_pool.req_to_token.shape[0], generator=g)
    idx, at = rows[:4].to(DEV), 0
    # 16-bit roundings on the way: input projection, K and V (or the absorbed query and the latent output), P, the heads'
    # output, the layer's: about 2^-9 (2^-12) each, a row's error 0.006 (0.0008) of its norm
    tol = 4e-3 if dtype == torch.float16 else 3e-2
    for pre, ext in (([0, 0, 0, 0], [700, 1, 513, 90]), ([700, 1, 513, 90], [600, 5, 300, 64])):
        loc, at = slots[at: at + sum(ext)], at + sum(ext)
        s0 = 0
        for b, (p, e) in enumerate(zip(pre, ext)):
            mr.req_to_token_pool.req_to_token[idx[b], p: p + e] = loc[s0: s0 + e].int().to(DEV)
            oracle.req_to_token[b, p: p + e] = loc[s0: s0 + e].int()
            s0 += e
        x = torch.randn(sum(ext), MINI["hidden_size"], generator=g).to(dtype)
        pos = torch.cat([torch.arange(p, p + e) for p, e in zip(pre, ext)])
        want = oracle._attention(0, x.float(), pos, torch.arange(4), torch.tensor([p + e for p, e in zip(pre, ext)]), pre, ext, loc,
                                 False).double()
        fb, before = _batch(mr, idx, pre, ext, loc.to(DEV)), pool.clone()
        got = attn.forward(fb.positions, x.to(DEV), fb)
        assert fb.mla_expanded is deepseek_v2.mla_expanded_pays(ext, pre, 16, 148) is True
        written = pool.clone()
        pool.copy_(before)
        fb = _batch(mr, idx, pre, ext, loc.to(DEV))
        fb.mla_expanded = False
        absorbed = attn.forward(fb.positions, x.to(DEV), fb)
        assert torch.equal(pool, written)
        for out in (got, absorbed):
            err = ((out.cpu().double() - want).norm(dim=-1) / want.norm(dim=-1)).max().item()
            assert err < tol, err


def test_small_batch_stays_absorbed():
    mr, _ = _layer(None, torch.bfloat16)
    attn = mr.model.model.layers[0].self_attn
    loc = torch.arange(1, 41, device=DEV)
    mr.req_to_token_pool.req_to_token[0, :40] = loc.int()
    fb = _batch(mr, torch.zeros(1, dtype=torch.int64, device=DEV), [0], [40], loc)
    assert attn.forward(fb.positions, torch.randn(40, MINI["hidden_size"], device=DEV).bfloat16(), fb).isfinite().all()
    assert fb.mla_expanded is False
