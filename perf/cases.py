"""What this framework's speed is measured on: single layers, operators and two whole calls of its forward path, at the sizes
that its model configurations, tests and benchmark use.

A case is a dict of plain values; its "kind" says which entry point it goes through:

  llama_step     ModelRunner.forward, decode step through the captured CUDA graph (Llama-3-8B widths, few layers, whole head)
  llama_extend   ModelRunner.forward, prefill of new prompts and of further chunks of longer ones
  attn_decode    ops.attn_decode, one new token per request over its pages
  attn_extend    ops.attn_prefill, ragged chunked prefill
  mlp            LlamaMLP.forward (decode batches and prefill chunks)
  mla_decode     SpdAttnBackend.forward_mla, decode over latent pages (DeepSeek-V2-Lite)
  mla_extend     DeepseekV2AttentionMLA.forward, the whole attention layer on a prefill batch
  moe            DeepseekV2MoE.forward: router, 64 routed experts, 2 shared ones
  window_extend  ops.attn_general, window + sinks + query temperature, ragged prefill (hybrid families)
  window_decode  ops.attn_general, the same layer one token per request
  retention      ops.retention, ragged prefill of a recurrent mixer in 32-bit state (hybrid families)

Lengths of the requests of a batch are unequal: half to one and a half times the case's mean, odd sizes among them.
"""
import math
import random

import torch

from semi_pd_b200 import ops
from semi_pd_b200.configs import ServerArgs, get_model_config
from semi_pd_b200.deepseek_v2 import DeepseekV2MoE
from semi_pd_b200.forward_batch_info import ForwardBatch, ForwardMode, ModelWorkerBatch
from semi_pd_b200.llama import LlamaMLP
from semi_pd_b200.memory_pool import MHATokenToKVPool, ReqToTokenPool, TokenToKVPoolAllocator
from semi_pd_b200.model_runner import ModelRunner

F64 = torch.float64
DEV = "cuda"


# ---------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------
def listed():
    return [
        # one user, one token: the smallest call a server makes, all weights read for a single row
        dict(name="llama_step_1", kind="llama_step", dtype="bfloat16", layers=4, batch=1, tokens=1000),
        # one prompt of a thousand tokens behind the last chunk of a longer one: what time to first token is made of
        dict(name="llama_extend_1300", kind="llama_extend", dtype="bfloat16", layers=2, requests=2, tokens=650, prefix=1024),
        # a saturated decode batch of the benchmark (64 requests, 1024 in / 128 out)
        dict(name="attn_decode_64", kind="attn_decode", dtype="bfloat16", batch=64, tokens=1088),
        # few requests with long contexts in the other 16-bit type
        dict(name="attn_decode_5_long", kind="attn_decode", dtype="float16", batch=5, tokens=7000),
        # a full prefill batch (8192 new tokens), some requests with cached prefixes
        dict(name="attn_extend_8192", kind="attn_extend", dtype="bfloat16", requests=8, tokens=1024, prefix=1024),
        # the feed-forward of a decode batch
        dict(name="mlp_64", kind="mlp", dtype="bfloat16", tokens=64),
        # DeepSeek-V2-Lite under load: decode attention over latent pages, prefill through the attention layer
        dict(name="mla_decode_64", kind="mla_decode", dtype="bfloat16", batch=64, tokens=1088),
        dict(name="mla_extend_4096", kind="mla_extend", dtype="bfloat16", requests=4, tokens=1024, prefix=512),
        # its mixture of experts on a decode batch and on a prefill batch
        dict(name="moe_40", kind="moe", dtype="bfloat16", tokens=40),
        dict(name="moe_4096", kind="moe", dtype="bfloat16", tokens=4096),
        # the hybrid families' windowed attention and recurrent mixer on a prefill batch
        dict(name="window_extend_8192", kind="window_extend", dtype="bfloat16", requests=4, tokens=2048, prefix=1024, window=1024),
        dict(name="retention_8192", kind="retention", dtype="bfloat16", requests=4, tokens=2048, prefix=1024),
    ]


def _spread(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["llama_step", "llama_extend", "attn_decode", "attn_extend", "mlp", "mla_decode", "mla_extend", "moe",
                       "window_extend", "window_decode", "retention"])
    c = dict(kind=kind, dtype=rng.choice(["bfloat16", "float16"]))
    if kind == "llama_step":
        batch = _spread(rng, 1, 160)
        c.update(layers=rng.choice([1, 2, 4]), batch=batch, tokens=_spread(rng, 16, min(1200, 40000 // batch)))
    elif kind == "llama_extend":
        requests = _spread(rng, 1, 8)
        c.update(layers=rng.choice([1, 2]), requests=requests, tokens=_spread(rng, 8, 2048 // requests),
                 prefix=rng.choice([0, 128, 1000]))
    elif kind == "attn_decode":
        batch = _spread(rng, 1, 160)
        c.update(batch=batch, tokens=_spread(rng, 32, min(8000, 160000 // batch)))
    elif kind == "attn_extend":
        requests = _spread(rng, 1, 16)
        c.update(requests=requests, tokens=_spread(rng, 16, 8192 // requests), prefix=rng.choice([0, 100, 1024, 3000]))
    elif kind == "mlp":
        c.update(tokens=_spread(rng, 1, 4096))
    elif kind == "mla_decode":
        batch = _spread(rng, 1, 160)
        c.update(batch=batch, tokens=_spread(rng, 32, min(8000, 160000 // batch)))
    elif kind == "mla_extend":
        requests = _spread(rng, 1, 8)
        c.update(requests=requests, tokens=_spread(rng, 16, 4096 // requests), prefix=rng.choice([0, 100, 512]))
    elif kind == "moe":
        c.update(tokens=_spread(rng, 1, 4096))
    elif kind == "window_extend":
        requests = _spread(rng, 1, 8)
        c.update(requests=requests, tokens=_spread(rng, 16, 8192 // requests), prefix=rng.choice([0, 100, 1500]),
                 window=rng.choice([128, 512, 1024]))
    elif kind == "window_decode":
        c.update(batch=_spread(rng, 1, 160), tokens=_spread(rng, 32, 3000), window=rng.choice([128, 512, 1024]))
    else:
        requests = _spread(rng, 1, 8)
        c.update(requests=requests, tokens=_spread(rng, 16, 8192 // requests), prefix=rng.choice([0, 700]))
    return c


def _lengths(n, mean, salt=0):
    """Unequal lengths around `mean` that add up to n * mean (a batch of one has just that length)."""
    if n == 1:
        return [mean]
    r = random.Random(1000003 * n + 101 * mean + salt)
    out = [max(1, int(mean * (0.5 + r.random()))) for _ in range(n)]
    short = n * mean - sum(out)
    for i in range(n):
        step = short // (n - i) if short >= 0 else -(-short // (n - i))
        step = max(step, 1 - out[i])
        out[i] += step
        short -= step
    return out


def _extend_lengths(c):
    """(new tokens, cached tokens) of every request: each second one continues a longer prompt."""
    new = _lengths(c["requests"], c["tokens"])
    old = [c["prefix"] + 3 * i if i % 2 == 1 or c["requests"] == 1 else 0 for i in range(c["requests"])]
    return new, [p if c["prefix"] else 0 for p in old]


def _seen(new, old, window=None):
    """Pairs (query, visible key) of a causal batch."""
    n = 0
    for e, p in zip(new, old):
        if window is None:
            n += e * p + e * (e + 1) // 2
        else:
            grow = max(0, min(e, window - 1 - p))  # queries that still see everything
            n += grow * p + grow * (grow + 1) // 2 + (e - grow) * window
    return n


# ---------------------------------------------------------------------------------------------
# sizes
# ---------------------------------------------------------------------------------------------
LLAMA = dict(H=4096, I=14336, HQ=32, HK=8, D=128, V=128256)
MLA = dict(H=2048, heads=16, nope=128, rope=64, v=128, rank=512)
MOE = dict(H=2048, E=64, top=6, inter=1408, shared=2816)
HYB = dict(heads=16, kv_heads=4, D=128, qtemp=(0.3, 128), rot=64, base=1e6)


def _dtype(c):
    return getattr(torch, c["dtype"])


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _randn(g, *shape, dtype=torch.float32, scale=1.0):
    return (torch.randn(*shape, generator=g, device=DEV, dtype=torch.float32) * scale).to(dtype)


# ---------------------------------------------------------------------------------------------
# what a program has in hand
# ---------------------------------------------------------------------------------------------
def _place(alloc, req_to_token, old, new, seed):
    """Slots for `old` cached and `new` further tokens of every request, and the page-table rows.  The requests come in
    any order, as they do in a server.  → (request slots, slots of the new tokens in batch order)"""
    n = len(new)
    order = list(range(n))
    random.Random(seed).shuffle(order)
    if any(old):
        alloc.alloc_extend(order, [0] * n, [old[i] for i in order])
        for i in order:
            slots = torch.from_numpy(alloc.req_slots(i).astype("int32")).to(DEV)
            req_to_token[i, : old[i]] = slots
    loc = alloc.alloc_extend(list(range(n)), old, [o + e for o, e in zip(old, new)])
    idx = torch.arange(n, dtype=torch.int64, device=DEV)
    as64 = lambda v: torch.tensor(v, dtype=torch.int64, device=DEV)  # noqa: E731
    ops.write_req_to_token_pool(req_to_token, idx, as64(old), as64([o + e for o, e in zip(old, new)]), as64(new), loc)
    return idx, loc


def _room(old, new):
    return 128 * (sum(-(-(o + e) // 128) + 1 for o, e in zip(old, new)) + 2)


def _runner(cfg, c, seed, old, new, graph_bs=None):
    n = len(new)
    sa = ServerArgs(model_path=cfg.name, dtype=c["dtype"], load_format="dummy", max_total_tokens=_room(old, new),
                    max_running_requests=n + 1, context_length=max(o + e for o, e in zip(old, new)) + 8,
                    disable_cuda_graph=graph_bs is None, cuda_graph_bs=graph_bs, random_seed=int(seed) % (1 << 30),
                    enable_semi_pd=True)
    mr = ModelRunner(cfg, 0.95, 0, 0, 1, 0, sa)
    mr.init_attention_backend()
    idx, loc = _place(mr.token_to_kv_pool_allocator, mr.req_to_token_pool.req_to_token, old, new, seed)
    g = _gen(seed + 7)
    for layer in range(cfg.num_hidden_layers):  # what earlier calls have cached
        bufs = mr.token_to_kv_pool.get_kv_buffer(layer)
        for b in bufs if isinstance(bufs, (tuple, list)) and bufs[0].data_ptr() != bufs[1].data_ptr() else bufs[:1]:
            b.normal_(generator=g)
    mr.init_cuda_graphs()
    return mr, idx, loc, g


def _extend_batch(mr, ids, idx, loc, old, new):
    return ModelWorkerBatch(bid=0, forward_mode=ForwardMode.EXTEND, input_ids=ids, req_pool_indices=idx,
                            seq_lens=torch.tensor([o + e for o, e in zip(old, new)], dtype=torch.int64, device=DEV),
                            out_cache_loc=loc, seq_lens_sum=sum(old) + sum(new), extend_num_tokens=sum(new),
                            extend_seq_lens=list(new), extend_prefix_lens=list(old))


def _decode_batch(ids, idx, loc, lens):
    return ModelWorkerBatch(bid=0, forward_mode=ForwardMode.DECODE, input_ids=ids, req_pool_indices=idx,
                            seq_lens=torch.tensor(lens, dtype=torch.int64, device=DEV), out_cache_loc=loc,
                            seq_lens_sum=sum(lens))


def _pages(c, seed, old, new, heads, dim):
    """A one-layer KV pool with everything cached, for the attention operators."""
    dt = _dtype(c)
    room = _room(old, new)
    pool = MHATokenToKVPool(room, 1, dt, heads, dim, 1, DEV)
    alloc = TokenToKVPoolAllocator(room, dt, DEV, pool)
    r2t = ReqToTokenPool(len(new) + 1, max(o + e for o, e in zip(old, new)) + 8, DEV).req_to_token
    idx, _ = _place(alloc, r2t, old, new, seed)
    g = _gen(seed + 7)
    k, v = pool.get_kv_buffer(0)
    k.normal_(generator=g)
    v.normal_(generator=g)
    return g, k, v, r2t, idx


def _i32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


def _starts(new):
    out, at = [], 0
    for e in new:
        out.append(at)
        at += e
    return out


def prepare(case, seed):
    c, kind, dt = case, case["kind"], _dtype(case)
    s = dict(case=c, kind=kind)
    if kind == "llama_step":
        lens = _lengths(c["batch"], c["tokens"])
        cfg = get_model_config("llama-3-8b", num_hidden_layers=c["layers"])
        old, new = [n - 1 for n in lens], [1] * len(lens)
        mr, idx, loc, g = _runner(cfg, c, seed, old, new, [c["batch"]])
        ids = torch.randint(0, cfg.vocab_size, (len(lens),), generator=g, device=DEV)
        s.update(mr=mr, old=old, new=new, ids=ids, batch=_decode_batch(ids, idx, loc, lens))
    elif kind == "llama_extend":
        new, old = _extend_lengths(c)
        cfg = get_model_config("llama-3-8b-2layer", num_hidden_layers=c["layers"])
        mr, idx, loc, g = _runner(cfg, c, seed, old, new)
        ids = torch.randint(0, cfg.vocab_size, (sum(new),), generator=g, device=DEV)
        s.update(mr=mr, old=old, new=new, ids=ids, batch=_extend_batch(mr, ids, idx, loc, old, new))
    elif kind == "attn_decode":
        lens = _lengths(c["batch"], c["tokens"])
        z = LLAMA
        g, k, v, r2t, idx = _pages(c, seed, [0] * len(lens), lens, z["HK"], z["D"])
        s.update(q=_randn(g, len(lens), z["HQ"] * z["D"], dtype=dt), k=k, v=v, r2t=r2t, idx=idx,
                 lens=torch.tensor(lens, dtype=torch.int64, device=DEV), old=[n - 1 for n in lens], new=[1] * len(lens))
    elif kind == "attn_extend":
        new, old = _extend_lengths(c)
        z = LLAMA
        g, k, v, r2t, idx = _pages(c, seed, old, new, z["HK"], z["D"])
        s.update(q=_randn(g, sum(new), z["HQ"] * z["D"], dtype=dt), k=k, v=v, r2t=r2t, idx=idx, old=old, new=new,
                 d_old=_i32(old), d_new=_i32(new), d_start=_i32(_starts(new)))
    elif kind == "mlp":
        z, g = LLAMA, _gen(seed)
        mlp = LlamaMLP(z["H"], z["I"], "silu")
        mlp.gate_up_proj.weight = _randn(g, 2 * z["I"], z["H"], dtype=dt, scale=z["H"] ** -0.5)
        mlp.down_proj.weight = _randn(g, z["H"], z["I"], dtype=dt, scale=z["I"] ** -0.5)
        s.update(mlp=mlp, x=_randn(g, c["tokens"], z["H"], dtype=dt))
    elif kind in ("mla_decode", "mla_extend"):
        z = MLA
        cfg = get_model_config("deepseek-v2-lite", num_hidden_layers=1, vocab_size=1024)
        if kind == "mla_decode":
            lens = _lengths(c["batch"], c["tokens"])
            old, new = [n - 1 for n in lens], [1] * len(lens)
        else:
            new, old = _extend_lengths(c)
        mr, idx, loc, g = _runner(cfg, c, seed, old, new)
        ids = torch.zeros(sum(new), dtype=torch.int64, device=DEV)
        attn = mr.model.model.layers[0].self_attn
        if kind == "mla_decode":
            fb = ForwardBatch.init_new(_decode_batch(ids, idx, loc, lens), mr)
            # an absorbed query: its latent part scores like a 128-wide head's
            q = _randn(g, len(lens), z["heads"], z["rank"] + z["rope"])
            q[:, :, : z["rank"]] *= (z["nope"] / z["rank"]) ** 0.5
            s.update(q=q.view(len(lens), -1).to(dt))
        else:
            fb = ForwardBatch.init_new(_extend_batch(mr, ids, idx, loc, old, new), mr)
            s.update(x=_randn(g, sum(new), z["H"], dtype=dt))
        mr.attn_backend.init_forward_metadata(fb)
        s.update(mr=mr, attn=attn, fb=fb, old=old, new=new)
    elif kind == "moe":
        z, g = MOE, _gen(seed)
        moe = DeepseekV2MoE(get_model_config("deepseek-v2-lite"))
        moe.gate.weight = _randn(g, z["E"], z["H"], dtype=dt, scale=z["H"] ** -0.5)
        moe.w_gate_up = _randn(g, z["E"] * 2 * z["inter"], z["H"], dtype=dt, scale=z["H"] ** -0.5)
        moe.w_down_cat = _randn(g, z["H"], z["E"] * z["inter"], dtype=dt, scale=z["inter"] ** -0.5)
        moe.shared_experts.gate_up_proj.weight = _randn(g, 2 * z["shared"], z["H"], dtype=dt, scale=z["H"] ** -0.5)
        moe.shared_experts.down_proj.weight = _randn(g, z["H"], z["shared"], dtype=dt, scale=z["shared"] ** -0.5)
        s.update(moe=moe, x=_randn(g, c["tokens"], z["H"], dtype=dt))
    elif kind in ("window_extend", "window_decode"):
        z = HYB
        if kind == "window_decode":
            lens = _lengths(c["batch"], c["tokens"])
            old, new = [n - 1 for n in lens], [1] * len(lens)
            s["lens"] = torch.tensor(lens, dtype=torch.int64, device=DEV)
        else:
            new, old = _extend_lengths(c)
            s.update(d_old=_i32(old), d_new=_i32(new), d_start=_i32(_starts(new)))
        g, k, v, r2t, idx = _pages(c, seed, old, new, z["kv_heads"], z["D"])
        s.update(q=_randn(g, sum(new), z["heads"] * z["D"], dtype=dt), k=k, v=v, r2t=r2t, idx=idx, old=old, new=new,
                 sinks=_randn(g, z["heads"]))
    else:
        z, g = HYB, _gen(seed)
        new, old = _extend_lengths(c)
        T, H, D = sum(new), z["heads"], z["D"]
        pos = torch.arange(max(o + e for o, e in zip(old, new)) + 8, dtype=F64, device=DEV)
        inv = z["base"] ** (-torch.arange(0, z["rot"], 2, dtype=F64, device=DEV) / z["rot"])
        ang = pos[:, None] * inv
        qkv = _randn(g, T, 3 * H * D, dtype=dt)  # one projection's output, read in place
        s.update(q=qkv[:, : H * D], k=qkv[:, H * D: 2 * H * D], v=qkv[:, 2 * H * D:], old=old, new=new,
                 state=_randn(g, len(new) + 1, H, D, D, scale=0.5),
                 decay=torch.tensor([1.0 - 2.0 ** (-5 - 0.5 * h) for h in range(H)], device=DEV),
                 cos_sin=torch.cat((ang.cos(), ang.sin()), -1).float().contiguous(),
                 idx=torch.arange(len(new), dtype=torch.int64, device=DEV), d_old=_i32(old), d_new=_i32(new),
                 d_start=_i32(_starts(new)))
    return s


# ---------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------
def run(s):
    kind = s["kind"]
    if kind in ("llama_step", "llama_extend"):
        mr = s["mr"]
        out = mr.forward(ForwardBatch.init_new(s["batch"], mr)).next_token_logits
        if kind == "llama_step":
            return out
        pool = mr.token_to_kv_pool
        return [out] + [b for i in range(s["case"]["layers"]) for b in pool.get_kv_buffer(i)]
    if kind == "attn_decode":
        z = LLAMA
        return ops.attn_decode(s["q"], s["k"], s["v"], s["r2t"], s["idx"], s["lens"], z["HQ"], z["HK"], z["D"], z["D"] ** -0.5)
    if kind == "attn_extend":
        z = LLAMA
        return ops.attn_prefill(s["q"], s["k"], s["v"], s["r2t"], s["idx"], s["d_old"], s["d_new"], s["d_start"],
                                max(s["new"]), z["HQ"], z["HK"], z["D"], z["D"] ** -0.5)
    if kind == "mlp":
        return s["mlp"].forward(s["x"])
    if kind == "mla_decode":
        return s["mr"].attn_backend.forward_mla(s["q"], s["attn"].attn_mqa, s["fb"])
    if kind == "mla_extend":
        out = s["attn"].forward(s["fb"].positions, s["x"], s["fb"])
        return [out, s["mr"].token_to_kv_pool.get_key_buffer(0)]
    if kind == "moe":
        return s["moe"].forward(s["x"])
    z = HYB
    if kind in ("window_extend", "window_decode"):
        common = dict(num_q_heads=z["heads"], num_kv_heads=z["kv_heads"], head_dim=z["D"], v_dim=z["D"], sm_scale=z["D"] ** -0.5,
                      window=s["case"]["window"], sinks=s["sinks"], qtemp_coef=z["qtemp"][0], qtemp_every=z["qtemp"][1])
        if kind == "window_decode":
            return ops.attn_general(s["q"], s["k"], s["v"], s["r2t"], s["idx"], seq_lens=s["lens"], **common)
        return ops.attn_general(s["q"], s["k"], s["v"], s["r2t"], s["idx"], prefix_lens=s["d_old"], extend_lens=s["d_new"],
                                extend_start_loc=s["d_start"], max_extend_len=max(s["new"]), **common)
    o = ops.retention(s["q"], s["k"], s["v"], s["state"], s["idx"], z["heads"], z["D"], z["D"], s["decay"], s["cos_sin"],
                      z["rot"], z["D"] ** -0.5, prefix_lens=s["d_old"], extend_lens=s["d_new"], extend_start_loc=s["d_start"])
    return [o, s["state"]]


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without: every input once, every output once, the products of the path
# ---------------------------------------------------------------------------------------------
def work(case):
    c, kind = case, case["kind"]
    if kind in ("llama_step", "attn_decode", "mla_decode", "window_decode"):
        lens = _lengths(c["batch"], c["tokens"])
        T, ctx = len(lens), sum(lens)
    elif kind not in ("mlp", "moe"):
        new, old = _extend_lengths(c)
        T, ctx, seen = sum(new), sum(new) + sum(old), _seen(new, old)
    else:
        T = c["tokens"]
    if kind in ("llama_step", "llama_extend"):
        z = LLAMA
        V, rows = (z["V"], T) if kind == "llama_step" else (4096, c["requests"])
        per = z["H"] * (z["HQ"] + 2 * z["HK"]) * z["D"] + z["HQ"] * z["D"] * z["H"] + 3 * z["H"] * z["I"]
        kv = 2 * z["HK"] * z["D"]
        pairs = ctx if kind == "llama_step" else seen
        return dict(bytes=2 * (c["layers"] * (per + kv * (ctx + T)) + V * z["H"] + T * z["H"]) + 4 * rows * V,
                    flops=2 * (c["layers"] * per * T + V * z["H"] * rows) + 4 * c["layers"] * pairs * z["HQ"] * z["D"])
    if kind in ("attn_decode", "attn_extend"):
        z = LLAMA
        pairs = ctx if kind == "attn_decode" else seen
        return dict(bytes=2 * (2 * ctx * z["HK"] * z["D"] + 2 * T * z["HQ"] * z["D"]) + 4 * ctx, flops=4 * pairs * z["HQ"] * z["D"])
    if kind == "mlp":
        z = LLAMA
        return dict(bytes=2 * (3 * z["H"] * z["I"] + 2 * T * z["H"]), flops=2 * T * 3 * z["H"] * z["I"])
    if kind == "mla_decode":
        z = MLA
        wide = z["rank"] + z["rope"]
        return dict(bytes=2 * (ctx * wide + T * z["heads"] * (wide + z["rank"])) + 4 * ctx,
                    flops=2 * ctx * z["heads"] * (wide + z["rank"]))
    if kind == "mla_extend":
        z = MLA
        wide, hd = z["rank"] + z["rope"], z["heads"]
        proj = z["H"] * (hd * (z["nope"] + z["rope"]) + wide) + hd * (z["nope"] + z["v"]) * z["rank"] + hd * z["v"] * z["H"]
        # per pair of query and key: the head's own widths (a cached row expands to them once)
        return dict(bytes=2 * (proj + 2 * T * z["H"] + (ctx + T) * wide),
                    flops=2 * (T * proj + seen * hd * (z["nope"] + z["rope"] + z["v"])))
    if kind == "moe":
        z = MOE
        used = z["E"] * (1 - (1 - z["top"] / z["E"]) ** T)
        expert = 3 * z["H"] * z["inter"]
        return dict(bytes=2 * (used * expert + 3 * z["H"] * z["shared"] + z["E"] * z["H"] + 2 * T * z["H"]),
                    flops=2 * T * (z["top"] * expert + 3 * z["H"] * z["shared"] + z["E"] * z["H"]))
    z = HYB
    row = z["D"] * z["heads"]
    if kind == "window_decode":
        keys = sum(min(n, c["window"]) for n in lens)
        return dict(bytes=2 * (2 * keys * z["kv_heads"] * z["D"] + 2 * T * row) + 4 * keys, flops=4 * keys * row)
    if kind == "window_extend":
        keys = sum(e + min(p, c["window"] - 1) for e, p in zip(new, old))
        return dict(bytes=2 * (2 * keys * z["kv_heads"] * z["D"] + 2 * T * row) + 4 * keys,
                    flops=4 * _seen(new, old, c["window"]) * row)
    state = len(new) * z["heads"] * z["D"] * z["D"]
    return dict(bytes=2 * 3 * T * row + 4 * T * row + 8 * state, flops=4 * T * z["heads"] * z["D"] * z["D"])


# About four times what another correct implementation shows: outputs in 16 bits differ by their rounding, and inside a
# layer the operands of the next product do.
def tolerance(case):
    kind, half = case["kind"], case["dtype"] == "float16"
    if kind == "retention":
        return {"rel": 1e-5, "max": 1e-4}
    if kind in ("llama_step", "llama_extend"):
        return {"rel": 0.004, "max": 0.03} if half else {"rel": 0.03, "max": 0.25}
    if kind in ("mlp", "moe", "mla_extend"):
        return {"rel": 0.003, "max": 0.03} if half else {"rel": 0.02, "max": 0.2}
    return {"rel": 0.0015, "max": 0.015} if half else {"rel": 0.01, "max": 0.1}


# ---------------------------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------------------------
def _d(t):
    return t.to(F64)


def _mm(x, w):
    """x [T, K] times a 16-bit weight [N, K] transposed, a block of rows of the weight at a time."""
    return torch.cat([x @ _d(b).T for b in w.split(32768)], -1)


def _norm(x, w, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * _d(w)


def _rope(x, table, pos):
    """Rotate-half over the first `table.shape[1]` channels of x [T, H, D]."""
    rot = table.shape[1]
    half = rot // 2
    cs = _d(table)[pos]
    cos, sin = cs[:, None, :half], cs[:, None, half:]
    a, b = x[..., :half], x[..., half:rot]
    return torch.cat((a * cos - b * sin, b * cos + a * sin, x[..., rot:]), -1)


def _rope_pairs(x, table, pos):
    half = table.shape[1] // 2
    cs = _d(table)[pos]
    cos, sin = cs[:, None, :half], cs[:, None, half:]
    a, b = x[..., 0::2], x[..., 1::2]
    return torch.stack((a * cos - b * sin, b * cos + a * sin), -1).flatten(-2)


def _attend(q, k, v, first, scale, window=None, sinks=None, temp=None):
    """q [e, H, D] at positions first.. over k / v [L, G, D] (causal), a block of queries at a time."""
    H, G, L = q.shape[1], k.shape[1], k.shape[0]
    k, v = k.repeat_interleave(H // G, 1), v.repeat_interleave(H // G, 1)
    j = torch.arange(L, device=DEV)
    out = []
    for at in range(0, q.shape[0], 256):
        i = first + at + torch.arange(min(256, q.shape[0] - at), device=DEV)
        s = torch.einsum("qhd,khd->hqk", q[at: at + 256], k) * scale
        if temp is not None:
            s = s * (1 + temp[0] * torch.log(torch.floor((_d(i) + 1) / temp[1]) + 1))[None, :, None]
        gone = j[None, :] > i[:, None]
        if window is not None:
            gone = gone | (i[:, None] - j[None, :] >= window)
        s = s.masked_fill(gone[None], float("-inf"))
        if sinks is not None:
            s = torch.cat((s, _d(sinks)[:, None, None].expand(-1, s.shape[1], 1)), -1)
        p = torch.softmax(s, -1)[..., :L]
        out.append(torch.einsum("hqk,khd->qhd", p, v))
    return torch.cat(out)


def _exact_llama(s):
    mr, new, old = s["mr"], s["new"], s["old"]
    m, z, pool = mr.model, LLAMA, mr.token_to_kv_pool
    x = _d(m.model.embed_tokens.weight[s["ids"]])
    pos = torch.cat([o + torch.arange(e, device=DEV) for o, e in zip(old, new)])
    r2t = mr.req_to_token_pool.req_to_token.long()
    cached = []
    for li, layer in enumerate(m.model.layers):
        a = layer.self_attn
        kb, vb = (_d(b) for b in pool.get_kv_buffer(li))
        qkv = _mm(_norm(x, layer.input_layernorm.weight, layer.input_layernorm.variance_epsilon), a.qkv_proj.weight)
        q, k, v = qkv.split([z["HQ"] * z["D"], z["HK"] * z["D"], z["HK"] * z["D"]], -1)
        q = _rope(q.view(-1, z["HQ"], z["D"]), a.rotary_emb.cos_sin_cache, pos)
        k = _rope(k.view(-1, z["HK"], z["D"]), a.rotary_emb.cos_sin_cache, pos)
        loc = s["batch"].out_cache_loc
        kb[loc], vb[loc] = k, v.view(-1, z["HK"], z["D"])
        cached += [kb, vb]
        outs = []
        for r, (at, o, e) in enumerate(zip(_starts(new), old, new)):
            rows = r2t[r, : o + e]
            outs.append(_attend(q[at: at + e], kb[rows], vb[rows], o, z["D"] ** -0.5))
        x = x + _mm(torch.cat(outs).flatten(1), a.o_proj.weight)
        h = _mm(_norm(x, layer.post_attention_layernorm.weight, layer.post_attention_layernorm.variance_epsilon),
                layer.mlp.gate_up_proj.weight)
        gate, up = h.chunk(2, -1)
        x = x + _mm(torch.nn.functional.silu(gate) * up, layer.mlp.down_proj.weight)
    x = _norm(x, m.model.norm.weight, m.model.norm.variance_epsilon)
    if s["kind"] == "llama_step":
        return _mm(x, m.lm_head.weight)
    last = torch.tensor([at + e - 1 for at, e in zip(_starts(new), new)], device=DEV)
    return [_mm(x[last], m.lm_head.weight)] + cached


def exact(case, seed):
    s = prepare(case, seed)
    kind = s["kind"]
    if kind in ("llama_step", "llama_extend"):
        return _exact_llama(s)
    if kind == "mlp":
        gate, up = _mm(_d(s["x"]), s["mlp"].gate_up_proj.weight).chunk(2, -1)
        return _mm(torch.nn.functional.silu(gate) * up, s["mlp"].down_proj.weight)
    if kind == "moe":
        z, moe, x = MOE, s["moe"], _d(s["x"])
        # the router's scores are 16-bit numbers by definition of the layer: which experts are chosen hangs on that
        logits = _d(_mm(x, moe.gate.weight).to(s["x"].dtype))
        p = torch.softmax(logits, -1)
        ids = torch.sort(logits, dim=-1, descending=True, stable=True)[1][:, : z["top"]]
        w = p.gather(1, ids)
        gate, up = _mm(x, moe.shared_experts.gate_up_proj.weight).chunk(2, -1)
        y = _mm(torch.nn.functional.silu(gate) * up, moe.shared_experts.down_proj.weight)
        for e in range(z["E"]):
            t, j = (ids == e).nonzero(as_tuple=True)
            if t.numel():
                gate, up = _mm(x[t], moe.w_gate_up[2 * e * z["inter"]: 2 * (e + 1) * z["inter"]]).chunk(2, -1)
                h = torch.nn.functional.silu(gate) * up
                y.index_add_(0, t, w[t, j][:, None] * _mm(h, moe.w_down_cat[:, e * z["inter"]: (e + 1) * z["inter"]]))
        return y
    new, old = s["new"], s["old"]
    if kind in ("mla_decode", "mla_extend"):
        z, attn, mr = MLA, s["attn"], s["mr"]
        pool = _d(mr.token_to_kv_pool.get_key_buffer(0))
        kv = pool.view(pool.shape[0], -1)
        r2t = mr.req_to_token_pool.req_to_token.long()
        hd, R = z["heads"], z["rank"]
        outs = []
        if kind == "mla_decode":
            q = _d(s["q"]).view(-1, hd, R + z["rope"])
            for r, n in enumerate(o + 1 for o in old):
                rows = kv[r2t[r, :n]]
                outs.append(_attend(q[r: r + 1], rows[:, None], rows[:, None, :R], n - 1, attn.scaling))
            return torch.cat(outs).flatten(1)
        pos = torch.cat([o + torch.arange(e, device=DEV) for o, e in zip(old, new)])
        qa = _mm(_d(s["x"]), attn.q_kv_a_proj.weight)
        q = qa[:, : attn.q_size].reshape(-1, hd, z["nope"] + z["rope"])
        q_pe = _rope_pairs(q[..., z["nope"]:], attn.cos_sin_cache, pos)
        c = _norm(qa[:, attn.q_size: attn.q_size + R], attn.kv_a_layernorm.weight, attn.kv_a_layernorm.variance_epsilon)
        k_pe = _rope_pairs(qa[:, None, attn.q_size + R:], attn.cos_sin_cache, pos)[:, 0]
        kv[s["fb"].out_cache_loc] = torch.cat((c, k_pe), -1)
        w_kc = _d(attn.w_kc_t).view(hd, R, z["nope"])
        w_vc = _d(attn.w_vc).view(hd, z["v"], R)
        for r, (at, o, e) in enumerate(zip(_starts(new), old, new)):
            rows = kv[r2t[r, : o + e]]
            k = torch.cat((torch.einsum("lr,hrn->lhn", rows[:, :R], w_kc), rows[:, None, R:].expand(-1, hd, -1)), -1)
            v = torch.einsum("lr,hvr->lhv", rows[:, :R], w_vc)
            outs.append(_attend(torch.cat((q[at: at + e, :, : z["nope"]], q_pe[at: at + e]), -1), k, v, o, attn.scaling))
        return [_mm(torch.cat(outs).flatten(1), attn.o_proj.weight), pool]
    if kind == "retention":
        z = HYB
        H, D = z["heads"], z["D"]
        q, k, v = (_d(s[n]).reshape(-1, H, D) for n in "qkv")
        pos = torch.cat([o + torch.arange(e, device=DEV) for o, e in zip(old, new)])
        q, k = _rope(q, s["cos_sin"], pos), _rope(k, s["cos_sin"], pos) * D ** -0.5
        state, o_all = _d(s["state"]), []
        log = torch.log(_d(s["decay"]))
        for r, (at, o, e) in enumerate(zip(_starts(new), old, new)):
            S = state[r] if o else torch.zeros_like(state[r])
            for b in range(at, at + e, 128):
                n = min(128, at + e - b)
                i = torch.arange(n, device=DEV, dtype=F64)
                far = (i[:, None] - i[None, :])[None] * log[:, None, None]
                mask = torch.where(far <= 0, torch.exp(far), torch.zeros_like(far))
                mask = torch.where((i[:, None] >= i[None, :])[None], mask, torch.zeros_like(mask))
                A = torch.einsum("ihd,jhd->hij", q[b: b + n], k[b: b + n]) * mask
                o_all.append(torch.einsum("hij,jhd->ihd", A, v[b: b + n])
                             + torch.einsum("ihk,hkd->ihd", q[b: b + n] * torch.exp((i[:, None] + 1) * log)[..., None], S))
                S = (torch.exp(n * log)[:, None, None] * S
                     + torch.einsum("jhk,jhd->hkd", k[b: b + n] * torch.exp((n - 1 - i[:, None]) * log)[..., None], v[b: b + n]))
            state[r] = S
        return [torch.cat(o_all).flatten(1), state]
    G, D = s["k"].shape[1], s["k"].shape[2]
    H = s["q"].shape[1] // D
    q, outs = _d(s["q"]).view(-1, H, D), []
    more = {}
    if kind.startswith("window"):
        more = dict(window=s["case"]["window"], sinks=s["sinks"], temp=HYB["qtemp"])
    for r, (at, o, e) in enumerate(zip(_starts(new), old, new)):
        rows = s["r2t"][r, : o + e].long()
        outs.append(_attend(q[at: at + e], _d(s["k"][rows]), _d(s["v"][rows]), o, D ** -0.5, **more))
    return torch.cat(outs).flatten(1)
