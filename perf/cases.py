"""What is measured: the work that a program on this framework has it do, through its public entry points.

Families (the `kind` of a case):

* steps       one decoded token through the cache steps of a whole stack of layers (evict, overwrite, attend, score), captured
              once in a CUDA graph as the framework's graph decoder does; `KVCache.decode_step`
* token       one decoded token of a Llama-family model with compressed caches; `Transformer.forward`
* scores      prompt attention with the score reductions that prompt compression needs; `prefill_attention_stats`
* block       a prompt through one transformer layer (norms, projections, rotation, attention, cache fill, feed-forward);
              `TransformerBlock.forward`
* rows        a prompt, or a portion of one, through the position-addressed attention of the sequence designs;
              `KVCache.sequence_step`
* rows_steps  one token through that attention in a stack of layers, in a CUDA graph; `KVCache.sequence_step`
* recurrence  a prompt portion through one recurrent mixer's scan; `seq_ops.wkv / delta_scan / mlstm`
* experts     a prompt portion through a mixture of experts; `RoutedExperts.forward`
* design      one decoded token of a sequence design through `generation_utils.GraphedDecoder`

Shapes are those of the configurations in model.transformer_configs and bench.py, or odd ones from the same ranges.
"""
import math

import torch

from cold_compress_b200 import _lib, seq_ops
from cold_compress_b200 import generation_utils as gu
from cold_compress_b200.attention_utils import prefill_attention_stats
from cold_compress_b200.cache import get_cache_constructor
from cold_compress_b200.detatar import RoutedExperts
from cold_compress_b200.model import ModelArgs, Transformer, TransformerBlock, precompute_freqs_cis
from cold_compress_b200.relanex import RelanexTransformer
from cold_compress_b200.tokenizer import SyntheticTokenizer

DEV = "cuda"
BF16, F32, F64 = torch.bfloat16, torch.float32, torch.float64


def listed():
    return [
        # smallest: a small sliding cache in every layer (recent + global tokens); latency only
        dict(name="steps_recent_64", kind="steps", policy="recent_global", layers=32, slots=64, kv=8, group=4, dim=128, filled=64),
        # the headline cache: 1024 heavy-hitter slots per layer, 32 layers, full caches
        dict(name="steps_heavy_1024", kind="steps", policy="heavy_hitter", layers=32, slots=1024, kv=8, group=4, dim=128, filled=1024),
        # the headline call: one decoded token of the 8B shape at 8k context with those caches
        dict(name="token_8b_heavy", kind="token", model="Meta-Llama-3-8B-Instruct", layers=32, policy="heavy_hitter", slots=1024),
        # prompt attention of the headline run (7680 tokens), and a short ragged prompt with 7 query heads per key head
        dict(name="scores_7680", kind="scores", tokens=7680, kv=8, group=4, dim=128),
        dict(name="scores_ragged", kind="scores", tokens=1531, kv=4, group=7, dim=128),
        # one layer's share of a prompt that fits its cache
        dict(name="block_4096", kind="block", model="Meta-Llama-3-8B-Instruct", tokens=4096, policy="heavy_hitter"),
        # global attention with learned sinks over a whole prompt, and an odd portion in the middle of a long prompt through
        # a sliding window with a sink of zero
        dict(name="rows_prompt", kind="rows", tokens=4096, past=0, heads=32, kv=8, dk=128, dv=128, window=0, sink=1, softcap=0.0, dtype="bf16"),
        dict(name="rows_portion", kind="rows", tokens=1001, past=3333, heads=16, kv=4, dk=128, dv=128, window=1024, sink=2, softcap=0.0, dtype="bf16"),
        # one token of a stack of global layers at 4k context
        dict(name="rows_steps_4096", kind="rows_steps", layers=8, past=4096, heads=32, kv=8, dk=128, dv=128, window=0, sink=1, dtype="bf16"),
        # a prompt through the matrix-state recurrence (width 2048: 32 heads of 64)
        dict(name="recurrence_4096", kind="recurrence", scan="wkv", tokens=4096, heads=32, dim=64),
        # a prompt through 16 experts of which each token takes 4, with two identity experts and a shared one
        dict(name="experts_2048", kind="experts", tokens=2048, width=2048, ff=1536, shared=2048),
        # one decoded token of a sequence design at 4k context: matrix memory, global and latent attention, gated units
        dict(name="design_token", kind="design", width=2048, heads=16, kv=4, ff=8192, past=4096),
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["steps", "steps", "token", "scores", "scores", "block", "rows", "rows", "rows", "rows_steps", "recurrence", "recurrence",
                       "experts", "design"])
    if kind == "steps":
        slots = 4 * _spread(rng, 12, 500)
        kv, group, dim = rng.choice([(8, 4, 128), (4, 7, 128), (2, 7, 64), (8, 1, 128), (8, 8, 128)])
        return dict(kind=kind, policy=rng.choice(["recent_global", "l2", "heavy_hitter"]), layers=rng.randint(4, 32), slots=slots, kv=kv,
                    group=group, dim=dim, filled=rng.choice([slots, slots, max(24, slots * 3 // 5)]))
    if kind == "token":
        return dict(kind=kind, model=rng.choice(["Meta-Llama-3-8B-Instruct", "Qwen2-7B-Instruct"]), layers=rng.randint(2, 28),
                    policy=rng.choice(["recent_global", "l2", "heavy_hitter"]), slots=4 * _spread(rng, 16, 500))
    if kind == "scores":
        kv, group, dim = rng.choice([(8, 4, 128), (4, 7, 128), (2, 7, 64), (8, 1, 128), (8, 8, 128), (8, 2, 64)])
        return dict(kind=kind, tokens=_spread(rng, 40, 7680 if group <= 4 else 6000), kv=kv, group=group, dim=dim)
    if kind == "block":
        return dict(kind=kind, model=rng.choice(["Meta-Llama-3-8B-Instruct", "Qwen2-7B-Instruct"]), tokens=_spread(rng, 64, 4096),
                    policy=rng.choice(["full", "heavy_hitter"]))
    if kind == "rows":
        heads, kv = rng.choice([(32, 8), (16, 4), (16, 16), (17, 1), (12, 4)])
        dk, dv = rng.choice([(128, 128), (128, 128), (64, 64), (96, 128), (130, 64), (72, 40)])
        window = rng.choice([0, 0, _spread(rng, 16, 2048)])
        dtype = rng.choice(["bf16", "bf16", "bf16", "bf16", "f32"])
        return dict(kind=kind, tokens=_spread(rng, 2, 4000 if dtype == "bf16" else 1500), past=rng.choice([0, 0, rng.randint(1, 4000)]), heads=heads, kv=kv,
                    dk=dk, dv=dv, window=window, sink=rng.randint(0, 2), softcap=rng.choice([0.0, 0.0, 30.0]), dtype=dtype)
    if kind == "rows_steps":
        heads, kv = rng.choice([(32, 8), (16, 4), (12, 4), (16, 16)])
        dk, dv = rng.choice([(128, 128), (128, 128), (64, 64), (96, 128)])
        return dict(kind=kind, layers=rng.randint(2, 8), past=_spread(rng, 16, 12000), heads=heads, kv=kv, dk=dk, dv=dv,
                    window=rng.choice([0, 0, _spread(rng, 64, 2048)]), sink=rng.randint(0, 2), dtype=rng.choice(["bf16", "bf16", "f32"]))
    if kind == "recurrence":
        scan = rng.choice(["wkv", "wkv", "delta", "mlstm"])
        heads, dim = rng.choice([(32, 64), (16, 64), (12, 64), (64, 64), (9, 72)] if scan == "wkv" else [(8, 128), (16, 64), (16, 128)])
        return dict(kind=kind, scan=scan, tokens=_spread(rng, 3, 4096), heads=heads, dim=dim)
    if kind == "experts":
        return dict(kind=kind, tokens=_spread(rng, 8, 4096), width=rng.choice([1024, 2048, 2048]), ff=rng.choice([512, 1536, 1000]), shared=rng.choice([0, 2048]))
    width, heads, kv, ff = rng.choice([(2048, 16, 4, 8192), (4096, 32, 8, 14336), (1024, 8, 8, 2816)])
    return dict(kind="design", width=width, heads=heads, kv=kv, ff=ff, past=_spread(rng, 64, 6000))


# ------------------------------------------------------------------------------------------------ inputs

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 11)


def _randn(gen, *shape, dtype=F32, scale=1.0):
    return (torch.randn(*shape, device=DEV, dtype=F32, generator=gen) * scale).to(dtype)


def _dtype(case):
    return F32 if case.get("dtype") == "f32" else BF16


def _cache(policy, kv, dim, slots, dtype=BF16, **extra):
    cls, relevant = get_cache_constructor(policy)
    kw = dict(max_cache_length=slots, global_tokens=4, max_seq_length=1 << 20, cache_bits=None, recent_window=10, history_window_size=1,
              attn_thresholding=False)
    kw.update({k: extra[k] for k in extra if k in kw})
    kw = {k: kw[k] for k in relevant}
    kw.update({k: extra[k] for k in extra if k == "v_head_dim"})
    return cls(1, kv, dim, dtype, **kw).to(DEV)


def _fill_policy_cache(cache, filled, gen, context):
    """A cache in the middle of a sequence: `filled` slots hold rows of the first `context` positions."""
    n, H = filled, cache.n_heads
    cache.k_cache[:, :, :n] = _randn(gen, 1, H, n, cache.head_dim, dtype=BF16, scale=1.2)
    cache.v_cache[:, :, :n] = _randn(gen, 1, H, n, cache.head_dim, dtype=BF16)
    kept = torch.arange(n, device=DEV, dtype=torch.int32) + torch.where(torch.arange(n, device=DEV) < 4, 0, context - n).to(torch.int32)
    cache.pos[:, :, :n] = kept
    cache.mask[:, :, :, :n] = True
    cache.cache_cts.fill_(n)
    if hasattr(cache, "attn_history_num"):
        cache.attn_history_num[:, :, :n] = torch.rand(1, H, n, 1, device=DEV, dtype=F64, generator=gen)
        cache.attn_history_denom[:, :, :n] = torch.randint(1, 50, (1, H, n), device=DEV, dtype=torch.int32, generator=gen)
        cache.attn_counter.fill_(50)
    if hasattr(cache, "key_norm"):
        cache.update_state(None, None, None, True, None)


def _captured(step):
    """`step` captured in a CUDA graph the way GraphedDecoder does it: library handles, plans and buffers exist already
    because `step` has run once before."""
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        with torch.cuda.graph(graph, stream=stream):
            out = step()
    torch.cuda.current_stream().wait_stream(stream)
    return graph, out


def _steps_inputs(case, seed):
    gen, c = _gen(seed), case
    caches, qkv = [], []
    for _ in range(c["layers"]):
        cache = _cache(c["policy"], c["kv"], c["dim"], c["slots"])
        _fill_policy_cache(cache, c["filled"], gen, 8192)
        caches.append(cache)
        qkv.append((_randn(gen, 1, c["kv"] * c["group"], 1, c["dim"], dtype=BF16, scale=1.5), _randn(gen, 1, c["kv"], 1, c["dim"], dtype=BF16),
                    _randn(gen, 1, c["kv"], 1, c["dim"], dtype=BF16)))
    return caches, qkv


_STATE = ("k_cache", "v_cache", "pos", "attn_history_num", "attn_history_denom", "key_norm")


def _prepare_steps(case, seed):
    caches, qkv = _steps_inputs(case, seed)
    pos = torch.full((1,), 8192, dtype=torch.int32, device=DEV)

    def step():
        return [cache.decode_step(q, k, v, pos) for cache, (q, k, v) in zip(caches, qkv)]

    state = [cache.state_dict() for cache in caches]
    saved = [{k: t.clone() for k, t in s.items()} for s in state]
    step()                                   # plans and output buffers; the caches then go back to where they were
    for s, old in zip(state, saved):
        for k, t in s.items():
            t.copy_(old[k])
    graph, y = _captured(step)
    # layers' buffers laid side by side would be another program's choice; the outputs are the first and last layers' whole
    # state and every layer's attention output
    ends = [{n: getattr(cache, n) for n in _STATE if hasattr(cache, n)} for cache in (caches[0], caches[-1])]
    return dict(kind="steps", graph=graph, pos=pos, out={"y": y, "state": ends}, keep=(caches, qkv))


def _llama_args(case, **more):
    cfg = ModelArgs.from_name(case["model"])
    for k, v in more.items():
        setattr(cfg, k, v)
    return cfg


def _random_weights(module, gen):
    with torch.no_grad():
        for name, p in module.named_parameters():
            if "norm" in name:
                p.fill_(1.0)
            else:
                p.normal_(0.0, 0.02, generator=gen)


def _prepare_token(case, seed):
    gen = _gen(seed)
    cfg = _llama_args(case, n_layer=case["layers"], block_size=65536)
    with torch.device("meta"):
        model = Transformer(cfg).to(BF16)
    model = model.to_empty(device=DEV).eval()
    _random_weights(model, gen)
    slots, policy = case["slots"], case["policy"]
    ck = dict(max_cache_length=[slots], cache_length_pattern="tile", cache_strategy=[policy], cache_strategy_pattern="tile",
              prompt_compression_strategy=["heavy_hitter" if policy == "heavy_hitter" else "recent_global"], global_tokens=4, recent_window=10,
              history_window_size=1, attn_thresholding=False, cache_bits=None, min_recovery_frac=0.9, max_seq_length=65536)
    gu.setup_caches(model, SyntheticTokenizer(vocab_size=cfg.vocab_size), torch.device(DEV), 65536, ck)
    for layer in model.layers:
        _fill_policy_cache(layer.attention.kv_cache, slots, gen, 8192)
    token = torch.randint(0, cfg.vocab_size, (1, 1), dtype=torch.int32, device=DEV, generator=gen)
    pos = torch.full((1,), 8192, dtype=torch.int32, device=DEV)
    return dict(kind="token", model=model, token=token, pos=pos)


def _scores_inputs(case, seed):
    gen, S = _gen(seed), case["tokens"]
    H, kv, D = case["kv"] * case["group"], case["kv"], case["dim"]
    # token-major rows as the fused projection leaves them; keys share a direction per head, as trained heads do
    q = _randn(gen, 1, S, H, D, dtype=BF16).transpose(1, 2)
    k = (_randn(gen, 1, S, kv, D) + 0.5 * _randn(gen, 1, 1, kv, D)).to(BF16).transpose(1, 2)
    v = _randn(gen, 1, S, kv, D, dtype=BF16).transpose(1, 2)
    return q, k, v


def _block_inputs(case, seed):
    gen, S = _gen(seed), case["tokens"]
    cfg = _llama_args(case)
    with torch.device("meta"):
        block = TransformerBlock(cfg).to(BF16)
    block = block.to_empty(device=DEV).eval()
    _random_weights(block, gen)
    x = _randn(gen, 1, S, cfg.dim, dtype=BF16)
    freqs = precompute_freqs_cis(S, cfg.head_dim, cfg.rope_base, BF16, cfg.rope_scaling).to(DEV)
    return cfg, block, x, freqs


def _prepare_block(case, seed):
    cfg, block, x, freqs = _block_inputs(case, seed)
    S = case["tokens"]
    cache = _cache(case["policy"], cfg.n_local_heads, cfg.head_dim, S)
    block.attention.kv_cache = cache
    ids = torch.zeros(1, S, dtype=torch.int32, device=DEV)
    return dict(kind="block", block=block, cache=cache, x=x, ids=ids, pos=torch.arange(S, device=DEV), freqs=freqs)


def _rows_cache(case, gen, past, room):
    """A position-addressed cache that holds what `past` earlier positions left."""
    dt, kv, dk, dv, window = _dtype(case), case["kv"], case["dk"], case["dv"], case["window"]
    slots = window or past + room
    cache = _cache("recent_global" if window else "full", kv, dk, slots, dt, v_head_dim=dv, global_tokens=0)
    have = min(past, slots)
    if have:
        at = torch.arange(past - have, past, device=DEV)
        slot = at % slots
        cache.k_cache[0][:, slot] = _randn(gen, kv, have, dk, dtype=dt)
        cache.v_cache[0][:, slot] = _randn(gen, kv, have, dv, dtype=dt)
        cache.pos[0, 0, slot] = at.to(torch.int32)
        cache.mask[0, :, 0, slot] = True
        cache.cache_cts.fill_(have)
    return cache


def _rows_inputs(case, seed, tokens):
    gen, dt = _gen(seed), _dtype(case)
    layers = []
    for _ in range(case.get("layers", 1)):
        cache = _rows_cache(case, gen, case["past"], tokens)
        q = _randn(gen, tokens, case["heads"], case["dk"], scale=1.3)
        k, v = _randn(gen, tokens, case["kv"], case["dk"], dtype=dt), _randn(gen, tokens, case["kv"], case["dv"], dtype=dt)
        sink = _randn(gen, case["heads"]) if case["sink"] == 1 else None
        layers.append((cache, q, k, v, sink))
    return layers


_SINK = {0: _lib.SINK_NONE, 1: _lib.SINK_LEARNED, 2: _lib.SINK_ZERO}


def _rows_step(case, cache, q, k, v, sink, ip, y):
    return cache.sequence_step(q, k, v, ip, y, window=case["window"], sink=sink, sink_mode=_SINK[case["sink"]], scale=case["dk"] ** -0.5,
                               softcap=case.get("softcap", 0.0))


def _prepare_rows(case, seed):
    layers = _rows_inputs(case, seed, case["tokens"])
    ip = torch.full((1,), case["past"], dtype=torch.int32, device=DEV)
    return dict(kind="rows", case=case, layer=layers[0], ip=ip, y=torch.empty(case["tokens"], case["heads"], case["dv"], dtype=_dtype(case), device=DEV))


def _prepare_rows_steps(case, seed):
    layers = _rows_inputs(case, seed, 1)
    ip = torch.full((1,), case["past"], dtype=torch.int32, device=DEV)
    ys = [torch.empty(1, case["heads"], case["dv"], dtype=_dtype(case), device=DEV) for _ in layers]

    def step():
        return [_rows_step(case, *layer, ip, y) for layer, y in zip(layers, ys)]

    step()               # workspaces; the step leaves the rows of position `past`, which the next pass stores again
    graph, y = _captured(step)
    return dict(kind="rows_steps", graph=graph, out={"y": y, "rows": [layers[-1][0].k_cache, layers[-1][0].v_cache]}, keep=(layers, ip))


def _recurrence_inputs(case, seed):
    gen, T, H, D = _gen(seed), case["tokens"], case["heads"], case["dim"]
    if case["scan"] == "wkv":
        r, k, v = (_randn(gen, T, H * D) for _ in range(3))
        w0 = -2.0 + _randn(gen, H * D, scale=0.5)
        return dict(r=r, k=k, v=v, wraw=_randn(gen, T, H * D, scale=0.3), w0=w0, u=_randn(gen, H, D, scale=0.5), state=torch.zeros(H, D, D, device=DEV))
    if case["scan"] == "delta":
        rows = _randn(gen, T, 3 * H * D + 2 * H)
        return dict(rows=rows, dt_bias=_randn(gen, H, scale=0.5) - 3.0, A_log=_randn(gen, H, scale=0.3), state=torch.zeros(H, D, D, device=DEV))
    rows = _randn(gen, T, 3 * H * D + 2 * H)
    return dict(rows=rows, i_bias=_randn(gen, H, scale=0.3), f_bias=3.0 + _randn(gen, H, scale=0.3), state=torch.zeros(H, D, D, device=DEV),
                aux=torch.zeros(H, D + 2, device=DEV))


def _prepare_recurrence(case, seed):
    s = _recurrence_inputs(case, seed)
    s["o"] = torch.empty(case["tokens"], case["heads"] * case["dim"], device=DEV)
    return dict(kind="recurrence", case=case, **s)


def _experts_inputs(case, seed):
    gen, T, E = _gen(seed), case["tokens"], case["width"]
    with torch.device(DEV):
        moe = RoutedExperts(E, 16, 2, case["ff"], 4, 6, 3, case["shared"], _lib.ACT_SILU, BF16)
    with torch.no_grad():
        for p in moe.parameters():
            p.normal_(0.0, 0.02, generator=gen)
    h = _randn(gen, T, E)
    w = _randn(gen, moe.n_rows(), E, dtype=BF16, scale=0.02)
    h_act = h.to(BF16)
    hp = torch.mm(h_act, w.t(), out_dtype=F32)       # the layer's fused projection of h: router | shared gate | shared gate and up rows
    return moe, hp, h, h_act


def _prepare_experts(case, seed):
    moe, hp, h, h_act = _experts_inputs(case, seed)
    return dict(kind="experts", moe=moe, hp=hp, h=h, h_act=h_act)


def _prepare_design(case, seed):
    gen, E, H = _gen(seed), case["width"], case["heads"]
    memory = {"heads": max(1, H // 2), "dim": 128, "vdim": 128, "gate_cap": 15.0}
    full = {"heads": H, "kv_heads": case["kv"], "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
            "rot": {"base": 500000.0, "dims": 64, "scaling": {"factor": 4.0, "original": 1024, "fast": 32.0, "slow": 1.0}}}
    latent = {"heads": H, "dim": 128, "vdim": 128, "q_rank": 768, "kv_rank": 192, "scale": 128 ** -0.5, "mask": {"size": 1024}}
    kinds, mixers = ("mlstm", "attention", "mlstm", "latent_attention"), {"mlstm": memory, "attention": full, "latent_attention": latent}
    layers = [{"type": k, "mixer": mixers[k], "mlp": {"kind": "dense", "ff": case["ff"]}} for k in kinds]
    cfg = {"architecture": "Relanex", "vocab": 32000, "width": E, "norm": {"eps": 1e-5}, "residual_mult": 0.5, "layers": layers}
    with torch.device(DEV):
        model = RelanexTransformer.from_config(cfg, BF16).eval()
    with torch.no_grad():
        for name, p in model.named_parameters():
            if p.dim() >= 2:
                p.normal_(0.0, 0.02, generator=gen)
            elif name.endswith("alpha"):
                p.fill_(0.7)
            elif name.endswith(("weight", "_norm", "norm_w")):
                p.fill_(1.0)
            elif name.endswith("f_bias"):
                p.fill_(3.0)
        m = model.layers[3].block.mixer
        m.w_uk_t.copy_(m.w_ukv[:m.heads * m.head_dim].reshape(m.heads, m.head_dim, m.kv_rank).transpose(1, 2))
        ck = dict(max_cache_length=[1.0], cache_length_pattern="tile", cache_strategy=["full"], cache_strategy_pattern="tile",
                  prompt_compression_strategy=["recent_global"], global_tokens=0, recent_window=10, cache_bits=None)
        P = case["past"]
        gu.setup_caches(model, SyntheticTokenizer(vocab_size=32000), torch.device(DEV), P + 64, ck)
        prompt = torch.randint(0, 32000, (1, P), dtype=torch.int32, device=DEV, generator=gen)
        gu.prefill(model, prompt, torch.arange(P, device=DEV))
        token, pos = prompt[:, :1].clone(), torch.full((1,), P, dtype=torch.int32, device=DEV)
        decoder = gu.GraphedDecoder()
        for _ in range(2):                           # the first token runs eagerly, the second is captured
            decoder(model, token, pos)
    return dict(kind="design", model=model, decoder=decoder, token=token, pos=pos)


_PREPARE = dict(steps=_prepare_steps, token=_prepare_token, block=_prepare_block, rows=_prepare_rows, rows_steps=_prepare_rows_steps,
                recurrence=_prepare_recurrence, experts=_prepare_experts, design=_prepare_design)


def prepare(case, seed):
    if case["kind"] == "scores":
        return dict(kind="scores", qkv=_scores_inputs(case, seed))
    return _PREPARE[case["kind"]](case, seed)


# ------------------------------------------------------------------------------------------------ one pass

def _delta_views(s, H, D):
    rows, n = s["rows"], H * D
    return rows[:, :n], rows[:, n:2 * n], rows[:, 2 * n:3 * n], rows[:, 3 * n:3 * n + H], rows[:, 3 * n + H:]


@torch.no_grad()
def run(state):
    kind = state["kind"]
    if kind == "steps":
        state["graph"].replay()
        state["pos"].add_(1)
        return state["out"]
    if kind == "rows_steps":
        state["graph"].replay()
        return state["out"]
    if kind == "token":
        logits = state["model"](state["token"], state["pos"], is_prefill=False)
        state["pos"].add_(1)
        first = state["model"].layers[0].attention.kv_cache      # its rows depend on the token alone, not on other layers' rounding
        return {"logits": logits, "first": {n: getattr(first, n) for n in _STATE if hasattr(first, n)}}
    if kind == "scores":
        y, stats = prefill_attention_stats(*state["qkv"])
        return {"y": y, "col_sum": stats.col_sum, "obs_mean": stats.obs_mean}
    if kind == "block":
        cache = state["cache"]
        cache.reset()
        y = state["block"](state["x"], state["ids"], state["pos"], True, state["freqs"], None)
        out = {"y": y, "k": cache.k_cache, "v": cache.v_cache, "pos": cache.pos}
        if hasattr(cache, "attn_history_num"):
            out["num"] = cache.attn_history_num
        return out
    if kind == "rows":
        case, (cache, q, k, v, sink) = state["case"], state["layer"]
        y = _rows_step(case, cache, q, k, v, sink, state["ip"], state["y"])
        if case["window"]:
            state["ip"].add_(case["tokens"])         # the next portion; a whole cache is given the same portion again
        return {"y": y, "k": cache.k_cache, "v": cache.v_cache, "pos": cache.pos}
    if kind == "recurrence":
        case, s = state["case"], state
        H, D = case["heads"], case["dim"]
        if case["scan"] == "wkv":
            seq_ops.wkv(s["r"], s["k"], s["v"], s["wraw"], s["w0"], s["u"], s["state"], s["o"], H, D)
        elif case["scan"] == "delta":
            q, k, v, b, a = _delta_views(s, H, D)
            seq_ops.delta_scan(q, k, v, b, a, s["dt_bias"], s["A_log"], s["state"], s["o"], H, H, D, D, D ** -0.5)
        else:
            q, k, v, i, f = _delta_views(s, H, D)
            seq_ops.mlstm(q, k, v, i, f, s["i_bias"], s["f_bias"], 15.0, D ** -0.5, s["state"], s["aux"], s["o"], H, D, D)
        return {"o": s["o"], "state": s["state"]}
    if kind == "experts":
        return state["moe"](state["hp"], 0, state["h"], state["h_act"])
    tok, probs = state["decoder"](state["model"], state["token"], state["pos"])
    return {"token": tok, "probs": probs, "memory": state["model"].layers[0].store.matrix}


# ------------------------------------------------------------------------------------------------ what a pass cannot do without

def _pairs(T, past, window):
    """(query, key) pairs of T consecutive queries after `past` positions."""
    if not window:
        return T * past + T * (T + 1) // 2
    return sum(min(past + i + 1, window) for i in range(T))


def work(case):
    kind, c = case["kind"], case
    if kind == "steps":
        live = min(c["filled"] + 1, c["slots"])
        return dict(bytes=c["layers"] * c["kv"] * c["dim"] * 2 * (2 * live + 2 + 2 * c["group"]), flops=4 * c["layers"] * c["kv"] * c["group"] * c["dim"] * live)
    if kind == "token":
        cfg = _llama_args(c)
        kvd = cfg.n_local_heads * cfg.head_dim
        n = c["layers"] * (cfg.dim * (cfg.dim + 2 * kvd) + cfg.dim * cfg.dim + 3 * cfg.dim * cfg.intermediate_size) + cfg.vocab_size * cfg.dim
        return dict(bytes=2 * n + c["layers"] * 4 * kvd * c["slots"], flops=2 * n + 4 * c["layers"] * cfg.dim * c["slots"])
    if kind == "scores":
        H = c["kv"] * c["group"]
        return dict(bytes=2 * c["tokens"] * c["dim"] * (2 * H + 2 * c["kv"]) + 4 * c["kv"] * c["tokens"], flops=4 * _pairs(c["tokens"], 0, 0) * c["dim"] * H)
    if kind == "block":
        cfg, S = _llama_args(c), c["tokens"]
        kvd = cfg.n_local_heads * cfg.head_dim
        n = cfg.dim * (cfg.dim + 2 * kvd) + cfg.dim * cfg.dim + 3 * cfg.dim * cfg.intermediate_size
        return dict(bytes=2 * n + 4 * S * cfg.dim + 4 * S * kvd, flops=2 * n * S + 4 * _pairs(S, 0, 0) * cfg.dim)
    if kind in ("rows", "rows_steps"):
        T, L, size = c.get("tokens", 1), c.get("layers", 1), 4 if c["dtype"] == "f32" else 2
        past = min(c["past"], c["window"]) if c["window"] else c["past"]
        b = T * c["heads"] * (4 * c["dk"] + size * c["dv"]) + c["kv"] * (c["dk"] + c["dv"]) * size * (past + 2 * T)
        return dict(bytes=L * b, flops=L * 2 * _pairs(T, c["past"], c["window"]) * c["heads"] * (c["dk"] + c["dv"]))
    if kind == "recurrence":
        n = c["tokens"] * c["heads"] * c["dim"]
        return dict(bytes=4 * n * (5 if c["scan"] == "wkv" else 4) + 8 * c["heads"] * c["dim"] ** 2, flops=(6 if c["scan"] == "wkv" else 8 if c["scan"] == "delta" else 5) * n * c["dim"])
    if kind == "experts":
        T, E, F = c["tokens"], c["width"], c["ff"]
        rows = 4 * T * 16 / 18                       # two of the 18 outputs are identity experts
        return dict(bytes=2 * 16 * 3 * F * E + 2 * c["shared"] * E + T * (E * (2 + 4 + 4) + 8 * c["shared"]), flops=6 * rows * F * E + 2 * T * c["shared"] * E)
    E, H, F, V = c["width"], c["heads"], c["ff"], 32000
    memory = 2 * (E * (4 * max(1, H // 2) * 128) + E * max(1, H // 2) * 128)
    full = E * (H + 2 * c["kv"]) * 128 + E * H * 128
    latent = E * 960 + 768 * H * 128 + 2 * 192 * H * 128 + E * H * 128
    n = memory + full + latent + 4 * 3 * E * F + V * E
    return dict(bytes=2 * n + 4 * c["past"] * c["kv"] * 128 + 2 * 192 * min(c["past"], 1024) + 16 * max(1, H // 2) * 128 * 128,
                flops=2 * n + 4 * c["past"] * H * 128 + 4 * min(c["past"], 1024) * H * 192)


def tolerance(case):
    kind = case["kind"]
    if kind == "rows" or kind == "rows_steps":
        return {"rel": 1e-5, "max": 1e-3} if case["dtype"] == "f32" else {"rel": 4e-3, "max": 0.05}
    return {
        "steps": {"rel": 4e-3, "max": 0.05},
        "token": {"rel": 3e-2, "max": 0.5},
        "scores": {"rel": 6e-3, "max": 0.1},
        "block": {"rel": 1e-2, "max": 0.2},
        "recurrence": {"rel": 1e-5, "max": 1e-3},
        "experts": {"rel": 4e-3, "max": 0.1},
        "design": {"rel": 2e-2, "max": 0.5, "differ": 0.01},
    }[kind]


# ------------------------------------------------------------------------------------------------ the same in 64 bits

def _attend64(q, k, v, mask_of, scale, sink=None, sink_zero=False, softcap=0.0, probs_to=None):
    """q [H, T, Dk], k/v [G, N, D] in 64 bits; mask_of(lo, hi) -> bool [hi - lo, N]; y [H, T, Dv].  probs_to(lo, hi, p [H, n, N])."""
    H, T, _ = q.shape
    G, N, Dv = v.shape
    y = torch.empty(H, T, Dv, dtype=F64, device=q.device)
    step = max(1, (1 << 27) // (N * H))
    for lo in range(0, T, step):
        hi = min(T, lo + step)
        s = torch.matmul(q[:, lo:hi].reshape(G, -1, q.shape[-1]), k.transpose(1, 2)).view(H, hi - lo, N) * scale
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        s = s.masked_fill(~mask_of(lo, hi), -math.inf)
        top = s.amax(-1, keepdim=True)
        extra = sink.double().view(H, 1, 1) if sink is not None else torch.zeros(H, 1, 1, dtype=F64, device=q.device) if sink_zero else None
        if extra is not None:
            top = torch.maximum(top, extra)
        p = torch.exp(s - top)
        den = p.sum(-1, keepdim=True)
        if extra is not None:
            den = den + torch.exp(extra - top)
        p = p / den
        if probs_to is not None:
            probs_to(lo, hi, p)
        y[:, lo:hi] = torch.matmul(p.view(G, -1, N), v).view(H, hi - lo, Dv)
    return y


def _causal(S):
    at = torch.arange(S, device=DEV)
    return lambda lo, hi: at.view(1, -1) <= at[lo:hi].view(-1, 1)


def _exact_steps(case, seed):
    caches, qkv = _steps_inputs(case, seed)
    G, D = case["group"], case["dim"]
    ys, ends = [], []
    for i, (cache, (q, k, v)) in enumerate(zip(caches, qkv)):
        H, L = cache.n_heads, cache.max_cache_length
        pos = cache.pos[0].expand(H, L).long()
        new = torch.arange(L, device=DEV).expand(H, L)
        if case["policy"] == "recent_global":
            score = pos.double().masked_fill(new < 4, math.inf)
        elif case["policy"] == "l2":
            score = (cache.key_norm.max() - cache.key_norm)[0].double()
            score = score.masked_fill((pos >= 8192 - 10) | (new < 4), math.inf).masked_fill(pos == -1, -math.inf)
        else:
            score = cache.attn_history_num[0, :, :, 0].float() / cache.attn_history_denom[0].clamp(min=1).float()
            score = score.masked_fill((pos < 4) | (pos >= 8192 - 10), 1.0).masked_fill(pos == -1, 0.0)
        idx = score.argmin(-1)
        at = torch.arange(H, device=DEV)
        kk, vv, live = cache.k_cache[0].double(), cache.v_cache[0].double(), cache.mask[0, :, 0].clone()
        kk[at, idx], vv[at, idx], live[at, idx] = k[0, :, 0].double(), v[0, :, 0].double(), True
        got = []
        y = _attend64(q[0].double(), kk, vv, lambda lo, hi: live.repeat_interleave(G, 0).unsqueeze(1), D ** -0.5, probs_to=lambda lo, hi, p: got.append(p))
        ys.append(y.unsqueeze(0))
        if i in (0, len(caches) - 1):
            end = {"k_cache": kk.unsqueeze(0), "v_cache": vv.unsqueeze(0), "pos": None}
            if hasattr(cache, "attn_history_num"):
                num = cache.attn_history_num[0, :, :, 0].clone()
                num[at, idx] = 0.0
                end["attn_history_num"] = (num + got[0].view(H, G, L).mean(1)).view(1, H, L, 1)
            ends.append(end)
    return {"y": ys, "state": ends if len(caches) > 1 else ends * 2}


def _exact_scores(case, seed):
    q, k, v = (t[0].double() for t in _scores_inputs(case, seed))
    S, kv, G = case["tokens"], case["kv"], case["group"]
    col, obs, n_obs = torch.zeros(kv, S, dtype=F64, device=DEV), torch.zeros(kv, S, dtype=F64, device=DEV), min(16, S)

    def take(lo, hi, p):
        pooled = p.view(kv, G, hi - lo, S).mean(1)
        col.add_(pooled.sum(1))
        if hi > S - n_obs:
            obs.add_(pooled[:, max(0, S - n_obs - lo):].sum(1))

    y = _attend64(q, k, v, _causal(S), case["dim"] ** -0.5, probs_to=take)
    return {"y": y.unsqueeze(0), "col_sum": col.unsqueeze(0), "obs_mean": (obs / n_obs).unsqueeze(0)}


def _exact_block(case, seed):
    cfg, block, x, freqs = _block_inputs(case, seed)
    S, H, kv, D = case["tokens"], cfg.n_head, cfg.n_local_heads, cfg.head_dim
    x, w = x[0].double(), {n: p.detach().double() for n, p in block.named_parameters()}

    def norm(t, g, eps):
        return t * torch.rsqrt(t.square().mean(-1, keepdim=True) + eps) * g

    def turn(t):
        re, im = t[..., 0::2], t[..., 1::2]
        c, s = freqs[:, None, :, 0].double(), freqs[:, None, :, 1].double()
        return torch.stack([re * c - im * s, im * c + re * s], -1).flatten(-2)

    qkv = norm(x, w["attention_norm.weight"], cfg.norm_eps) @ w["attention.wqkv.weight"].t()
    if "attention.wqkv.bias" in w:
        qkv = qkv + w["attention.wqkv.bias"]
    q, k, v = qkv.split([H * D, kv * D, kv * D], -1)
    q, k, v = turn(q.view(S, H, D)).transpose(0, 1), turn(k.view(S, kv, D)).transpose(0, 1), v.view(S, kv, D).transpose(0, 1)
    col = torch.zeros(kv, S, dtype=F64, device=DEV)
    y = _attend64(q, k, v, _causal(S), D ** -0.5, probs_to=lambda lo, hi, p: col.add_(p.view(kv, H // kv, hi - lo, S).mean(1).sum(1)))
    h = x + y.transpose(0, 1).reshape(S, H * D) @ w["attention.wo.weight"].t()
    n = norm(h, w["ffn_norm.weight"], cfg.norm_eps)
    out = h + (torch.nn.functional.silu(n @ w["feed_forward.w1.weight"].t()) * (n @ w["feed_forward.w3.weight"].t())) @ w["feed_forward.w2.weight"].t()
    res = {"y": out.unsqueeze(0), "k": k.unsqueeze(0), "v": v.unsqueeze(0), "pos": None}
    if case["policy"] == "heavy_hitter":
        res["num"] = (col / (S - torch.arange(S, device=DEV))).view(1, kv, S, 1)
    return res


def _exact_rows_layer(case, layer, T):
    cache, q, k, v, sink = layer
    p0, window = case["past"], case["window"]
    held = cache.pos[0, 0] >= 0
    at = torch.cat([cache.pos[0, 0][held].long(), p0 + torch.arange(T, device=DEV)])
    at_q = p0 + torch.arange(T, device=DEV)

    def mask_of(lo, hi):
        i, j = at_q[lo:hi].view(-1, 1), at.view(1, -1)
        return (j <= i) & (i - j < window) if window else j <= i

    kk = torch.cat([cache.k_cache[0][:, held], k.transpose(0, 1)], 1).double()
    vv = torch.cat([cache.v_cache[0][:, held], v.transpose(0, 1)], 1).double()
    return _attend64(q.double().transpose(0, 1), kk, vv, mask_of, case["dk"] ** -0.5, sink, case["sink"] == 2, case.get("softcap", 0.0)).transpose(0, 1)


def _exact_recurrence(case, seed):
    s = _recurrence_inputs(case, seed)
    T, H, D = case["tokens"], case["heads"], case["dim"]
    S, out = torch.zeros(H, D, D, dtype=F64, device=DEV), torch.empty(T, H, D, dtype=F64, device=DEV)
    if case["scan"] == "wkv":
        r, k, v = (s[n].double().view(T, H, D) for n in "rkv")
        w, u = torch.exp(-torch.exp((s["wraw"].double() + s["w0"].double()))).view(T, H, D, 1), s["u"].double()
        uk = u * k
        for t in range(T):
            out[t] = torch.einsum("hij,hi->hj", S, r[t]) + (r[t] * uk[t]).sum(-1, keepdim=True) * v[t]
            S = w[t] * S + k[t].unsqueeze(-1) * v[t].unsqueeze(-2)
        return {"o": out.view(T, H * D), "state": S}
    q, k, v, a, b = (t.double() for t in _delta_views(s, H, D))
    q, k, v = q.reshape(T, H, D), k.reshape(T, H, D), v.reshape(T, H, D)
    if case["scan"] == "delta":
        q, k = (t / torch.sqrt(t.square().sum(-1, keepdim=True) + 1e-6) for t in (q, k))
        beta, g = torch.sigmoid(a), torch.exp(-torch.exp(s["A_log"].double()) * torch.nn.functional.softplus(b + s["dt_bias"].double()))
        for t in range(T):
            S = S * g[t].view(H, 1, 1)
            S = S + k[t].unsqueeze(-1) * (beta[t].view(H, 1) * (v[t] - torch.einsum("hij,hi->hj", S, k[t]))).unsqueeze(-2)
            out[t] = torch.einsum("hij,hi->hj", S, q[t]) * D ** -0.5
        return {"o": out.view(T, H * D), "state": S}
    gi = 15.0 * torch.tanh((a + s["i_bias"].double()) / 15.0)
    gf = torch.nn.functional.logsigmoid(15.0 * torch.tanh((b + s["f_bias"].double()) / 15.0))
    n, m = torch.zeros(H, D, dtype=F64, device=DEV), torch.zeros(H, dtype=F64, device=DEV)
    for t in range(T):
        m2 = torch.maximum(gf[t] + m, gi[t])
        fw, iw = torch.exp(gf[t] + m - m2), torch.exp(gi[t] - m2)
        S = fw.view(H, 1, 1) * S + iw.view(H, 1, 1) * k[t].unsqueeze(-1) * v[t].unsqueeze(-2)
        n, m = fw.view(H, 1) * n + iw.view(H, 1) * k[t], m2
        qs = q[t] * D ** -0.5
        out[t] = torch.einsum("hij,hi->hj", S, qs) / (torch.maximum((n * qs).sum(-1).abs(), torch.exp(-m)) + 1e-6).unsqueeze(-1)
    return {"o": out.view(T, H * D), "state": S}


def _exact_experts(case, seed):
    moe, hp, h, h_act = _experts_inputs(case, seed)
    T, E, F, n = case["tokens"], case["width"], case["ff"], 18
    act = torch.nn.functional.silu
    p = torch.softmax(hp[:, :n].double(), -1)
    pick = p + moe.correction.double()
    best = pick.view(T, 6, 3).amax(-1).topk(3, -1).indices
    allowed = torch.zeros(T, 6, dtype=torch.bool, device=DEV).scatter_(1, best, True).repeat_interleave(3, 1)
    ids = pick.masked_fill(~allowed, -math.inf).topk(4, -1).indices
    wts = p.gather(1, ids)
    wts = wts / wts.sum(-1, keepdim=True)
    out = torch.zeros(T, E, dtype=F64, device=DEV)
    for e in range(n):
        t, c = (ids == e).nonzero(as_tuple=True)
        if e < 16:
            gu_rows = h_act[t].double() @ moe.w_gu[e].double().t()
            y = (act(gu_rows[:, :F]) * gu_rows[:, F:]) @ moe.w_d[e].double().t()
        else:
            y = h[t].double()
        out.index_add_(0, t, wts[t, c].unsqueeze(-1) * y)
    if case["shared"]:
        g = hp[:, n + 1:n + 1 + 2 * case["shared"]].double()
        y = (act(g[:, :case["shared"]]) * g[:, case["shared"]:]) @ moe.w_shared_down.double().t()
        out += torch.sigmoid(hp[:, n:n + 1].double()) * y
    return out


@torch.no_grad()
def exact(case, seed):
    kind = case["kind"]
    if kind == "steps":
        return _exact_steps(case, seed)
    if kind == "scores":
        return _exact_scores(case, seed)
    if kind == "block":
        return _exact_block(case, seed)
    if kind == "rows":
        return {"y": _exact_rows_layer(case, _rows_inputs(case, seed, case["tokens"])[0], case["tokens"]), "k": None, "v": None, "pos": None}
    if kind == "rows_steps":
        return {"y": [_exact_rows_layer(case, layer, 1) for layer in _rows_inputs(case, seed, 1)], "rows": None}
    if kind == "recurrence":
        return _exact_recurrence(case, seed)
    if kind == "experts":
        return _exact_experts(case, seed)
    return None          # whole models: their single layers and blocks are measured above
