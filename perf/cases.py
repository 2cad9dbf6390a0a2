"""Performance cases of the framework: the attention, expert, layer and linear work of training and of serving, through the public
entry points, at the sizes of the shipped configurations.

``listed()`` names the cases, ``draw(rng)`` gives further ones of the same ranges, ``prepare`` makes what a program has in hand
before the call, ``run`` is one pass, ``exact`` the same pass in 64-bit torch.
"""
import math

import torch

DEV = "cuda"
BF = torch.bfloat16

# heads, key / value heads of the shipped dense families (head size 128)
HEADS = [(32, 8), (28, 4), (64, 8), (32, 32), (32, 4)]
# hidden size, expert width, experts, experts per token
EXPERTS = {"qwen3_30b_a3b": (2048, 768, 128, 8), "mixtral_8x7b": (4096, 14336, 8, 2)}
# rows and columns of weights: projections of Llama-3.1-8B and of DeepSeek-V3 (multiples of 128)
WEIGHTS = [(6144, 4096), (28672, 4096), (4096, 14336), (4096, 7168), (7168, 2048), (24576, 1536)]


def listed():
    return [
        # one user's request in a serving batch of its own: the smallest call, where launches and latency count
        dict(name="decode_one", kind="decode", batch=1, heads=32, kv_heads=8, dim=128, context=700, reach=8192, block=128, cache="bf16"),
        # a full serving batch of Llama-3.1-8B between two tokens, contexts of mixed length
        dict(name="decode_batch", kind="decode", batch=64, heads=32, kv_heads=8, dim=128, context=4096, reach=8192, block=128,
             cache="bf16"),
        # the same with the int8 cache option, at the heads of Qwen2.5-7B
        dict(name="decode_int8", kind="decode", batch=48, heads=28, kv_heads=4, dim=128, context=6000, reach=8192, block=128,
             cache="int8"),
        # prompts as users send them, of any length, prefilled in one call
        dict(name="prefill_prompts", kind="prefill", seqs=6, new=2900, history=0, heads=32, kv_heads=8, dim=128, block=128, cache="bf16",
             layers=2),
        # portions of long prompts (chunked prefill): new rows behind what the cache already holds
        dict(name="prefill_portions", kind="prefill", seqs=4, new=512, history=5000, heads=32, kv_heads=8, dim=128, block=16, cache="bf16",
             layers=2),
        # DeepSeek-V3 decode with data-parallel attention: all 128 heads on one GPU
        dict(name="latent_decode", kind="latent_decode", batch=32, heads=128, context=2304, reach=4096, block=128),
        # DeepSeek-V3 prefill of prompts and portions on one of eight tensor-parallel ranks
        dict(name="latent_prefill", kind="latent_prefill", seqs=4, new=900, history=1200, heads=16, hidden=7168, block=128),
        # one layer of the Llama-3.1-8B pretraining step: forward and backward of a micro-batch
        dict(name="layer_llama", kind="layer", model="llama3_1_8b", batch=1, seq=4096, documents=0),
        # one layer of Qwen3-8B on packed documents (per-head query / key norms, attention inside documents)
        dict(name="layer_packed", kind="layer", model="qwen3_8b", batch=1, seq=2048, documents=7),
        # the expert layer of Qwen3-30B-A3B in training: forward and backward of a micro-batch
        dict(name="experts_train", kind="experts", model="qwen3_30b_a3b", tokens=4096, train=True),
        # the same layer between two tokens of a serving batch
        dict(name="experts_decode", kind="experts", model="qwen3_30b_a3b", tokens=24, train=False),
        # a linear layer on block-scaled fp8 weights in a decode step (DeepSeek-V3 checkpoints)
        dict(name="linear_fp8", kind="linear", format="fp8", tokens=32, rows=4096, cols=7168),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "prefill", "prefill", "latent_decode", "latent_prefill", "layer", "layer", "experts",
                       "experts", "linear"])
    if kind == "decode":
        h, g = rng.choice(HEADS)
        context = _log(rng, 64, 8192)
        return dict(kind=kind, batch=max(1, min(_log(rng, 1, 128), 400000 * 8 // (context * g))), heads=h, kv_heads=g, dim=128,
                    context=context, reach=rng.choice([8192, 32768]), block=rng.choice([16, 64, 128]), cache=rng.choice(["bf16", "int8"]))
    if kind == "prefill":
        h, g = rng.choice(HEADS)
        new = _log(rng, 24, 3000)
        return dict(kind=kind, seqs=max(1, min(rng.randint(1, 8), 12000 // new)), new=new, history=rng.choice([0, _log(rng, 100, 6000)]),
                    heads=h, kv_heads=g, dim=128, block=rng.choice([16, 64, 128]), cache=rng.choice(["bf16", "bf16", "int8"]), layers=2)
    if kind == "latent_decode":
        context = _log(rng, 100, 4096)
        return dict(kind=kind, batch=max(1, min(_log(rng, 1, 128), 200000 // context)), heads=rng.choice([16, 32, 64, 128]),
                    context=context, reach=4096, block=rng.choice([16, 64, 128]))
    if kind == "latent_prefill":
        new = _log(rng, 24, 1500)
        return dict(kind=kind, seqs=max(1, min(rng.randint(1, 6), 4000 // new)), new=new, history=rng.choice([0, _log(rng, 100, 1500)]),
                    heads=rng.choice([16, 32]), hidden=7168, block=rng.choice([16, 64, 128]))
    if kind == "layer":
        batch, seq = rng.choice([1, 1, 2]), rng.randint(2, 16) * 128
        return dict(kind=kind, model=rng.choice(["llama3_1_8b", "qwen3_8b", "qwen2_5_7b"]), batch=batch, seq=seq,
                    documents=rng.choice([0, rng.randint(2, 12)]))
    if kind == "experts":
        model = rng.choice(list(EXPERTS))
        if rng.random() < 0.5:
            return dict(kind=kind, model=model, tokens=_log(rng, 1, 256), train=False)
        return dict(kind=kind, model=model, tokens=_log(rng, 300, 4096 if model == "qwen3_30b_a3b" else 1500), train=True)
    n, k = rng.choice(WEIGHTS)
    return dict(kind=kind, format=rng.choice(["bf16", "fp8", "int8"]), tokens=_log(rng, 1, 4000), rows=n, cols=k)


# ---------------------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed), torch.Generator().manual_seed(seed)


def _randn(g, *shape, dtype=BF, scale=1.0):
    return torch.randn(*shape, generator=g, device=DEV, dtype=torch.float32).mul_(scale).to(dtype)


def _lens(g, n, most, least):
    """``n`` lengths, the first ``most``, the others between ``least`` and ``most``."""
    return [most] + torch.randint(max(1, least), most + 1, (n - 1,), generator=g).tolist()


def _history(case, g):
    h = case["history"]
    return _lens(g, case["seqs"], h, h // 2) if h else [0] * case["seqs"]


def _pages(g, lens, block, reach):
    """Block tables ``[B, reach / block]`` (-1 where a sequence has no block) from a pool in random order that could hold every
    sequence at the longest length, and the pool's number of blocks."""
    need = [-(-n // block) for n in lens]
    pool = len(lens) * max(need)
    order = torch.randperm(pool, generator=g).to(torch.int32)
    tables = torch.full((len(lens), -(-reach // block)), -1, dtype=torch.int32)
    at = 0
    for b, n in enumerate(need):
        tables[b, :n] = order[at:at + n]
        at += n
    return tables, pool


def _slots(tables, block, lens, new):
    """The cache slots of the last ``new[b]`` of ``lens[b]`` tokens."""
    out = []
    for b, (n, m) in enumerate(zip(lens, new)):
        pos = torch.arange(n - m, n)
        out.append(tables[b, pos // block].long() * block + pos % block)
    return torch.cat(out).to(torch.int32)


def _fill(ctx, g, int8):
    """What earlier steps left in the cache."""
    for layer in range(len(ctx.key_cache)):
        for name in ("key", "value"):
            cache = getattr(ctx, name + "_cache")[layer]
            if cache is None:
                continue
            if not int8:
                for rows in cache.split(256):
                    rows.copy_(_randn(g, *rows.shape))
                continue
            scale = getattr(ctx, name + "_scale")[layer]
            for rows, sc in zip(cache.split(256), scale.split(256)):
                x = _randn(g, *rows.shape, dtype=torch.float32)
                s = x.abs().amax(-1) / 127.0
                sc.copy_(s)
                rows.copy_(torch.round(x / s.unsqueeze(-1)).clamp_(-127, 127).to(torch.int8))


def _step(case, gc):
    """Lengths, pages and slots of one serving step: one new token per sequence (decode) or a portion each. The lengths
    belong to the case, the pages to the generator."""
    block = case["block"]
    sizes = torch.Generator().manual_seed(case.get("batch", 0) + 1000 * case.get("context", 0) + 7 * case.get("new", 0)
                                          + 100003 * case.get("history", 0) + 13 * case.get("seqs", 0))
    if case["kind"] in ("decode", "latent_decode"):
        lens = _lens(sizes, case["batch"], case["context"], case["context"] // 2)
        new = [1] * len(lens)
        tables, blocks = _pages(gc, lens, block, case["reach"])
        prefill = False
    else:
        hist = _history(case, sizes)
        new = _lens(sizes, case["seqs"], case["new"], case["new"] // 4)
        lens = [h + n for h, n in zip(hist, new)]
        tables, blocks = _pages(gc, lens, block, max(lens))
        prefill = True
    return lens, new, blocks, dict(is_prefill=prefill, block_tables=tables.numpy(), slot_mapping=_slots(tables, block, lens, new).numpy(),
                                   context_lens=lens, q_seq_lens=new, device=DEV)


def _config(name, **over):
    from mindformers_b200.models.presets import get_preset, preset_is_mla
    from mindformers_b200.parallel.transformer_config_utils import convert_to_transformer_config
    cfg = get_preset(name, **over)
    cfg.update(params_dtype="bfloat16", compute_dtype="bfloat16")
    out = convert_to_transformer_config(cfg, is_mla_model=preset_is_mla(cfg))
    out.device = DEV
    return out


def _vary_norms(module, g):
    """Norm weights of a trained model are not all one."""
    with torch.no_grad():
        for name, p in module.named_parameters():
            if "layernorm" in name:
                p.copy_(1.0 + 0.1 * torch.randn(p.shape, generator=g, device=DEV))


def prepare(case, seed):
    g, gc = _gen(seed)
    torch.manual_seed(seed)
    s = {"case": dict(case)}
    kind = case["kind"]
    if kind in ("decode", "prefill"):
        from mindformers_b200.inference.paged_attention import KVCacheContext
        from mindformers_b200.parallel.layers.attention import AttnMeta
        H, G, D, int8 = case["heads"], case["kv_heads"], case["dim"], case["cache"] == "int8"
        lens, new, blocks, step = _step(case, gc)
        layers = case.get("layers", 1)
        ctx = KVCacheContext(layers, blocks, case["block"], G, D, BF, DEV, kv_cache_dtype="int8" if int8 else None)
        _fill(ctx, g, int8)
        s.update(ctx=ctx, step=step, lens=lens, new=new, meta=AttnMeta(batch=1, seq_len=sum(new), cache=ctx))
        s["qkv"] = [_randn(g, sum(new), H + 2 * G, D) for _ in range(layers)]      # as the fused projection leaves them
        if kind == "decode":
            ctx.set_step(**step)
    elif kind == "latent_decode":
        lens, _, blocks, step = _step(case, gc)
        s["cache"] = torch.empty(blocks, case["block"], 1, 576, dtype=BF, device=DEV)
        for rows in s["cache"].split(256):
            rows.copy_(_randn(g, *rows.shape))
        s["q"] = _randn(g, case["batch"], case["heads"], 576)
        s["tables"] = torch.as_tensor(step["block_tables"]).to(DEV)
        s["ctx_lens"] = torch.tensor(lens, dtype=torch.int32, device=DEV)
        s["lens"], s["holder"] = lens, type("Holder", (), {})()
    elif kind == "latent_prefill":
        from mindformers_b200.inference.paged_attention import KVCacheContext
        from mindformers_b200.parallel.layers.attention import AttnMeta, MLASelfAttention
        from mindformers_b200.parallel.layers.rotary import get_rope
        cfg = _config("deepseek_v3", num_attention_heads=case["heads"], num_key_value_heads=case["heads"], hidden_size=case["hidden"],
                      max_position_embeddings=8192)
        s["layer"] = MLASelfAttention(cfg).eval()
        _vary_norms(s["layer"], g)
        lens, new, blocks, step = _step(case, gc)
        ctx = KVCacheContext(1, blocks, case["block"], 1, 0, BF, DEV, mla_latent_dim=576)
        _fill(ctx, g, False)
        pos = torch.cat([torch.arange(n - m, n) for n, m in zip(lens, new)]).to(DEV)
        s.update(ctx=ctx, step=step, lens=lens, new=new, rotary=get_rope(cfg, device=DEV)(),
                 meta=AttnMeta(batch=1, seq_len=sum(new), positions=pos, cache=ctx))
        s["x"] = _randn(g, sum(new), case["hidden"])
    elif kind == "layer":
        from mindformers_b200.parallel.distributed.param_grad_buffer import build_buffers
        from mindformers_b200.parallel.layers.rotary import get_rope
        from mindformers_b200.parallel.layers.transformer_layer import TransformerLayer
        B, S = case["batch"], case["seq"]
        cfg = _config(case["model"], seq_length=S, max_position_embeddings=8192)
        layer = s["layer"] = TransformerLayer(cfg, 1).train()
        _vary_norms(layer, g)
        s["buffers"] = build_buffers(layer, tp=1, sequence_parallel=False)
        s["rotary"] = get_rope(cfg, device=DEV)()
        s["positions"] = torch.arange(S, device=DEV).repeat(B)
        s["ends"] = None
        if case["documents"]:
            cuts = [sorted(torch.randperm(S - 1, generator=gc)[:case["documents"] - 1].add(1).tolist()) + [S] for _ in range(B)]
            s["ends"] = torch.tensor(cuts, dtype=torch.int64, device=DEV)
        s["x"] = [_randn(g, B * S, cfg.hidden_size).requires_grad_() for _ in range(2)]
        s["dout"] = [_randn(g, B * S, cfg.hidden_size) for _ in range(2)]
    elif kind == "experts":
        from mindformers_b200.parallel.distributed.param_grad_buffer import build_buffers
        from mindformers_b200.parallel.layers.moe import MoELayer
        H, F, E, K = EXPERTS[case["model"]]
        cfg = _config("qwen3_30b_a3b", hidden_size=H, moe_intermediate_size=F, num_experts=E, num_experts_per_tok=K)
        layer = s["layer"] = MoELayer(cfg).train(case["train"])
        s["x"] = _randn(g, case["tokens"], H)
        if case["train"]:
            s["buffers"] = build_buffers(layer, tp=1, sequence_parallel=False)
            s["x"].requires_grad_()
            s["dout"] = _randn(g, case["tokens"], H)
    else:
        from mindformers_b200.ops import functional as Fn
        n, k = case["rows"], case["cols"]
        w = _randn(g, n, k, scale=0.02)
        s["x"] = _randn(g, case["tokens"], k)
        if case["format"] == "fp8":
            s["w"], s["scale"] = Fn.quantize_weight_128x128(w)
        elif case["format"] == "int8":
            s["scale"] = w.float().abs().amax(1) / 127.0
            s["w"] = torch.round(w.float() / s["scale"].unsqueeze(1)).clamp_(-127, 127).to(torch.int8)
        else:
            s["w"] = w
    return s


# ---------------------------------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------------------------------
def _grads(module, buffers):
    for b in buffers.values():
        b.collect_autograd_grads()
    return {n: p.main_grad for n, p in module.named_parameters()}


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind in ("decode", "prefill"):
        from mindformers_b200.inference.paged_attention import paged_attention_forward
        H, G, ctx = case["heads"], case["kv_heads"], s["ctx"]
        if kind == "prefill":
            ctx.set_step(**s["step"])
        with torch.no_grad():
            out = [paged_attention_forward(x[:, :H], x[:, H:H + G], x[:, H + G:], s["meta"], i + 1, case["dim"] ** -0.5)
                   for i, x in enumerate(s["qkv"])]
        res = {"out": out, "keys": ctx.key_cache, "values": ctx.value_cache}
        if case["cache"] == "int8":
            res["scales"] = [ctx.key_scale, ctx.value_scale]
        return res
    if kind == "latent_decode":
        from mindformers_b200.inference.paged_attention import mla_decode_attention
        return mla_decode_attention(s["q"], s["cache"], s["tables"], s["ctx_lens"], case["block"], 192 ** -0.5, s["holder"])
    if kind == "latent_prefill":
        with torch.no_grad():
            s["ctx"].set_step(**s["step"])
            return {"out": s["layer"](s["x"], s["rotary"], s["meta"])[0], "cache": s["ctx"].key_cache}
    if kind == "layer":
        from mindformers_b200.parallel.layers.attention import AttnMeta
        meta = AttnMeta(batch=case["batch"], seq_len=case["seq"], positions=s["positions"], actual_seq_len=s["ends"])
        for x in s["x"]:
            x.grad = None
        out, residual, _ = s["layer"](s["x"][0], s["x"][1], s["rotary"], meta)
        torch.autograd.backward([out, residual], s["dout"])
        return {"out": out, "residual": residual, "dx": [x.grad for x in s["x"]], "grads": _grads(s["layer"], s["buffers"])}
    if kind == "experts":
        if not case["train"]:
            with torch.no_grad():
                return s["layer"](s["x"])[0]
        s["x"].grad = None
        out, aux = s["layer"](s["x"])
        torch.autograd.backward([out, aux], [s["dout"], torch.ones_like(aux)])
        return {"out": out, "aux": aux, "dx": s["x"].grad, "grads": _grads(s["layer"], s["buffers"])}
    from mindformers_b200.ops import functional as Fn
    with torch.no_grad():
        if case["format"] == "fp8":
            return Fn.fp8_linear(s["x"], s["w"], s["scale"])
        if case["format"] == "int8":
            return Fn.w8a8_linear(s["x"], s["w"], s["scale"])
        return Fn.linear(s["x"], s["w"])


# ---------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------------------------------
def _pairs(case):
    """Keys read, new rows and query-key pairs of a serving step."""
    lens, new, _, _ = _step(case, torch.Generator())
    return sum(lens), sum(new), sum(m * (n - m) + m * (m + 1) // 2 for n, m in zip(lens, new))


def work(case):
    kind = case["kind"]
    if kind in ("decode", "prefill"):
        H, G, D, layers = case["heads"], case["kv_heads"], case["dim"], case.get("layers", 1)
        keys, rows, pairs = _pairs(case)
        row = G * (D + 4) if case["cache"] == "int8" else 2 * G * D
        return {"bytes": layers * (2 * keys * row + rows * (2 * row + 4 * H * D + 4 * G * D)), "flops": layers * 4 * pairs * H * D}
    if kind == "latent_decode":
        keys, rows, pairs = _pairs(case)
        H = case["heads"]
        return {"bytes": keys * 1152 + rows * H * (576 + 512) * 2, "flops": 2 * pairs * H * (576 + 512)}
    if kind == "latent_prefill":
        keys, rows, pairs = _pairs(case)
        H, W = case["heads"], case["hidden"]
        weights = W * 2112 + 1536 * H * 192 + 512 * H * 256 + H * 128 * W
        return {"bytes": 2 * weights + keys * 1152 + rows * W * 4,
                "flops": 2 * rows * (weights - 512 * H * 256) + 2 * keys * 512 * H * 256 + 2 * pairs * H * 320}
    if kind == "layer":
        p = {"llama3_1_8b": (4096, 32, 8, 14336), "qwen3_8b": (4096, 32, 8, 12288), "qwen2_5_7b": (3584, 28, 4, 18944)}[case["model"]]
        W, H, G, F = p
        T = case["batch"] * case["seq"]
        weights = W * (H + 2 * G) * 128 + H * 128 * W + 3 * W * F
        pairs = T * case["seq"] // 2 // max(1, case["documents"])
        return {"bytes": weights * (2 + 8) + T * W * 2 * 8, "flops": 6 * T * weights + 14 * pairs * H * 128}
    if kind == "experts":
        W, F, E, K = EXPERTS[case["model"]]
        T = case["tokens"]
        used = E * (1 - (1 - K / E) ** T)
        if case["train"]:
            return {"bytes": used * 3 * W * F * (2 + 8) + T * W * 2 * 4, "flops": 18 * T * K * W * F + 6 * T * W * E}
        return {"bytes": used * 3 * W * F * 2 + T * W * 4 + W * E * 4, "flops": 6 * T * K * W * F + 2 * T * W * E}
    T, n, k = case["tokens"], case["rows"], case["cols"]
    return {"bytes": n * k * (2 if case["format"] == "bf16" else 1) + 2 * T * (n + k), "flops": 2 * T * n * k}


def tolerance(case):
    kind = case["kind"]
    if kind in ("decode", "prefill"):
        return {"rel": 0.01, "differ": 0.0001}
    if kind == "latent_decode":
        return {"rel": 0.01}
    if kind == "latent_prefill":      # the 16-bit query, latent and key before the softmax alone: 0.02 off the 64-bit result
        return {"rel": 0.03}
    if kind == "layer":               # a norm weight's gradient sums terms that cancel: 0.026 off the 64-bit one, the others 0.006
        return {"rel": 0.03, "max": 0.5}
    if kind == "experts":
        return {"rel": 0.018, "max": 0.5}
    return {"rel": 0.01}


# ---------------------------------------------------------------------------------------------------------------------
# the same pass in 64 bits
# ---------------------------------------------------------------------------------------------------------------------
def _attend(q, k, v, scale, offset, start=None):
    """q ``[n, H, D]`` at positions ``offset ..`` of k / v ``[L, G, D]``, causal; ``start [n]``: first visible key of every row."""
    n, H, D = q.shape
    L, G, _ = k.shape
    kp = torch.arange(L, device=q.device)
    qp = torch.arange(n, device=q.device) + offset
    hide = kp[None, :] > qp[:, None]
    if start is not None:
        hide = hide | (kp[None, :] < start[:, None])
    out = []
    for h in range(H):
        j = h // (H // G)
        sc = (q[:, h] @ k[:, j].t()) * scale
        out.append(torch.softmax(sc.masked_fill(hide, float("-inf")), -1) @ v[:, j])
    return torch.stack(out, 1)


def _rms(x, w, eps):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w


def _angles(dim, base, positions, scaling=None):
    i = torch.arange(0, dim, 2, dtype=torch.float64, device=DEV)
    inv = base ** (-i / dim)
    if scaling == "llama3":          # factor 8, low 1, high 4, original length 8192
        wave = 2 * math.pi / inv
        smooth = ((8192 / wave - 1) / 3).clamp(0, 1)
        inv = (1 - smooth) * inv / 8 + smooth * inv
    elif scaling == "yarn":          # factor 40, fast 32, slow 1, original length 4096
        turn = lambda n: dim * math.log(4096 / (n * 2 * math.pi)) / (2 * math.log(base))
        lo, hi = max(math.floor(turn(32)), 0), min(math.ceil(turn(1)), dim - 1)
        ramp = ((i / 2 - lo) / (hi - lo)).clamp(0, 1)
        inv = inv / 40 * ramp + inv * (1 - ramp)
    ang = positions.double()[:, None] * inv[None]
    return ang.cos()[:, None], ang.sin()[:, None]


def _rotate(x, cos, sin, pairs=False):
    if pairs:
        a, b = x[..., 0::2], x[..., 1::2]
        return torch.stack((a * cos - b * sin, b * cos + a * sin), -1).flatten(-2)
    a, b = x.chunk(2, -1)
    return torch.cat((a * cos - b * sin, b * cos + a * sin), -1)


def _cached(cache, scale, tables, b, n, block):
    rows = cache[tables[b, :-(-n // block)].long()].flatten(0, 1)[:n].double()
    return rows if scale is None else rows * scale[tables[b, :-(-n // block)].long()].flatten(0, 1)[:n].double().unsqueeze(-1)


def _store(ctx, layer, step, k, v, int8):
    """The step's rows in a copy of the cache, as the cache's format has them."""
    slots = torch.as_tensor(step["slot_mapping"]).long().to(DEV)
    out = []
    for name, x in (("key", k), ("value", v)):
        cache = getattr(ctx, name + "_cache")[layer].clone()
        scale = None
        if int8:
            scale = getattr(ctx, name + "_scale")[layer].clone()
            amax = x.float().abs().amax(-1)
            sc = torch.where(amax > 0, amax / 127.0, torch.ones_like(amax))
            scale.flatten(0, 1)[slots] = sc
            x = torch.round(x.float() / sc.unsqueeze(-1)).clamp(-127, 127).to(torch.int8)
        cache.flatten(0, 1)[slots] = x
        out += [cache, scale]
    return out


def _exact_step(case, s):
    H, G, int8, ctx, block = case["heads"], case["kv_heads"], case["cache"] == "int8", s["ctx"], case["block"]
    tables = torch.as_tensor(s["step"]["block_tables"]).to(DEV)
    outs = []
    for layer, x in enumerate(s["qkv"]):
        q, k, v = x[:, :H], x[:, H:H + G], x[:, H + G:]
        kc, ks, vc, vs = _store(ctx, layer, s["step"], k, v, int8)
        res, at = [], 0
        for b, (n, m) in enumerate(zip(s["lens"], s["new"])):
            rows = slice(at, at + m)
            at += m
            if n == m and case["kind"] == "prefill":          # nothing cached before: the rows themselves, not what the cache keeps
                kk, vv = k[rows].double(), v[rows].double()
            else:
                kk, vv = _cached(kc, ks, tables, b, n, block), _cached(vc, vs, tables, b, n, block)
            res.append(_attend(q[rows].double(), kk, vv, case["dim"] ** -0.5, n - m))
        outs.append(torch.cat(res).flatten(1))
    out = {"out": outs, "keys": None, "values": None}
    if int8:
        out["scales"] = None
    return out


def _exact_latent_prefill(case, s):
    H = case["heads"]
    w = {n: p.double() for n, p in s["layer"].named_parameters()}
    x = s["x"].double() @ w["linear_qkv.weight"].t()
    qc, kvc, kpe = x.split([1536, 512, 64], -1)
    q = (_rms(qc, w["q_layernorm.weight"], 1e-6) @ w["linear_qb.weight"].t()).view(-1, H, 192)
    cos, sin = _angles(64, 10000.0, s["meta"].positions, "yarn")
    q = torch.cat((q[..., :128], _rotate(q[..., 128:], cos, sin, True)), -1)
    new = torch.cat((_rms(kvc, w["k_layernorm.weight"], 1e-6), _rotate(kpe[:, None], cos, sin, True)[:, 0]), -1)
    tables = torch.as_tensor(s["step"]["block_tables"]).to(DEV)
    m = 0.1 * math.log(40.0) + 1.0
    out, at = [], 0
    for b, (n, k) in enumerate(zip(s["lens"], s["new"])):
        lat = torch.cat((_cached(s["ctx"].key_cache[0], None, tables, b, n, case["block"])[:n - k, 0], new[at:at + k]))
        kv = (lat[:, :512] @ w["linear_kvb.weight"].t()).view(n, H, 256)
        keys = torch.cat((kv[..., :128], lat[:, None, 512:].expand(n, H, 64)), -1)
        out.append(_attend(q[at:at + k], keys, kv[..., 128:], m * m * 192 ** -0.5, n - k).flatten(1))
        at += k
    return {"out": torch.cat(out) @ w["linear_proj.weight"].t(), "cache": None}


def _exact_layer(case, s):
    model = case["model"]
    W, H, G, eps, base, scaling = {"llama3_1_8b": (4096, 32, 8, 1e-5, 500000.0, "llama3"), "qwen3_8b": (4096, 32, 8, 1e-6, 1e6, None),
                                   "qwen2_5_7b": (3584, 28, 4, 1e-6, 1e6, None)}[model]
    B, S = case["batch"], case["seq"]
    w = {n: p.detach().double().requires_grad_() for n, p in s["layer"].named_parameters()}
    x = [t.detach().double().requires_grad_() for t in s["x"]]
    res = x[0] + x[1]
    qkv = _rms(res, w["input_layernorm.weight"], eps) @ w["self_attention.linear_qkv.weight"].t()
    if "self_attention.linear_qkv.bias" in w:
        qkv = qkv + w["self_attention.linear_qkv.bias"]
    q, k, v = qkv.view(B * S, H + 2 * G, 128).split([H, G, G], 1)
    if "self_attention.q_layernorm.weight" in w:
        q, k = _rms(q, w["self_attention.q_layernorm.weight"], eps), _rms(k, w["self_attention.k_layernorm.weight"], eps)
    cos, sin = _angles(128, base, s["positions"], scaling)
    q, k = _rotate(q, cos, sin), _rotate(k, cos, sin)
    att = []
    for b in range(B):
        r, start = slice(b * S, (b + 1) * S), None
        if s["ends"] is not None:
            ends = s["ends"][b]
            at = torch.searchsorted(ends, torch.arange(S, device=DEV), right=True)
            start = torch.cat((ends.new_zeros(1), ends))[at]
        att.append(_attend(q[r], k[r], v[r], 128 ** -0.5, 0, start).flatten(1))
    y = torch.cat(att) @ w["self_attention.linear_proj.weight"].t()
    residual = res + y
    gate, up = (_rms(residual, w["pre_mlp_layernorm.weight"], eps) @ w["mlp.linear_fc1.weight"].t()).chunk(2, -1)
    out = (torch.nn.functional.silu(gate) * up) @ w["mlp.linear_fc2.weight"].t()
    torch.autograd.backward([out, residual], [t.double() for t in s["dout"]])
    return {"out": out.detach(), "residual": residual.detach(), "dx": [t.grad for t in x], "grads": {n: p.grad for n, p in w.items()}}


def _exact_experts(case, s):
    E, K = EXPERTS[case["model"]][2:]
    train = case["train"]
    w = {n: p.detach().double().requires_grad_(train) for n, p in s["layer"].named_parameters()}
    x = s["x"].detach().double().requires_grad_(train)
    scores = torch.softmax(x @ w["router.weight"].t(), -1)
    probs, ids = scores.topk(K, -1)
    probs = probs / probs.sum(-1, keepdim=True)
    out = torch.zeros_like(x)
    for e in range(E):
        t, j = (ids == e).nonzero(as_tuple=True)
        if t.numel():
            gate, up = (x[t] @ w["experts.weight1"][e]).chunk(2, -1)
            y = (torch.nn.functional.silu(gate) * up) @ w["experts.weight2"][e]
            out = out.index_add(0, t, y * probs[t, j, None])
    if not train:
        return out
    share = torch.bincount(ids.flatten(), minlength=E).double() / ids.numel()
    aux = 1e-3 * E * (scores.mean(0) * share).sum()
    torch.autograd.backward([out, aux], [s["dout"].double(), torch.ones_like(aux)])
    return {"out": out.detach(), "aux": aux.detach(), "dx": x.grad, "grads": {n: p.grad for n, p in w.items()}}


def _exact_linear(case, s):
    x, w = s["x"].double(), s["w"].double()
    if case["format"] == "fp8":
        blocks = s["x"].float().unflatten(1, (-1, 128))           # the format's own rounding of the activations
        amax = blocks.abs().amax(-1, keepdim=True)
        sc = torch.where(amax > 0, amax / 448.0, torch.ones_like(amax))
        x = ((blocks / sc).clamp(-448, 448).to(torch.float8_e4m3fn).double() * sc.double()).flatten(1)
        n, k = w.shape
        w = (w.view(n // 128, 128, k // 128, 128) * s["scale"].double()[:, None, :, None]).view(n, k)
    elif case["format"] == "int8":
        amax = s["x"].float().abs().amax(1, keepdim=True)
        sc = torch.where(amax > 0, amax / 127.0, torch.ones_like(amax))
        x = torch.round(s["x"].float() / sc).clamp(-127, 127).double() * sc.double()
        w = w * s["scale"].double()[:, None]
    return x @ w.t()


def exact(case, seed):
    s = prepare(case, seed)
    kind = case["kind"]
    if kind in ("decode", "prefill"):
        return _exact_step(case, s)
    if kind == "latent_decode":
        out = []
        for b, n in enumerate(s["lens"]):
            lat = _cached(s["cache"], None, s["tables"], b, n, case["block"])[:, 0]
            p = torch.softmax((s["q"][b].double() @ lat.t()) * 192 ** -0.5, -1)
            out.append(p @ lat[:, :512])
        return torch.stack(out)
    if kind == "latent_prefill":
        return _exact_latent_prefill(case, s)
    if kind == "layer":
        return _exact_layer(case, s)
    if kind == "experts":
        return _exact_experts(case, s)
    return _exact_linear(case, s)
