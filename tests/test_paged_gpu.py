"""Attention over the paged cache on the tensor cores (ragged prefill, decode over int8 rows), against 64-bit PyTorch."""
import copy
import types

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _attend(q, k, v, scale):
    """Causal attention of the last rows of a sequence in 64 bits: q [n, H, D], k / v [L, G, D]."""
    n, H, _ = q.shape
    L, G, _ = k.shape
    k, v = (t.double().repeat_interleave(H // G, 1) for t in (k, v))
    s = torch.einsum("qhd,khd->hqk", q.double(), k) * scale
    hide = torch.arange(L, device=DEV)[None] > torch.arange(L - n, L, device=DEV)[:, None]
    return torch.einsum("hqk,khd->qhd", torch.softmax(s.masked_fill(hide, float("-inf")), -1), v).flatten(1)


def _tables(lens, block):
    need = [-(-n // block) for n in lens]
    order = torch.randperm(sum(need)).to(torch.int32)
    tables = torch.full((len(lens), max(need) + 1), -1, dtype=torch.int32)
    at = 0
    for b, n in enumerate(need):
        tables[b, :n] = order[at:at + n]
        at += n
    return tables, sum(need)


def _slots(tables, block, lens, news):
    out = []
    for b, (n, m) in enumerate(zip(lens, news)):
        pos = torch.arange(n - m, n)
        out.append(tables[b, pos // block].long() * block + pos % block)
    return torch.cat(out)


def _cached(rows, tables, b, n, block):
    return rows[tables[b, :-(-n // block)].long().to(DEV)].flatten(0, 1)[:n]


# lengths at the edges of the 128-row tiles, sequences without new rows and with one, histories of all kinds in one batch
NEWS = [[1, 127, 0, 300], [128, 129, 1, 64], [257, 5]]
PAST = [[0, 0, 0, 0], [700, 129, 64, 0], [128, 1]]


@pytest.mark.parametrize("step", range(3))
@pytest.mark.parametrize("heads,kv,dim", [(8, 2, 128), (7, 1, 128), (4, 4, 64)])
@pytest.mark.parametrize("block,int8", [(16, False), (128, False), (64, True), (24, False)])
def test_ragged_prefill(step, heads, kv, dim, block, int8):
    from mindformers_b200.inference import paged_attention as pa
    from mindformers_b200.ops import _lib
    torch.manual_seed(step)
    news, past = NEWS[step], PAST[step]
    lens = [n + p for n, p in zip(news, past)]
    tables, blocks = _tables(lens, block)
    ctx = pa.KVCacheContext(1, blocks, block, kv, dim, torch.bfloat16, DEV, kv_cache_dtype="int8" if int8 else None)
    T = sum(news)
    qkv = torch.randn(T, heads + 2 * kv, dim, device=DEV).to(torch.bfloat16)
    q, k, v = qkv[:, :heads], qkv[:, heads:heads + kv], qkv[:, heads + kv:]
    hist = torch.randn(2, sum(lens), kv, dim, device=DEV).to(torch.bfloat16)
    step_meta = dict(block_tables=tables.numpy(), context_lens=lens, device=DEV)
    if not int8:                       # what earlier users of the pages left behind has no effect
        ctx.key_cache[0].fill_(float("nan"))
        ctx.value_cache[0].fill_(float("inf"))
    ctx.set_step(is_prefill=True, slot_mapping=_slots(tables, block, lens, lens).numpy(), q_seq_lens=lens, **step_meta)
    pa._write_cache(ctx, 0, hist[0], hist[1])
    ctx.set_step(is_prefill=True, slot_mapping=_slots(tables, block, lens, news).numpy(), q_seq_lens=news, **step_meta)
    meta = types.SimpleNamespace(cache=ctx)
    before = _lib.launch_count()
    with torch.no_grad():
        got = pa.paged_attention_forward(q, k, v, meta, 1, dim ** -0.5)
        again = pa.paged_attention_forward(q, k, v, meta, 1, dim ** -0.5)
    assert _lib.launch_count() > before + 2 and got.shape == (T, heads * dim)
    assert torch.equal(got, again)
    at = 0
    for b, (n, m) in enumerate(zip(news, lens)):
        rows = slice(at, at + n)
        at += n
        if not n:
            continue
        if n == m:
            kk, vv = k[rows], v[rows]
        else:
            sc = pa._layer_scales(ctx, 0)
            kk, vv = (pa._gather(c[0], tables[b].to(DEV), m, block, s, torch.bfloat16)
                      for c, s in zip((ctx.key_cache, ctx.value_cache), sc))
        want = _attend(q[rows], kk, vv, dim ** -0.5)
        err = (got[rows].double() - want).norm() / want.norm()
        # rounding of the result alone: at most 2^-8 of a number, 1.5e-3 to 1.7e-3 in the mean square of many; the weights of
        # sequences without history are rounded too
        assert err < (2e-3 if n < m else 4e-3), (b, float(err))
    assert _lib.read_status() == 0


@pytest.mark.parametrize("step", range(3))
@pytest.mark.parametrize("heads,block,share", [(16, 128, 1 << 30), (3, 16, 1 << 30), (5, 64, 1)])
def test_latent_prefill(step, heads, block, share, monkeypatch):
    """``share``: bytes of expanded keys and values at a time (1: head by head)."""
    from mindformers_b200.inference import paged_attention as pa
    from mindformers_b200.ops import _lib
    torch.manual_seed(step)
    monkeypatch.setattr(pa, "_EXPANDED_BYTES", share)
    news, past = NEWS[step], PAST[step]
    lens = [n + p for n, p in zip(news, past)]
    tables, blocks = _tables(lens, block)
    ctx = pa.KVCacheContext(1, blocks, block, 1, 0, torch.bfloat16, DEV, mla_latent_dim=576)
    ctx.key_cache[0].fill_(float("nan"))
    w = (torch.randn(heads * 256, 512, device=DEV) * 512 ** -0.5).to(torch.bfloat16)
    attn = types.SimpleNamespace(nh=heads, nope=128, rope_d=64, vd=128, kv_rank=512, layer_number=1, scale=192 ** -0.5,
                                 linear_kvb=types.SimpleNamespace(weight=w))
    T = sum(news)
    q = torch.randn(T, heads, 192, device=DEV).to(torch.bfloat16)
    lat = torch.randn(sum(lens), 576, device=DEV).to(torch.bfloat16)
    step_meta = dict(block_tables=tables.numpy(), context_lens=lens, device=DEV)
    ctx.set_step(is_prefill=True, slot_mapping=_slots(tables, block, lens, lens).numpy(), q_seq_lens=lens, **step_meta)
    pa._write_cache(ctx, 0, lat.unsqueeze(1), None)
    ctx.set_step(is_prefill=True, slot_mapping=_slots(tables, block, lens, news).numpy(), q_seq_lens=news, **step_meta)
    new = torch.randn(T, 576, device=DEV).to(torch.bfloat16)
    q_pe = q[..., 128:].clone()
    with torch.no_grad():
        got = pa.mla_paged_attention_forward(attn, q[..., :128], q_pe, new[:, :512], new[:, 512:], types.SimpleNamespace(cache=ctx))
    assert got.shape == (T, heads * 128)
    at = 0
    for b, (n, m) in enumerate(zip(news, lens)):
        rows = slice(at, at + n)
        at += n
        if not n:
            continue
        lt = _cached(ctx.key_cache[0][:, :, 0], tables, b, m, block).double()
        kv = (lt[:, :512] @ w.double().t()).view(m, heads, 256)
        keys = torch.cat((kv[..., :128], lt[:, None, 512:].expand(m, heads, 64)), -1)
        want = _attend(q[rows], keys, kv[..., 128:], attn.scale)
        err = (got[rows].double() - want).norm() / want.norm()
        assert err < 2e-3, (b, float(err))         # rounding of the result alone
    assert _lib.read_status() == 0


# context lengths at the edges of a warp's 16 tokens and a round's 64, one of many splits, an idle row without blocks
@pytest.mark.parametrize("heads,kv,dim", [(8, 8, 128), (14, 2, 128), (8, 1, 64), (9, 1, 128), (32, 2, 64), (16, 1, 128)])
@pytest.mark.parametrize("block,cache", [(16, "int8"), (48, "int8"), (128, "int8"), (24, "int8"), (16, "bf16"), (128, "bf16")])
def test_decode(heads, kv, dim, block, cache):
    from mindformers_b200.inference import paged_attention as pa
    from mindformers_b200.ops import _lib
    torch.manual_seed(heads)
    lens = [1, 15, 16, 17, 64, 65, 1000, 3, 5000]
    idle, B, int8 = 7, len(lens), cache == "int8"
    tables, blocks = _tables(lens, block)
    ctx = pa.KVCacheContext(1, blocks, block, kv, dim, torch.bfloat16, DEV, kv_cache_dtype="int8" if int8 else None)
    if int8:                           # scales of rows that nobody wrote
        ctx.key_scale[0].fill_(float("nan"))
        ctx.value_scale[0].fill_(float("inf"))
    step = dict(block_tables=tables.numpy(), context_lens=lens, device=DEV)
    ctx.set_step(is_prefill=True, slot_mapping=_slots(tables, block, lens, lens).numpy(), q_seq_lens=lens, **step)
    rows = torch.randn(2, sum(lens), kv, dim, device=DEV).to(torch.bfloat16) * torch.rand(sum(lens), 1, 1, device=DEV).to(torch.bfloat16)
    pa._write_cache(ctx, 0, rows[0], rows[1])
    slots = _slots(tables, block, lens, [1] * B)
    slots[idle], tables[idle] = -1, -1
    ctx.set_step(is_prefill=False, slot_mapping=slots.numpy(), q_seq_lens=[1] * B, **step)
    qkv = torch.randn(B, heads + 2 * kv, dim, device=DEV).to(torch.bfloat16)
    with torch.no_grad():
        got = pa.paged_attention_forward(qkv[:, :heads], qkv[:, heads:heads + kv], qkv[:, heads + kv:], types.SimpleNamespace(cache=ctx), 1,
                                         dim ** -0.5)
    for b, n in enumerate(lens):
        if b == idle:
            assert not got[b].any()
            continue
        k, v = (_cached(c[0], tables, b, n, block).double() for c in (ctx.key_cache, ctx.value_cache))
        if int8:
            k, v = (x * _cached(s[0], tables, b, n, block).double().unsqueeze(-1) for x, s in ((k, ctx.key_scale), (v, ctx.value_scale)))
        want = _attend(qkv[b:b + 1, :heads], k, v, dim ** -0.5)[0]
        err = (got[b].double() - want).norm() / want.norm()
        # rounding of the result alone (1.5e-3 to 1.7e-3 in the mean square); the bf16 cache's kernel rounds the weights as well
        assert err < (2e-3 if int8 or dim == 64 else 4e-3), (b, float(err))
    assert _lib.read_status() == 0


# heads on the rows of the products: chunks of 32, 64 and 128 rows with and without a remainder; splits with one tile, several and none
@pytest.mark.parametrize("heads", [17, 32, 40, 64, 100, 128, 130])
@pytest.mark.parametrize("block", [16, 64, 128])
def test_latent_decode_heads_on_rows(heads, block):
    from mindformers_b200.inference import paged_attention as pa
    from mindformers_b200.ops import _lib
    torch.manual_seed(heads)
    lens = [1, 127, 128, 129, 700, 3000]
    tables, blocks = _tables(lens, block)
    cache = torch.randn(blocks, block, 1, 576, device=DEV).to(torch.bfloat16)
    q = torch.randn(len(lens), heads, 576, device=DEV).to(torch.bfloat16)
    got = pa.mla_decode_attention(q, cache, tables.to(DEV), torch.tensor(lens, dtype=torch.int32, device=DEV), block, 192 ** -0.5)
    for b, n in enumerate(lens):
        lat = _cached(cache[:, :, 0], tables, b, n, block).double()
        want = torch.softmax(q[b].double() @ lat.t() * 192 ** -0.5, -1) @ lat[:, :512]
        err = (got[b].double() - want).norm() / want.norm()
        assert err < 4e-3, (b, float(err))           # the weights and the result are rounded, 1.7e-3 in the mean square each
    assert _lib.read_status() == 0


def _set(ctx, tables, block, lens, news):
    ctx.set_step(is_prefill=True, slot_mapping=_slots(tables, block, lens, news).numpy(), q_seq_lens=news, block_tables=tables.numpy(),
                 context_lens=lens, device=DEV)


def _prefill_call(path, rows):
    """A context of two sequences and a prefill call on it: grouped-query attention over a bf16 cache, multi-latent attention by expansion
    or (other head sizes) by the general path."""
    from mindformers_b200.inference import paged_attention as pa
    torch.manual_seed(rows)
    if path == "grouped":
        ctx = pa.KVCacheContext(1, 16, 16, 2, 64, torch.bfloat16, DEV)
        ctx.key_cache[0].normal_()
        ctx.value_cache[0].normal_()
        x = torch.randn(rows, 8, 64, device=DEV).to(torch.bfloat16)
        return ctx, lambda: pa.paged_attention_forward(x[:, :4], x[:, 4:6], x[:, 6:], types.SimpleNamespace(cache=ctx), 1, 0.125)
    nope, heads = (128 if path == "expanded" else 64), 3
    ctx = pa.KVCacheContext(1, 16, 16, 1, 0, torch.bfloat16, DEV, mla_latent_dim=576)
    ctx.key_cache[0].normal_()
    w = (torch.randn(heads * 2 * nope, 512, device=DEV) * 512 ** -0.5).to(torch.bfloat16)
    attn = types.SimpleNamespace(nh=heads, nope=nope, rope_d=64, vd=nope, kv_rank=512, layer_number=1, scale=0.07,
                                 linear_kvb=types.SimpleNamespace(weight=w))
    q = torch.randn(rows, heads, nope + 64, device=DEV).to(torch.bfloat16)
    new = torch.randn(rows, 576, device=DEV).to(torch.bfloat16)
    return ctx, lambda: pa.mla_paged_attention_forward(attn, q[..., :nope], q[..., nope:].clone(), new[:, :512], new[:, 512:],
                                                       types.SimpleNamespace(cache=ctx))


@pytest.mark.parametrize("path", ["grouped", "expanded", "general"])
@pytest.mark.parametrize("how", ["inference", "data", "version", "kept", "boundaries"])
def test_step_changed_after_set_step(path, how):
    """A prefill call answers for the lengths and boundaries that its context has now."""
    first, then, news = [90, 70], [85, 70], [3, 5]
    tables, _ = _tables([96, 96], 16)
    ctx, call = _prefill_call(path, sum(news))
    with torch.inference_mode(how == "inference"), torch.no_grad():
        _set(ctx, tables, 16, first, news)
        slots = ctx.slot_mapping.clone()
        kept = ctx.context_lens if how == "kept" else None
        if how in ("kept", "boundaries"):
            call()                                   # what the layers of a step share has been made
        if how == "boundaries":
            ctx.cu_q[1] = 4
            then, news = first, [4, 4]
        elif how == "kept":
            kept.data.copy_(torch.tensor(then))
        elif how == "data":
            ctx.context_lens.data.copy_(torch.tensor(then))
        else:
            ctx.context_lens.copy_(torch.tensor(then))
        got = call()
        _set(ctx, tables, 16, then, news)
        ctx.slot_mapping = slots
        assert torch.equal(got, call())


@pytest.mark.parametrize("kind", ["int8", "odd pages", "latent"])
def test_more_tables_than_sequences(kind):
    """Rows of the block tables past the step's sequences are not looked at, where the rows that a step sees are copied out first."""
    from mindformers_b200.inference import paged_attention as pa
    block, lens, news = (24 if kind == "odd pages" else 16), [90, 70], [3, 5]
    tables, blocks = _tables([96, 96], block)
    if kind == "latent":
        ctx, call = _prefill_call("expanded", sum(news))
    else:
        ctx = pa.KVCacheContext(1, blocks, block, 1, 64, torch.bfloat16, DEV, kv_cache_dtype="int8" if kind == "int8" else None)
        x = torch.randn(sum(news), 4, 64, device=DEV).to(torch.bfloat16)
        rows = torch.randn(2, sum(lens), 1, 64, device=DEV).to(torch.bfloat16)
        _set(ctx, tables, block, lens, lens)
        pa._write_cache(ctx, 0, rows[0], rows[1])

        def call():
            return pa.paged_attention_forward(x[:, :2], x[:, 2:3], x[:, 3:], types.SimpleNamespace(cache=ctx), 1, 0.125)
    with torch.no_grad():
        _set(ctx, tables, block, lens, news)
        want = call()
        more = torch.cat((tables, torch.full((5, tables.shape[1]), -1, dtype=torch.int32)))
        _set(ctx, more, block, lens, news)
        assert torch.equal(call(), want)


@pytest.mark.parametrize("path", ["grouped", "expanded", "general"])
@pytest.mark.parametrize("planned", [False, True])
def test_prefill_is_not_captured(path, planned):
    """A graph would keep the tiles of one step's lengths: a prefill call under capture raises, also where its plan is there already."""
    tables, _ = _tables([96, 96], 16)
    ctx, call = _prefill_call(path, 8)
    with torch.no_grad():
        _set(ctx, tables, 16, [90, 70], [3, 5])
        want = call()
        if not planned:
            _set(ctx, tables, 16, [90, 70], [3, 5])
        torch.cuda.synchronize()
        with pytest.raises(RuntimeError, match="captured"):
            with torch.cuda.graph(torch.cuda.CUDAGraph()):
                call()
        torch.cuda.synchronize()
        assert torch.equal(call(), want)


def _decode_call(int8=False):
    """A context of three sequences with full caches, its step and a decode call on it."""
    from mindformers_b200.inference import paged_attention as pa
    torch.manual_seed(0)
    ctx = pa.KVCacheContext(1, 32, 16, 2, 128, torch.bfloat16, DEV, kv_cache_dtype="int8" if int8 else None)
    for c in (ctx.key_cache[0], ctx.value_cache[0]):
        c.copy_(torch.randn(c.shape, device=DEV) * (50 if int8 else 1))
    lens = [90, 33, 128]
    tables, _ = _tables(lens, 16)
    step = dict(is_prefill=False, slot_mapping=_slots(tables, 16, lens, [1] * 3).numpy(), q_seq_lens=[1] * 3, block_tables=tables.numpy(),
                context_lens=lens, device=DEV)
    x = torch.randn(3, 8, 128, device=DEV).to(torch.bfloat16)
    return ctx, step, lambda: pa.paged_attention_forward(x[:, :4], x[:, 4:6], x[:, 6:], types.SimpleNamespace(cache=ctx), 1, 0.09)


def test_step_used_on_another_stream():
    """The tensors of a step are complete for whoever reads them, and the attention of the step may run on another stream, although the
    stream of ``set_step`` is still busy."""
    ctx, step, call = _decode_call()
    side = torch.cuda.Stream()
    with torch.no_grad():
        ctx.set_step(**step)
        want = call()
        wide = torch.arange(100000, dtype=torch.int32)
        torch.cuda.synchronize()
        torch.cuda._sleep(100_000_000)               # some tens of milliseconds
        ctx.set_step(**dict(step, slot_mapping=wide.numpy()))
        with torch.cuda.stream(side):
            assert torch.equal(ctx.slot_mapping.cpu(), wide)
        torch.cuda.synchronize()
        torch.cuda._sleep(100_000_000)
        ctx.set_step(**step)
        with torch.cuda.stream(side):
            got = call()
        side.synchronize()
        assert torch.equal(got, want)
        torch.cuda.synchronize()
        torch.cuda._sleep(100_000_000)
        ctx.set_step(**step)
        twin = copy.deepcopy(ctx)
        assert all(torch.equal(getattr(twin, n), getattr(ctx, n)) for n in ("block_tables", "slot_mapping", "context_lens"))


def test_step_in_a_captured_graph():
    """A step that was set before a capture serves the captured call; setting one under capture raises."""
    ctx, step, call = _decode_call()
    with torch.no_grad():
        ctx.set_step(**step)
        want = call()
        ctx.set_step(**step)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            got = call()
        got.zero_()
        graph.replay()
        assert torch.equal(got, want)
        torch.cuda.synchronize()
        with pytest.raises(RuntimeError, match="captured"):
            with torch.cuda.graph(torch.cuda.CUDAGraph()):
                ctx.set_step(**step)
        torch.cuda.synchronize()


def test_step_from_the_host():
    """Where new tensors go by default does not matter to a step; numbers that do not fit into 32 bits are refused."""
    ctx, step, call = _decode_call()
    with torch.no_grad():
        ctx.set_step(**step)
        want = call()
        with torch.device(DEV):
            ctx.set_step(**step)
        assert torch.equal(call(), want)
        for name in ("slot_mapping", "context_lens", "q_seq_lens"):
            with pytest.raises((RuntimeError, OverflowError)):
                ctx.set_step(**dict(step, **{name: [2 ** 31 + 5, 1, 1]}))


@pytest.mark.parametrize("block,int8", [(64, True), (24, False)])
def test_copied_rows_in_turns(block, int8, monkeypatch):
    """A step whose sequences see more cached rows than may be copied out at a time: the same result in less memory."""
    from mindformers_b200.inference import paged_attention as pa
    lens, news = [900, 1400, 64, 2000, 33, 700], [3, 200, 64, 130, 1, 5]
    tables, blocks = _tables(lens, block)
    ctx = pa.KVCacheContext(1, blocks, block, 4, 128, torch.bfloat16, DEV, kv_cache_dtype="int8" if int8 else None)
    rows = torch.randn(2, sum(lens), 4, 128, device=DEV).to(torch.bfloat16)
    x = torch.randn(sum(news), 16, 128, device=DEV).to(torch.bfloat16)
    _set(ctx, tables, block, lens, lens)
    pa._write_cache(ctx, 0, rows[0], rows[1])
    taken = []
    with torch.no_grad():
        for budget in (pa._COPIED_BYTES, 1):
            monkeypatch.setattr(pa, "_COPIED_BYTES", budget)
            _set(ctx, tables, block, lens, news)
            torch.cuda.reset_peak_memory_stats()
            before = torch.cuda.memory_allocated()
            taken.append((pa.paged_attention_forward(x[:, :8], x[:, 8:12], x[:, 12:], types.SimpleNamespace(cache=ctx), 1, 0.09),
                          torch.cuda.max_memory_allocated() - before))
    assert torch.equal(taken[0][0], taken[1][0])
    row = 2 * 4 * 128 * 2
    assert taken[1][1] < (2000 + 500) * row < sum(lens) * row < taken[0][1] + 64 * row     # 500: the result and the step's lists


def test_latent_prefill_of_few_rows():
    """One and two new rows behind long histories: the queries go into the latent space."""
    from mindformers_b200.inference import paged_attention as pa
    torch.manual_seed(0)
    heads, block, lens, news = 128, 16, [3000, 2900], [1, 2]
    tables, blocks = _tables(lens, block)
    ctx = pa.KVCacheContext(1, blocks, block, 1, 0, torch.bfloat16, DEV, mla_latent_dim=576)
    ctx.key_cache[0].normal_()
    w = (torch.randn(heads * 256, 512, device=DEV) * 512 ** -0.5).to(torch.bfloat16)
    attn = types.SimpleNamespace(nh=heads, nope=128, rope_d=64, vd=128, kv_rank=512, layer_number=1, scale=192 ** -0.5,
                                 linear_kvb=types.SimpleNamespace(weight=w))
    q = torch.randn(3, heads, 192, device=DEV).to(torch.bfloat16)
    new = torch.randn(3, 576, device=DEV).to(torch.bfloat16)
    _set(ctx, tables, block, lens, news)
    assert not pa._prefill_plan(ctx, 3, latent=True).expands(heads)
    with torch.no_grad():
        got = pa.mla_paged_attention_forward(attn, q[..., :128], q[..., 128:].clone(), new[:, :512], new[:, 512:],
                                             types.SimpleNamespace(cache=ctx))
    for rows, b, m in ((slice(0, 1), 0, 3000), (slice(1, 3), 1, 2900)):
        lat = _cached(ctx.key_cache[0][:, :, 0], tables, b, m, block).double()
        kv = (lat[:, :512] @ w.double().t()).view(m, heads, 256)
        want = _attend(q[rows], torch.cat((kv[..., :128], lat[:, None, 512:].expand(m, heads, 64)), -1), kv[..., 128:], attn.scale)
        assert (got[rows].double() - want).norm() / want.norm() < 2e-3           # rounding of the result alone


def _latent_layer(**over):
    from mindformers_b200.models.presets import get_preset
    from mindformers_b200.parallel.layers.attention import MLASelfAttention
    from mindformers_b200.parallel.layers.rotary import get_rope
    from mindformers_b200.parallel.transformer_config_utils import convert_to_transformer_config
    cfg = get_preset("deepseek_v3", num_attention_heads=4, num_key_value_heads=4, hidden_size=256, max_position_embeddings=512, **over)
    cfg.update(params_dtype="bfloat16", compute_dtype="bfloat16")
    cfg = convert_to_transformer_config(cfg, is_mla_model=True)
    cfg.device = DEV
    return MLASelfAttention(cfg).eval(), get_rope(cfg, device=DEV)()


@pytest.mark.parametrize("prefill,seqs", [(True, 3), (False, 3), (False, 1)])
def test_latent_layer_leaves_its_projections_alone(prefill, seqs):
    """What a forward hook keeps of a projection's output in serving is that output."""
    from mindformers_b200.inference import paged_attention as pa
    from mindformers_b200.parallel.layers.attention import AttnMeta
    torch.manual_seed(0)
    layer, rotary = _latent_layer()
    lens = [40, 70, 3][:seqs]
    news = ([7, 20, 3] if prefill else [1] * 3)[:seqs]
    tables, blocks = _tables(lens, 16)
    ctx = pa.KVCacheContext(1, blocks, 16, 1, 0, torch.bfloat16, DEV, mla_latent_dim=576)
    ctx.set_step(is_prefill=prefill, slot_mapping=_slots(tables, 16, lens, news).numpy(), q_seq_lens=news, block_tables=tables.numpy(),
                 context_lens=lens, device=DEV)
    pos = torch.cat([torch.arange(n - m, n) for n, m in zip(lens, news)]).to(DEV)
    x = torch.randn(sum(news), 256, device=DEV).to(torch.bfloat16)
    kept = []
    layer.linear_qkv.register_forward_hook(lambda mod, args, out: kept.append(out[0]))
    with torch.no_grad():
        layer(x, rotary, AttnMeta(batch=1, seq_len=sum(news), positions=pos, cache=ctx))
        assert torch.equal(kept[0], layer.linear_qkv(x)[0])


@pytest.mark.parametrize("which", ["query columns", "keys interleaved", "values off by one"])
def test_decode_of_other_layouts(which):
    """Rows of a bf16 step that no tensor map describes run on the tensor cores like others."""
    from mindformers_b200.inference import paged_attention as pa
    ctx, step, _ = _decode_call()
    x = torch.randn(3, 8, 128, device=DEV).to(torch.bfloat16)
    plain = [x[:, :4].contiguous(), x[:, 4:6].contiguous(), x[:, 6:].contiguous()]
    q, k, v = plain
    if which == "query columns":
        q = q.transpose(1, 2).contiguous().transpose(1, 2)
    elif which == "keys interleaved":
        k = torch.stack((k, k), 2)[:, :, 0]
    else:
        v = torch.cat((v.flatten(), v.flatten()[:1])).roll(1)[1:].view(3, 2, 128)
    ctx.set_step(**step)
    with torch.no_grad():
        want = pa._decode_step(*plain, ctx, 0, 0.09)
        ctx.key_cache[0].view(-1, 2, 128)[ctx.slot_mapping.long()] = 0
        got = pa._decode_step(q, k, v, ctx, 0, 0.09)
    assert got is not None and torch.equal(got, want)


def _bits(t):
    return t.view(torch.int16 if t.dtype == torch.bfloat16 else torch.int32 if t.dtype == torch.float32 else t.dtype)


@pytest.mark.parametrize("heads,kv,block", [(8, 2, 16), (4, 4, 128)])
@pytest.mark.parametrize("int8", [False, True])
@pytest.mark.parametrize("fused", [True, False])
def test_new_rows_reach_the_cache(heads, kv, block, int8, fused):
    """The rows of a step lie in its slots, in no others, and a row without a slot nowhere; ``fused``: written by the call that attends."""
    from mindformers_b200.inference import paged_attention as pa
    torch.manual_seed(kv)
    dim, B = 128, 5
    ctx = pa.KVCacheContext(1, 12, block, kv, dim, torch.bfloat16, DEV, kv_cache_dtype="int8" if int8 else None)
    caches = [ctx.key_cache[0], ctx.value_cache[0]]
    scales = [ctx.key_scale[0], ctx.value_scale[0]] if int8 else []
    for c in caches:
        c.fill_(77 if int8 else float("nan"))
    for s in scales:
        s.fill_(float("inf"))
    before = [t.clone() for t in caches + scales]
    tables = torch.randperm(10).view(B, 2).to(torch.int32)
    lens = [1, block, block + 1, 2 * block, 7]
    slots = _slots(tables, block, lens, [1] * B)
    slots[3] = -1
    ctx.set_step(is_prefill=False, block_tables=tables.numpy(), slot_mapping=slots.numpy(), context_lens=lens, q_seq_lens=[1] * B, device=DEV)
    x = torch.randn(B, heads + 2 * kv, dim, device=DEV).to(torch.bfloat16)
    x[1] = 0                                                # a row of zeros has scale one
    k, v = x[:, heads:heads + kv], x[:, heads + kv:]
    with torch.no_grad():
        if fused:
            assert pa._decode_step(x[:, :heads], k, v, ctx, 0, 0.09) is not None
        else:
            pa._write_cache(ctx, 0, k, v)
    used = [0, 1, 2, 4]
    at = slots[used].to(DEV)
    for i, (cache, rows) in enumerate(zip(caches, (k, v))):
        got, rows = cache.view(-1, kv, dim)[at], rows[used]
        if int8:
            top = rows.float().abs().amax(-1)
            scale = torch.where(top > 0, top / 127, torch.ones_like(top))
            assert torch.allclose(scales[i].view(-1, kv)[at], scale, rtol=1e-6)
            # codes are the nearest ones: half a step, and what a reciprocal instead of a division adds
            assert ((got.float() * scale.unsqueeze(-1) - rows.float()).abs() <= scale.unsqueeze(-1) * 0.5001).all()
        else:
            assert torch.equal(got, rows)
    for now, old in zip(caches + scales, before):
        now, old = (_bits(t).flatten(0, 1).clone() for t in (now, old))
        now[at] = old[at]
        assert torch.equal(now, old)


@pytest.mark.parametrize("view", [True, False])
def test_latents_reach_the_cache(view):
    """``view``: the parts are columns of wider rows that start on 16 bytes; otherwise on other addresses (the general path)."""
    from mindformers_b200.inference import paged_attention as pa
    torch.manual_seed(0)
    ctx = pa.KVCacheContext(1, 6, 16, 1, 0, torch.bfloat16, DEV, mla_latent_dim=576)
    ctx.key_cache[0].fill_(float("nan"))
    before = ctx.key_cache[0].clone()
    slots = torch.randperm(96)[:33]
    slots[5] = -1
    ctx.set_step(is_prefill=True, block_tables=[[0, 1, 2, 3, 4, 5]], slot_mapping=slots.numpy(), context_lens=[33], q_seq_lens=[33], device=DEV)
    wide = torch.randn(33, 640, device=DEV).to(torch.bfloat16)
    at = 16 if view else 3
    pa._write_latents(ctx, 0, wide[:, at:at + 512], wide[:, at + 512:at + 576])
    used = [i for i in range(33) if i != 5]
    to = slots[used].to(DEV)
    rows = ctx.key_cache[0].view(-1, 576)
    assert torch.equal(rows[to], wide[used, at:at + 576])
    rest, old = _bits(rows).clone(), _bits(before).view(-1, 576)
    rest[to] = old[to]
    assert torch.equal(rest, old)


@pytest.mark.parametrize("T,heads,hd,rot,left", [(1, 1, 64, 64, 32), (33, 1, 64, 64, 64), (33, 5, 192, 64, 0), (1, 3, 192, 64, 0), (7, 2, 40, 24, 0)])
@pytest.mark.parametrize("interleaved", [False, True])
def test_rope_of_heads_in_place(T, heads, hd, rot, left, interleaved):
    """The last columns of every head, in rows that may be a slice of wider ones; the other columns keep their bits."""
    from mindformers_b200.ops import functional as Fn
    torch.manual_seed(T)
    wide = torch.randn(T, left + heads * hd + 8 * (left > 0), device=DEV).to(torch.bfloat16)
    old = wide.clone()
    angle = torch.rand(50, rot // 2, device=DEV) * 6
    cos, sin, pos = angle.cos(), angle.sin(), torch.randint(0, 50, (T,), device=DEV)
    view = lambda t: t[:, left:left + heads * hd].view(T, heads, hd)
    assert Fn.rope_heads_supported(view(wide), rot)
    Fn.rope_heads_(view(wide), cos, sin, pos.to(torch.int32), rot, interleaved)
    want = Fn.rope_reference(view(old)[..., hd - rot:].contiguous(), cos, sin, pos, heads, rot, interleaved)
    got = view(wide)[..., hd - rot:]
    # rounded once, at most 2^-8 of a number; a difference of two products may cancel, so relative to the pair
    assert (got.float() - want.float()).abs().max() <= 2 ** -8 * 2 * want.float().abs().max()
    view(old)[..., hd - rot:] = got
    assert torch.equal(_bits(wide), _bits(old))


@pytest.mark.parametrize("heads", [16, 17, 64, 128])
@pytest.mark.parametrize("block", [16, 128])
def test_latent_decode_of_idle_rows(heads, block):
    """Sequences of no tokens and rows without blocks give zeros and leave the others as they are; large numbers behind a sequence's end
    have no effect."""
    from mindformers_b200.inference import paged_attention as pa
    from mindformers_b200.ops import _lib
    torch.manual_seed(heads)
    lens = [300, 0, 130, 5, 1]
    tables, blocks = _tables([300, 1, 130, 5, 1], block)
    cache = torch.full((blocks, block, 1, 576), 1e30, device=DEV).to(torch.bfloat16)
    for b, n in enumerate(lens):
        for i in range(-(-n // block)):
            rows = min(block, n - i * block)
            cache[tables[b, i].long(), :rows] = torch.randn(rows, 1, 576, device=DEV).to(torch.bfloat16)
    want = cache.clone()
    tables[3] = -1                                          # an idle slot: a length, no blocks
    q = torch.randn(5, heads, 576, device=DEV).to(torch.bfloat16)
    got = pa.mla_decode_attention(q, cache, tables.to(DEV), torch.tensor(lens, dtype=torch.int32, device=DEV), block, 192 ** -0.5)
    assert not got[1].any() and not got[3].any()
    for b in (0, 2, 4):
        lat = _cached(want[:, :, 0], tables, b, lens[b], block).double()
        ref = torch.softmax(q[b].double() @ lat.t() * 192 ** -0.5, -1) @ lat[:, :512]
        assert (got[b].double() - ref).norm() / ref.norm() < 4e-3        # as above
    assert _lib.read_status() == 0


def test_prefill_with_gradients():
    """A call whose result needs a gradient goes through operations that have one."""
    from mindformers_b200.inference import paged_attention as pa
    torch.manual_seed(0)
    ctx = pa.KVCacheContext(1, 16, 16, 2, 64, torch.bfloat16, DEV)
    x = torch.randn(128, 8, 64, device=DEV).to(torch.bfloat16).requires_grad_()
    tables, _ = _tables([128], 16)
    _set(ctx, tables, 16, [128], [128])

    def call(x):
        return pa.paged_attention_forward(x[:, :4], x[:, 4:6], x[:, 6:], types.SimpleNamespace(cache=ctx), 1, 0.125)
    out = call(x)
    dy = torch.randn_like(out)
    got = torch.autograd.grad(out, x, dy)[0]
    x64 = x.detach().double().requires_grad_()
    q, k, v = x64[:, :4], x64[:, 4:6].repeat_interleave(2, 1), x64[:, 6:].repeat_interleave(2, 1)
    s = torch.einsum("qhd,khd->hqk", q, k) * 0.125
    hide = torch.ones(128, 128, device=DEV, dtype=torch.bool).triu(1)
    ref = torch.einsum("hqk,khd->qhd", torch.softmax(s.masked_fill(hide, float("-inf")), -1), v).flatten(1)
    want = torch.autograd.grad(ref, x64, dy.double())[0]
    # the weights, their gradients and the results are rounded to 16 bits, at most 2^-8 each
    assert (got.double() - want).norm() / want.norm() < 1.2e-2
    with torch.no_grad():
        plain = call(x)
    assert (plain.double() - ref.detach()).norm() / ref.detach().norm() < 4e-3


def test_decode_kernel_first_in_a_thread():
    """A thread whose first work on the GPU is the decode kernel."""
    import threading
    from mindformers_b200.ops import _lib
    torch.manual_seed(0)
    lib = _lib.get_lib()
    q, kc, vc = (torch.randn(*s, device=DEV).to(torch.bfloat16) for s in ((2, 4, 128), (6, 16, 2, 128), (6, 16, 2, 128)))
    tables, lens = (torch.tensor(t, dtype=torch.int32, device=DEV) for t in ([[0, 1, 2], [3, 4, 5]], [40, 17]))
    splits = lib.mfb_paged_decode_tc_splits(2, 2, 48)
    scratch = torch.empty(lib.mfb_paged_decode_scratch_bytes(2, 4, 128, splits) // 4 + 4, device=DEV)
    outs = [torch.zeros(2, 4, 128, device=DEV, dtype=torch.bfloat16) for _ in range(2)]
    args = [(q.data_ptr(), kc.data_ptr(), vc.data_ptr(), tables.data_ptr(), lens.data_ptr(), out.data_ptr(), scratch.data_ptr(), splits, 2, 4,
             2, 6, 16, 3, 0.09, _lib.status_word(DEV).data_ptr(), 0) for out in outs]
    torch.cuda.synchronize()
    codes = [lib.mfb_paged_decode_attention_tc(*args[0])]
    torch.cuda.synchronize()
    other = threading.Thread(target=lambda: codes.append(lib.mfb_paged_decode_attention_tc(*args[1])))
    other.start()
    other.join()
    torch.cuda.synchronize()
    assert codes == [0, 0], lib.mfb_last_error()
    assert outs[0].any() and torch.equal(outs[0], outs[1])


def test_latents_copied_in_turns(monkeypatch):
    """A multi-latent step whose sequences see more cached rows than may be copied out at a time."""
    from mindformers_b200.inference import paged_attention as pa
    torch.manual_seed(0)
    heads, block, lens, news = 2, 64, [2900, 2700, 64, 3000, 20], [700, 5, 64, 130, 0]
    tables, blocks = _tables(lens, block)
    ctx = pa.KVCacheContext(1, blocks, block, 1, 0, torch.bfloat16, DEV, mla_latent_dim=576)
    ctx.key_cache[0].normal_()
    w = (torch.randn(heads * 256, 512, device=DEV) * 512 ** -0.5).to(torch.bfloat16)
    attn = types.SimpleNamespace(nh=heads, nope=128, rope_d=64, vd=128, kv_rank=512, layer_number=1, scale=192 ** -0.5,
                                 linear_kvb=types.SimpleNamespace(weight=w))
    T = sum(news)
    q = torch.randn(T, heads, 192, device=DEV).to(torch.bfloat16)
    new = torch.randn(T, 576, device=DEV).to(torch.bfloat16)
    taken = []
    for budget in (pa._COPIED_BYTES, 1):
        monkeypatch.setattr(pa, "_COPIED_BYTES", budget)
        _set(ctx, tables, block, lens, news)
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        with torch.no_grad():
            got = pa.mla_paged_attention_forward(attn, q[..., :128], q[..., 128:].clone(), new[:, :512], new[:, 512:],
                                                 types.SimpleNamespace(cache=ctx))
        taken.append(torch.cuda.max_memory_allocated() - before)
        at = 0
        for b, (n, m) in enumerate(zip(news, lens)):
            rows, at = slice(at, at + n), at + n
            if not n:
                continue
            lt = _cached(ctx.key_cache[0][:, :, 0], tables, b, m, block).double()
            kv = (lt[:, :512] @ w.double().t()).view(m, heads, 256)
            want = _attend(q[rows], torch.cat((kv[..., :128], lt[:, None, 512:].expand(m, heads, 64)), -1), kv[..., 128:], attn.scale)
            assert (got[rows].double() - want).norm() / want.norm() < 2e-3           # rounding of the result alone
    row = 576 * 2 + heads * 256 * 8
    assert taken[1] < taken[0] - 5000 * row                 # at most 3000 rows at a time instead of 8664
