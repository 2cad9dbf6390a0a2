"""What a prefill step's plan is made from, and which steps it leaves to the general path."""
import numpy as np
import torch

from mindformers_b200.inference import paged_attention as pa


def _ctx(tables, lens=(40, 20), news=(8, 4)):
    ctx = pa.KVCacheContext(1, 8, 16, 1, 64, torch.float32, "cpu")
    ctx.set_step(is_prefill=True, block_tables=tables, slot_mapping=np.zeros(sum(news), np.int32), context_lens=list(lens),
                 q_seq_lens=list(news), device="cpu")
    return ctx


def test_plan_follows_the_values_it_was_made_from():
    ctx = _ctx(np.zeros((2, 3), np.int32))
    plan = pa._prefill_plan(ctx, 12)
    assert plan.ok and plan.n_past_rows == 60 and pa._prefill_plan(ctx, 12) is plan
    ctx.cu_q[1] = 9                                          # the same list, other boundaries
    assert pa._prefill_plan(ctx, 12).cu.tolist() == [0, 9, 12]
    ctx.context_lens.data.add_(1)
    assert pa._prefill_plan(ctx, 12).n_past_rows == 62
    ctx.block_tables = torch.zeros((2, 2), dtype=torch.int32)
    assert not pa._prefill_plan(ctx, 12).ok                  # 41 tokens in tables of 32


def test_host_copy_of_the_lengths_ends_when_the_tensor_is_handed_out():
    ctx = _ctx(np.zeros((2, 3), np.int32))
    ctx.host_lens = [40, 20]                                 # as set_step leaves it for a CUDA device
    assert pa._host_lens(ctx) == [40, 20] and ctx.host_lens is not None
    held = ctx.context_lens
    held.data.add_(1)
    assert pa._host_lens(ctx) == [41, 21]
    ctx.host_lens = [41, 21]
    ctx.context_lens = torch.tensor([7, 7], dtype=torch.int32)
    assert pa._host_lens(ctx) == [7, 7]


def test_tables_of_another_form_stay_on_the_general_path():
    good = np.zeros((2, 3), np.int32)
    for tables, ok in ((good, True), (np.zeros((3, 3), np.int32), True), (good[:1], False), (np.zeros(0, np.int32), False)):
        assert pa._prefill_plan(_ctx(tables), 12).ok == ok, tables.shape
    ctx = _ctx(good)
    ctx.block_tables = torch.zeros((2, 3), dtype=torch.int64)
    assert not pa._prefill_plan(ctx, 12).ok
    ctx.block_tables = torch.zeros((3, 2), dtype=torch.int32).t()
    assert not pa._prefill_plan(ctx, 12).ok


def test_copies_in_groups():
    """Every tile in one group with the rows of its sequence, no group above the limit but for a sequence that is alone."""
    lens, news = [40, 20, 8, 300, 30, 25], [8, 4, 8, 200, 0, 25]         # the third and the last have no history, the fifth no new rows
    ctx = _ctx(np.zeros((6, 20), np.int32), lens, news)
    plan = pa._prefill_plan(ctx, sum(news))
    assert [(w[1], r) for w, _, r in plan.copied(360)] == [(4, 360)]
    for limit, rows in ((359, [60, 300]), (59, [40, 20, 300]), (1, [40, 20, 300])):
        groups = plan.copied(limit)
        assert [r for _, _, r in groups] == rows
        seen = []
        for (work, n, _), first, total in groups:
            tiles = work.view(n, 4).tolist()
            assert first.numel() == 7 and first[-1] == total
            assert all(first[b + 1] - first[b] == lens[b] for b, *_ in tiles)
            seen += tiles
        assert sorted(seen) == sorted(plan.past[0].view(-1, 4).tolist())


def test_form_of_latent_attention():
    """Few new rows behind long histories are not worth expanding every cached latent for all heads."""
    def expands(B, past, new, heads):
        ctx = _ctx(np.zeros((B, (past + new) // 16 + 1), np.int32), [past + new] * B, [new] * B)
        return pa._prefill_plan(ctx, B * new, latent=True).expands(heads)
    assert not expands(32, 8000, 1, 128) and not expands(32, 8000, 4, 128) and expands(32, 8000, 64, 128)
    assert not expands(1, 8000, 4, 128) and expands(1, 8000, 64, 128)
    assert expands(32, 8000, 1, 16) and expands(4, 1200, 900, 16) and expands(32, 500, 1, 128)
