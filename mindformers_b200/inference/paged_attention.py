"""Attention over the paged KV cache: cache allocation, prefill and decode paths.

Reference: ``parallel_core/inference/transformer/flash_attention.py`` (prefill = cache write + varlen flash
attention :94-107; decode = paged attention :109-145), MLA mode with one latent "head" of width
``kv_lora_rank + rope_dim`` (``multi_latent_attention.py:401-448``), cache shapes from
``generation/text_generator.py:114-160``.

``KVCacheContext`` travels in ``AttnMeta.cache``; it owns the per-layer cache tensors and the device copies of
the block table, slot mapping and lengths for the current step.
"""
from __future__ import annotations

import os

import math
from typing import List, Optional

import numpy as np
import torch

from ..ops import _lib
from ..ops import functional as Fn


def _strides(shape) -> list:
    out = [1] * len(shape)
    for i in range(len(shape) - 1, 0, -1):
        out[i - 1] = out[i] * shape[i]
    return out


def _to_device(arrays, device):
    """int32 arrays as device tensors, each on 16 bytes, through one pinned buffer and one copy in stream order."""
    at, spans = 0, []
    for a in arrays:
        spans.append((at, a.size, a.shape))
        at += -(-a.size // 4) * 4
    host = torch.empty(max(at, 1), dtype=torch.int32, device="cpu", pin_memory=torch.device(device).type == "cuda")
    flat = host.numpy()
    for a, (start, n, _) in zip(arrays, spans):
        flat[start:start + n] = a.reshape(-1)
    dev = host.to(device, non_blocking=True)       # the pinned buffer is not handed out again before the copy is done
    return [dev.as_strided(shape, _strides(shape), start) for start, n, shape in spans]


def _host_lens(cache) -> list:
    """The step's context lengths on the host: those ``set_step`` was given, or a read of the device once somebody else may have changed
    them (``KVCacheContext.context_lens``)."""
    if cache._context_lens.is_cuda and torch.cuda.is_current_stream_capturing():
        # a replay would go on with the tiles of the captured step's lengths
        raise RuntimeError("attention of this step needs the context lengths on the host: it cannot be captured in a CUDA graph")
    return cache.host_lens if cache.host_lens is not None else cache._context_lens.tolist()


class _StepTensor:
    """A tensor of the step's metadata. ``set_step`` queues its copy on the current stream and does not wait. The kernels of this module
    follow in the order of that stream (``_in_order``); whoever reads the attribute may use the tensor on any stream, so it is complete
    by then."""

    def __set_name__(self, owner, name):
        self.name = "_" + name

    def __get__(self, ctx, owner=None):
        if ctx is None:
            return self
        ctx._await_copy()
        if self.name == "_context_lens":
            # the reader may keep the tensor and write to it at any time (in inference mode, through .data or from a kernel nothing would
            # show it): the host's copy is not used from then on
            ctx.host_lens = None
        return ctx.__dict__[self.name]

    def __set__(self, ctx, value):
        ctx.__dict__[self.name] = value
        if self.name == "_context_lens":
            ctx.host_lens = None


class KVCacheContext:
    """Per-layer paged caches ``[num_blocks, block_size, kv_heads, head_dim]`` (or the 576-wide latent cache of
    multi-latent attention) plus the metadata of the current step: block tables, slot mapping, context lengths, new
    tokens per sequence. A tensor of the step that is read from here is on the device, for any stream; the attention calls follow a
    change of it."""

    block_tables = _StepTensor()      # int32 [B, max_blocks]
    slot_mapping = _StepTensor()      # int32 [T]
    context_lens = _StepTensor()      # int32 [B] tokens in cache after this step
    q_seq_lens = _StepTensor()        # int32 [B] new tokens of each sequence in this step
    last_token_index = _StepTensor()  # int64 [B] row of the last new token of each sequence

    def __init__(self, num_layers: int, num_blocks: int, block_size: int, kv_heads: int, head_dim: int,
                 dtype=torch.bfloat16, device="cuda", mla_latent_dim: Optional[int] = None,
                 kv_cache_dtype: Optional[str] = None, layer_shapes: Optional[list] = None,
                 state_shapes: Optional[list] = None, slots: int = 0, carry_width: int = 0):
        """``layer_shapes``: ``(kv heads, key size, value size)`` of every layer's cache, for models whose layers differ or
        whose keys and values differ in size (None: the layer caches no keys; value size 0: the layer's values are its keys);
        such a cache also carries the step metadata of ragged attention.

        ``state_shapes``: per layer None, ``(heads, key size, value size, conv channels, conv taps)`` or a list of shapes.
        Layers with a recurrent state have, for each of ``slots`` sequences (row b of a batch uses slot b), ``S [heads, key,
        value]`` in fp32 and a ring of the last conv inputs, or one fp32 tensor per listed shape (``recurrent[layer]``).
        ``carry_width``: every layer has a vector of that many fp32 values per slot that goes from one token to the next
        (``carry [layers, slots, width]``; ``carry_before`` is its value before a prefill step). A sequence that starts at
        position 0 reads none of them, so a slot changes hands without being cleared.

        ``kv_cache_dtype="int8"`` stores keys and values as int8 codes with one fp32 scale per token and KV head
        (``key_scale`` / ``value_scale`` ``[num_blocks, block_size, kv_heads]``): half the bytes per cached token, read
        back by the decode kernel and by prefill with history. Not available for the multi-latent cache."""
        self.num_layers, self.num_blocks, self.block_size = num_layers, num_blocks, block_size
        self.kv_heads, self.head_dim, self.mla_dim = kv_heads, head_dim, mla_latent_dim
        self.int8 = str(kv_cache_dtype or "").lower() in ("int8", "torch.int8")
        self.key_scale = self.value_scale = None
        self.compute_dtype = dtype
        if self.int8 and mla_latent_dim:
            raise ValueError("an int8 KV cache is not available for multi-latent attention")
        self.ragged = layer_shapes is not None
        if self.ragged:
            if self.int8 or mla_latent_dim or len(layer_shapes) != num_layers:
                raise ValueError("per-layer cache shapes: one per layer, and no int8 or latent cache")
            rows = (num_blocks, block_size)
            self.key_cache = [None if s is None else torch.zeros(rows + (s[0], s[1]), dtype=dtype, device=device)
                              for s in layer_shapes]
            self.value_cache = [None if s is None or not s[2] else torch.zeros(rows + (s[0], s[2]), dtype=dtype, device=device)
                                for s in layer_shapes]
        elif self.int8:
            shape = (num_blocks, block_size, kv_heads, head_dim)
            self.key_cache = [torch.zeros(shape, dtype=torch.int8, device=device) for _ in range(num_layers)]
            self.value_cache = [torch.zeros(shape, dtype=torch.int8, device=device) for _ in range(num_layers)]
            self.key_scale = [torch.ones(shape[:3], dtype=torch.float32, device=device) for _ in range(num_layers)]
            self.value_scale = [torch.ones(shape[:3], dtype=torch.float32, device=device) for _ in range(num_layers)]
        elif mla_latent_dim:
            self.key_cache = [torch.zeros(num_blocks, block_size, 1, mla_latent_dim, dtype=dtype, device=device)
                              for _ in range(num_layers)]
            self.value_cache = [None] * num_layers
        else:
            shape = (num_blocks, block_size, kv_heads, head_dim)
            self.key_cache = [torch.zeros(shape, dtype=dtype, device=device) for _ in range(num_layers)]
            self.value_cache = [torch.zeros(shape, dtype=dtype, device=device) for _ in range(num_layers)]

        def state(s):
            if s is None:
                return None
            if isinstance(s, list):
                return tuple(torch.zeros((slots,) + tuple(x), dtype=torch.float32, device=device) for x in s)
            return (torch.zeros((slots,) + tuple(s[:3]), dtype=torch.float32, device=device),
                    torch.zeros((slots, s[4], s[3]), dtype=dtype, device=device))
        self.recurrent = [state(s) for s in state_shapes or [None] * num_layers]
        self.carry = torch.zeros((num_layers, slots, carry_width), dtype=torch.float32, device=device) if carry_width else None
        self.carry_before = torch.zeros_like(self.carry) if carry_width else None
        self.is_prefill = True
        self._copied = None           # (event behind the copy of the step's tensors, its stream, asked before) while it may be under way
        self._event = None            # (the event, its device)
        self.block_tables = self.slot_mapping = self.context_lens = self.q_seq_lens = self.last_token_index = None
        self.cu_q = None              # python list of cumulative q lengths
        self.layer_offset = 0
        self.host_lens = None         # the lengths as set_step was given them, while nobody else holds the tensor
        self.cu_q_dev = None          # int32 [B+1]: cu_q on the device (ragged caches, prefill steps)
        self.prefill_work = {}        # work lists of the prefill kernels, made when a layer needs them
        self.q_lens_host = self.context_lens_host = ()
        self.n_long_rows = self.n_single_rows = 0     # sequences with several new rows / with one

    def _await_copy(self):
        """Returns when the step's tensors are on the device."""
        copied = self._copied
        if copied is not None:
            rc = _lib.get_lib().mfb_event_done(copied[0].cuda_event, 1)
            _lib.check(rc, "mfb_event_done")
            if self._copied is copied:           # and not the next step's, of another thread
                self._copied = None

    def _in_order(self):
        """Before kernels on the current stream read the step's tensors: on the stream that copies them there is nothing to wait for."""
        copied = self._copied
        if copied is None:
            return
        if copied[1] != _lib.stream_ptr() or torch.cuda.is_current_stream_capturing():
            self._await_copy()
        elif not self.is_prefill:
            # the short layers of a decode step need not ask again once it is done; the first one would mostly find it under way
            done = copied[2] and _lib.get_lib().mfb_event_done(copied[0].cuda_event, 0) == 0
            self._copied = None if done else copied[:2] + (True,)

    def _mark_copy(self, index: Optional[int]):
        """Behind the copy of the step's tensors on the current stream of a device."""
        here = torch.cuda.current_device()
        index = here if index is None else index
        stream = _lib.stream_ptr(index)
        if self._event is None or self._event[1] != index or index != here:
            self._event = (torch.cuda.Event(), index)
            self._event[0].record(torch.cuda.current_stream(index))
        else:                                # (a stream object costs more host time than this)
            _lib.check(_lib.get_lib().mfb_event_record(self._event[0].cuda_event, stream), "mfb_event_record")
        self._copied = (self._event[0], stream, False)

    def __getstate__(self):
        self._await_copy()
        return dict(self.__dict__, _event=None)

    @property
    def has_state(self) -> bool:
        """Whether some layer has a recurrent state: such a step cannot be run twice, nor tokens taken back."""
        return self.carry is not None or any(r is not None for r in self.recurrent)

    def _states(self) -> list:
        """Every state tensor, slots first."""
        return [t for r in self.recurrent for t in r or ()] + ([] if self.carry is None else [self.carry.transpose(0, 1)])

    def save_state(self) -> list:
        """Copy of the recurrent states (for runs that warm up or capture a step and must leave no trace)."""
        return [t.clone() for t in self._states()]

    def restore_state(self, saved: list):
        for t, old in zip(self._states(), saved):
            t.copy_(old)

    def copy_state(self, dst: List[int], src: List[int]):
        """Slot ``dst[i]`` continues from what slot ``src[i]`` holds now."""
        for t in self._states():
            t[dst] = t[src].clone()

    def set_step(self, *, is_prefill, block_tables, slot_mapping, context_lens, q_seq_lens, device):
        self.is_prefill = is_prefill
        q = [int(x) for x in q_seq_lens]
        cu = [0]
        for n in q:
            cu.append(cu[-1] + n)
        self.cu_q = cu
        self.prefill_work = {}
        # sequences without new tokens in this step (finished prompts of a chunked prefill, idle serving slots) have
        # no row of their own: one entry per sequence that has tokens
        last = [c - 1 for c, n in zip(cu[1:], q) if n > 0]
        given = (block_tables, slot_mapping, context_lens)
        self._copied = None
        if torch.device(device).type != "cuda" or any(isinstance(x, torch.Tensor) and x.is_cuda for x in given):
            self.block_tables, self.slot_mapping, self.context_lens = (
                torch.as_tensor(x, dtype=torch.int32, device=device).contiguous() for x in given)
            self.q_seq_lens = torch.as_tensor(q, dtype=torch.int32, device=device)
            self.last_token_index = torch.as_tensor(last, dtype=torch.int64, device=device)
        else:
            # one copy, in the order of the current stream, that the host does not wait for
            if torch.cuda.is_current_stream_capturing():
                raise RuntimeError("a step's metadata come from the host: set_step cannot be captured in a CUDA graph")
            # (numbers that do not fit are refused, as in the copies above)
            given = [np.asarray(x, dtype=np.int32) for x in given + (q,)]
            self.block_tables, self.slot_mapping, self.context_lens, self.q_seq_lens, index = _to_device(
                given + [np.asarray(last, np.int64).view(np.int32)], device)
            self.last_token_index = index.view(torch.int64)
            self._mark_copy(torch.device(device).index)
            self.host_lens = given[2].tolist()
        if self.carry is not None and is_prefill:
            self.carry_before.copy_(self.carry)
        if self.ragged and is_prefill:
            self.q_lens_host, self.context_lens_host = q, [int(x) for x in context_lens]
            self.n_long_rows, self.n_single_rows = sum(n > 1 for n in q), sum(n == 1 for n in q)
            self.cu_q_dev = torch.tensor(cu, dtype=torch.int32).to(device)


def _write_cache(cache: KVCacheContext, layer: int, k: torch.Tensor, v: Optional[torch.Tensor]):
    """k, v: [T, heads, hd] (views with token stride); scatter rows into the layer's cache by slot."""
    T = k.shape[0]
    kc, vc = cache.key_cache[layer], cache.value_cache[layer]
    row = k.shape[1] * k.shape[2]
    if getattr(cache, "int8", False):
        ks, vs = cache.key_scale[layer], cache.value_scale[layer]
        if k.is_cuda and k.dtype == torch.bfloat16 and k.stride(2) == 1 and k.stride(1) == k.shape[2] \
                and v.stride(2) == 1 and v.stride(1) == v.shape[2]:
            rc = _lib.get_lib().mfb_reshape_and_cache_int8(
                k.data_ptr(), v.data_ptr(), kc.data_ptr(), vc.data_ptr(), ks.data_ptr(), vs.data_ptr(),
                cache._slot_mapping.data_ptr(), T, k.shape[1], k.shape[2], k.stride(0), v.stride(0), _lib.stream_ptr())
            _lib.check(rc, "mfb_reshape_and_cache_int8")
            _lib.count_launch()
            return
        slots = cache._slot_mapping.long()
        ok = slots >= 0
        for src, dst, sc in ((k, kc, ks), (v, vc, vs)):
            x = src.reshape(T, src.shape[1], src.shape[2])[ok].float()
            amax = x.abs().amax(-1)
            scale = torch.where(amax > 0, amax / 127.0, torch.ones_like(amax))
            q = torch.round(x / scale.unsqueeze(-1)).clamp(-127, 127).to(torch.int8)
            dst.view(-1, src.shape[1], src.shape[2])[slots[ok]] = q
            sc.view(-1, src.shape[1])[slots[ok]] = scale
        return
    if k.is_cuda and k.dtype == torch.bfloat16 and row % 8 == 0 and k.stride(2) == 1 and k.stride(1) == k.shape[2]:
        rc = _lib.get_lib().mfb_reshape_and_cache(k.data_ptr(), _lib.ptr(v), kc.data_ptr(), _lib.ptr(vc),
                                                  cache._slot_mapping.data_ptr(), T, row, k.stride(0),
                                                  v.stride(0) if v is not None else 0, _lib.stream_ptr())
        _lib.check(rc, "mfb_reshape_and_cache")
        _lib.count_launch()
        return
    slots = cache._slot_mapping.long()
    ok = slots >= 0
    kc.view(-1, row)[slots[ok]] = k.reshape(T, row)[ok].to(kc.dtype)
    if v is not None:
        vc.view(-1, row)[slots[ok]] = v.reshape(T, row)[ok].to(vc.dtype)


def _gather(cache_t: torch.Tensor, table_row: torch.Tensor, n: int, block_size: int,
            scale_t: Optional[torch.Tensor] = None, dtype=None) -> torch.Tensor:
    """The first ``n`` cached rows of one sequence as a contiguous tensor (de-quantised when ``scale_t`` is given)."""
    nb = -(-n // block_size)
    blocks = table_row[:nb].long()
    rows = cache_t[blocks].reshape(nb * block_size, *cache_t.shape[2:])[:n]
    if scale_t is not None:
        sc = scale_t[blocks].reshape(nb * block_size, -1)[:n]
        rows = (rows.float() * sc.unsqueeze(-1)).to(dtype or torch.bfloat16)
    return rows


def _layer_scales(cache, layer):
    if getattr(cache, "int8", False):
        return cache.key_scale[layer], cache.value_scale[layer]
    return None, None


# Decode attention runs on the tensor cores: ``paged_decode_tc.cu`` over a bf16 cache with head dim 128, ``paged_decode_int8.cu`` over an
# int8 cache with blocks of a multiple of 16 tokens. ``MFB_PAGED_DECODE=cuda_core`` (or ``set_paged_decode_kernel``) keeps the split-KV
# kernel on the CUDA cores, which also serves what those two do not take: a bf16 cache with head dim 64, other block sizes.
_DECODE_KERNEL = "cuda_core" if os.environ.get("MFB_PAGED_DECODE", "tensor_core") == "cuda_core" else "tensor_core"


def set_paged_decode_kernel(kind: str) -> None:
    global _DECODE_KERNEL
    if kind not in ("tensor_core", "cuda_core"):
        raise ValueError("kind must be 'tensor_core' or 'cuda_core'")
    _DECODE_KERNEL = kind


_TILE = 128              # query rows of a tile of the prefill kernel
# Mean key tiles per query tile up to which a launch's CTAs walk over several tiles each (their loads then run under the softmax of
# the tile before); longer tiles differ too much in length for that and get a CTA each.
_PERSISTENT_UP_TO = 8.0


class _PrefillPlan:
    """What the prefill kernels need to know about a step: per query tile ``(sequence, first row of q, rows, position of the first
    row)``, longest first, for the sequences whose keys are all new (``fresh``) and for those with cached ones (``past``; of a cache of
    latents, all that have new rows); the first row of every sequence in q (``cu``), and in a gathered copy of the cached rows that the
    sequences of ``past`` see (``past_rows``). ``ok`` False: a step that
    these kernels do not take (a sequence longer than its block table or without one, rows that are not there, tables of another form)."""

    def __init__(self, cache, rows: int, lens: list, latent: bool):
        cu = cache.cu_q
        B = len(lens)
        tables = cache._block_tables
        fits = tables.dim() == 2 and tables.shape[0] >= B and tables.dtype == torch.int32 and tables.is_contiguous()
        reach = tables.shape[1] * cache.block_size if fits else -1
        news = [cu[b + 1] - cu[b] for b in range(B)] if len(cu) == B + 1 else []
        self.rows = cu[-1]
        self.ok = 0 < self.rows <= rows and len(news) == B and cu[0] == 0 and all(0 <= n <= m <= reach for n, m in zip(news, lens) if n)
        if not self.ok:
            return
        fresh, seeing = [], []
        first = [0]                            # rows of the copy
        for b, (n, m) in enumerate(zip(news, lens)):
            copied = n and (latent or n < m)
            (seeing if copied else fresh).extend((b, cu[b] + r, min(_TILE, n - r), m - n + r) for r in range(0, n, _TILE))
            first.append(first[-1] + (m if copied else 0))
        flat, self.longest = [], max(lens)
        spans = [self._add(flat, items) for items in (fresh, seeing)]
        at = len(flat)
        dev, = _to_device([np.asarray(flat + list(cu) + first, np.int32)], tables.device)
        (a, n, p), (b, m, s) = spans
        self.fresh, self.past = (dev[a:a + 4 * n], n, p), (dev[b:b + 4 * m], m, s)
        self.cu, self.past_rows, self.n_past_rows = dev[at:at + B + 1], dev[at + B + 1:], first[-1]
        self.past_host, self.groups, self.forms = (seeing, first), {}, {}
        self.new_and_seen = [(n, m) for n, m in zip(news, lens) if n] if latent else None

    def expands(self, heads: int) -> bool:
        """Whether multi-latent attention of ``heads`` heads expands the cached latents (one product over all rows that the step sees, whatever
        the new ones, 0.9 ns per row and head) or takes the queries into the latent space (sequence by sequence, 32-bit products: 0.056 ns per new
        row, cached row and head, some 0.1 ms besides, and 265 us of launches at least). Measured, expanded and absorbed: 128 heads, 32 sequences
        of 8000 rows, 1 / 4 / 16 new ones each 29.8 / 30.1 / 29.9 and 9.5 / 15.8 / 35.2 ms; 1 sequence 0.97 / 0.99 / 0.96 and 0.41 / 0.56 / 1.19 ms;
        32 of 2300 rows 8.5 / 8.5 / 8.8 and 8.5 / 9.1 / 14.2 ms; 16 heads, 4 of 2300 rows, 1 / 200 new ones 0.26 / 0.28 and 1.15 / 2.5 ms."""
        if heads not in self.forms:
            expanded = 110 + 0.9e-3 * self.n_past_rows * heads
            absorbed = sum(max(265, 90 + m * (0.005 + 0.0002 * heads) + 0.056e-3 * n * m * heads) for n, m in self.new_and_seen)
            self.forms[heads] = expanded <= absorbed
        return self.forms[heads]

    @staticmethod
    def _add(flat: list, items: list):
        """Appends a launch's tiles, longest first: where they start in ``flat``, how many they are, whether CTAs walk over several."""
        keys = lambda t: (t[3] + t[2] - 1) // _TILE + 1
        at, items = len(flat), sorted(items, key=keys, reverse=True)
        flat += [x for t in items for x in t]
        return at, len(items), sum(map(keys, items)) <= _PERSISTENT_UP_TO * len(items)

    def copied(self, limit: int) -> list:
        """``past`` in groups of sequences that see at most ``limit`` rows together (or one sequence): per group the work, the first row of
        every sequence in a copy of the rows that the group sees (``[B + 1]``, none for the others) and the rows of that copy."""
        if self.n_past_rows <= limit:
            return [(self.past, self.past_rows, self.n_past_rows)]
        if limit not in self.groups:
            tiles, first = self.past_host
            rows = [b - a for a, b in zip(first, first[1:])]
            members, held = [[]], 0
            for b, n in enumerate(rows):
                if n and held and held + n > limit:
                    members.append([])
                    held = 0
                if n:
                    members[-1].append(b)
                    held += n
            flat, parts = [], []
            for seqs in members:
                own, cu = set(seqs), [0]
                for b, n in enumerate(rows):
                    cu.append(cu[-1] + (n if b in own else 0))
                span = self._add(flat, [t for t in tiles if t[0] in own])
                parts.append((span, len(flat), cu[-1]))
                flat += cu + [0] * (-len(cu) % 4)            # the next group's tiles start on 16 bytes
            dev, = _to_device([np.asarray(flat, np.int32)], self.past_rows.device)
            self.groups[limit] = [((dev[a:a + 4 * n], n, p), dev[at:at + len(rows) + 1], total) for (a, n, p), at, total in parts]
        return self.groups[limit]


def _prefill_plan(cache, rows: int, latent: bool = False) -> _PrefillPlan:
    """The step's plan, shared by its layers: kept while all that it follows from has the values it had, on the stream that made it. A cache of
    latents wants other lists than one of keys and values."""
    lens, tables = _host_lens(cache), cache._block_tables
    key = (rows, latent, tuple(lens), tuple(cache.cu_q), tables.shape, cache.block_size, _lib.stream_ptr() if tables.is_cuda else 0)
    plan = cache.prefill_work.get("plan")
    if plan is None or plan.key != key:
        plan = cache.prefill_work["plan"] = _PrefillPlan(cache, rows, lens, latent)
        plan.key = key
    return plan


def _needs_graph(*tensors) -> bool:
    """Whether a derivative is wanted: the kernels of this module have none."""
    return (torch.is_grad_enabled() and any(t.requires_grad for t in tensors)) or torch.autograd.forward_ad._current_level >= 0


def _strided(q: torch.Tensor) -> torch.Tensor:
    """``[T, heads, dim]`` that a tensor map can describe: itself, or a copy."""
    ok = q.stride(2) == 1 and q.stride(1) >= q.shape[2] and q.stride(0) >= q.shape[2] and q.stride(1) % 8 == 0 and q.stride(0) % 8 == 0 \
        and q.data_ptr() % 16 == 0
    return q if ok else q.clone(memory_format=torch.contiguous_format)


def _decode_scratch(cache, need: int, device) -> torch.Tensor:
    """The partial results of decode steps (one buffer per cache)."""
    scratch = getattr(cache, "_decode_scratch", None)
    if scratch is None or scratch.numel() * 4 < need:
        scratch = cache._decode_scratch = torch.empty((need + 3) // 4, dtype=torch.float32, device=device)
    return scratch


def _decode_step(q, k, v, cache, layer: int, scale: float):
    """One new row per sequence: into the cache and attention over it in one call (bf16 cache of head dim 128: ``paged_decode_tc.cu``, int8
    cache: ``paged_decode_int8.cu``). None where those kernels do not take the call; nothing was written then."""
    B, nq, hd = q.shape
    kc, lens = cache.key_cache[layer], cache._context_lens
    ksc, vsc = _layer_scales(cache, layer)
    if not q.is_cuda or not (q.dtype == k.dtype == v.dtype == torch.bfloat16) or B != lens.shape[0] or k.shape != v.shape \
            or k.shape[0] != B or k.shape[2] != hd or kc.dtype != (torch.bfloat16 if ksc is None else torch.int8):
        return None
    out = torch.empty((B, nq * hd), dtype=torch.bfloat16, device=q.device)
    tables = cache._block_tables
    need = 0
    for _ in range(2):
        scratch = _decode_scratch(cache, need, q.device)
        rc = _lib.get_lib().mfb_paged_decode_step(
            q.data_ptr(), *q.stride(), k.data_ptr(), *k.stride(), v.data_ptr(), *v.stride(), kc.data_ptr(),
            cache.value_cache[layer].data_ptr(), _lib.ptr(ksc), _lib.ptr(vsc), cache._slot_mapping.data_ptr(), tables.data_ptr(),
            lens.data_ptr(), out.data_ptr(), scratch.data_ptr(), scratch.numel() * 4, B, nq, k.shape[1], hd, kc.shape[0],
            cache.block_size, tables.shape[1], scale, _lib.status_word(q.device).data_ptr(), _lib.stream_ptr())
        if rc <= 0:
            break
        need = rc
    if rc == -2:
        return _decode_step(*(t.clone(memory_format=torch.contiguous_format) for t in (q, k, v)), cache, layer, scale)
    if rc == -1:
        return None
    _lib.check(rc, "mfb_paged_decode_step")
    _lib.count_launch(3)
    return out


def _rows_ok(t: torch.Tensor) -> bool:
    """``[T, heads, dim]`` whose heads lie side by side and whose rows start on 16 bytes."""
    return (t.dtype == torch.bfloat16 and t.stride(2) == 1 and t.stride(1) == t.shape[2] and t.stride(0) % 8 == 0
            and t.stride(0) >= t.shape[1] * t.shape[2] and t.data_ptr() % 16 == 0)


_COPIED_BYTES = 1 << 30          # of cached rows copied out at a time; the sequences of a step that see more take turns


def _ragged_prefill(q, k, v, cache, layer: int, scale: float):
    """Prefill attention of a step's sequences: those without history attend over their own rows of ``k`` / ``v``, the others over
    the cache (an int8 cache, or one of other block sizes than the kernel's, through a copy of the rows they see) with weights that are not
    rounded. None where the kernel does not take the call."""
    T, nq, hd = q.shape
    nkv = k.shape[1]
    if not (q.is_cuda and q.dtype == torch.bfloat16 and hd in (64, 128) and v.shape == k.shape and k.shape[2] == hd and k.shape[0] == T
            and T and nkv and nq % nkv == 0 and Fn.get_attention_backend() == "auto") or _needs_graph(q, k, v):
        return None
    plan = _prefill_plan(cache, T)
    if not plan.ok or (plan.fresh[1] and not (_rows_ok(k) and _rows_ok(v))):
        return None
    kc, vc = cache.key_cache[layer], cache.value_cache[layer]
    ksc, vsc = _layer_scales(cache, layer)
    if plan.past[1] and (kc.dtype != (torch.bfloat16 if ksc is None else torch.int8) or not kc.is_contiguous() or not vc.is_contiguous()
                         or plan.n_past_rows >= 1 << 31 or plan.longest * nkv * hd >= 1 << 34):
        return None
    q = _strided(q)
    lib, st, stream = _lib.get_lib(), _lib.status_word(q.device).data_ptr(), _lib.stream_ptr()
    out = torch.empty((plan.rows, nq * hd), dtype=q.dtype, device=q.device)

    def launch(work, keys, values, ld_k, ld_v, key_rows, key_row, exact):
        rc = lib.mfb_ragged_prefill_tc(
            q.data_ptr(), q.stride(0), q.stride(1), keys, values, ld_k, ld_v, work[0].data_ptr(), work[1], cache._block_tables.data_ptr(),
            cache._block_tables.shape[1], cache.block_size, key_rows, _lib.ptr(key_row), out.data_ptr(), out.stride(0), T, nq, nkv, hd,
            hd, int(exact), int(work[2]), float(scale), st, stream)
        _lib.check(rc, "mfb_ragged_prefill_tc")
        _lib.count_launch()

    if plan.fresh[1]:
        launch(plan.fresh, k.data_ptr(), v.data_ptr(), k.stride(0), v.stride(0), T, plan.cu, False)
    if plan.past[1]:
        row = nkv * hd
        if ksc is None and lib.mfb_ragged_prefill_tc_supported(nq, nkv, hd, hd, cache.block_size):
            launch(plan.past, kc.data_ptr(), vc.data_ptr(), row, row, kc.shape[0] * cache.block_size, None, True)
        else:
            groups = plan.copied(max(1, _COPIED_BYTES // (2 * row * 2)))
            copies = torch.empty((2, max(g[2] for g in groups), row), dtype=q.dtype, device=q.device)
            for work, first, rows in groups:
                _gather_rows(cache, copies, (kc, vc), (ksc, vsc), first, plan.longest)
                launch(work, copies[0].data_ptr(), copies[1].data_ptr(), row, row, rows, first, True)
    return out


def _gather_rows(cache, outs, rows, scales, cu, longest: int):
    """Cached rows of the sequences of ``cu [B + 1]``, one after the other, out of one or two caches of the same shape; de-quantised where
    ``scales`` are given."""
    lib, tables = _lib.get_lib(), cache._block_tables
    B, max_blocks = cu.numel() - 1, tables.shape[1]
    heads, dim = rows[0].shape[2:]
    if scales[0] is None:
        rc = lib.mfb_gather_cache2(rows[0].data_ptr(), rows[1].data_ptr() if len(rows) > 1 else 0, tables.data_ptr(), cu.data_ptr(),
                                   outs[0].data_ptr(), outs[1].data_ptr() if len(rows) > 1 else 0, B, longest, cache.block_size, max_blocks,
                                   heads * dim, _lib.stream_ptr())
        _lib.check(rc, "mfb_gather_cache2")
        _lib.count_launch()
        return
    for out, src, scale in zip(outs, rows, scales):
        rc = lib.mfb_gather_cache_int8(src.data_ptr(), scale.data_ptr(), tables.data_ptr(), cu.data_ptr(), out.data_ptr(), B, longest,
                                       cache.block_size, max_blocks, heads, dim, _lib.stream_ptr())
        _lib.check(rc, "mfb_gather_cache_int8")
        _lib.count_launch()


def paged_attention_forward(q, k, v, meta, layer_number: int, scale: float):
    """q: [T, nq, hd]; k/v: [T, nkv, hd] of the new tokens. Returns [T, nq*hd]."""
    cache: KVCacheContext = meta.cache
    cache._in_order()
    layer = layer_number - 1 - cache.layer_offset
    if not cache.is_prefill and _DECODE_KERNEL == "tensor_core":
        out = _decode_step(q, k, v, cache, layer, scale)
        if out is not None:
            return out
    _write_cache(cache, layer, k, v)
    T, nq, hd = q.shape
    nkv = k.shape[1]
    B = cache._context_lens.shape[0]
    if not cache.is_prefill and T == B:
        out = torch.empty((T, nq, hd), dtype=q.dtype, device=q.device)
        if q.is_cuda and q.dtype == torch.bfloat16 and hd in (64, 128) and nq // nkv <= 16:
            lib = _lib.get_lib()
            max_blocks = cache._block_tables.shape[1]
            ksc, vsc = _layer_scales(cache, layer)
            qc = q.contiguous()
            splits = lib.mfb_paged_decode_splits(B, nkv, cache.block_size, max_blocks)
            rc = lib.mfb_paged_decode_attention_ex(
                qc.data_ptr(), cache.key_cache[layer].data_ptr(), cache.value_cache[layer].data_ptr(),
                _lib.ptr(ksc), _lib.ptr(vsc),
                cache._block_tables.data_ptr(), cache._context_lens.data_ptr(), out.data_ptr(),
                _decode_scratch(cache, lib.mfb_paged_decode_scratch_bytes(B, nq, hd, splits), q.device).data_ptr(), splits, B, nq, nkv, hd,
                cache.block_size, max_blocks, float(scale), _lib.stream_ptr())
            _lib.check(rc, "mfb_paged_decode_attention_ex")
            _lib.count_launch(2)
            return out.view(T, nq * hd)
        lens = cache._context_lens.tolist()
        ksc, vsc = _layer_scales(cache, layer)
        for b in range(B):
            kk = _gather(cache.key_cache[layer], cache._block_tables[b], lens[b], cache.block_size, ksc, q.dtype)
            vv = _gather(cache.value_cache[layer], cache._block_tables[b], lens[b], cache.block_size, vsc, q.dtype)
            o = Fn.attention_reference(q[b:b + 1].unsqueeze(0), kk.unsqueeze(0), vv.unsqueeze(0), causal=False, scale=scale)
            out[b] = o[0, 0]
        return out.view(T, nq * hd)
    # prefill (optionally with history, e.g. chunked prefill): causal attention of all sequences in one or two launches
    out = _ragged_prefill(q, k, v, cache, layer, scale)
    if out is not None:
        return out
    # other types, sizes and layouts: sequence by sequence
    outs = []
    lens = _host_lens(cache)
    for b in range(B):
        a, e = cache.cu_q[b], cache.cu_q[b + 1]
        if e == a:
            continue
        nq_tok = e - a
        if lens[b] == nq_tok:
            o = Fn.attention(q[a:e].unsqueeze(0), k[a:e].unsqueeze(0), v[a:e].unsqueeze(0), causal=True, scale=scale)
        else:
            ksc, vsc = _layer_scales(cache, layer)
            kk = _gather(cache.key_cache[layer], cache._block_tables[b], lens[b], cache.block_size, ksc, q.dtype)
            vv = _gather(cache.value_cache[layer], cache._block_tables[b], lens[b], cache.block_size, vsc, q.dtype)
            o = Fn.attention_reference(q[a:e].unsqueeze(0), kk.unsqueeze(0), vv.unsqueeze(0), causal=True, scale=scale,
                                       q_offset=lens[b] - nq_tok)
        outs.append(o.reshape(nq_tok, nq * v.shape[-1]))
    return torch.cat(outs, dim=0)


def set_mla_decode_variant(variant: str) -> None:
    """Choose the MLA decode kernel: ``"single"`` (one CTA per work item, ``ops/csrc/mla_decode.cu``) or ``"cluster"``
    (two CTAs of a cluster split the latent columns and read the cache once, ``ops/csrc/mla_decode_cluster.cu``)."""
    if variant not in ("single", "cluster"):
        raise ValueError(f"unknown MLA decode variant {variant!r}")
    _lib.get_lib().mfb_mla_decode_set_variant(1 if variant == "cluster" else 0)


def mla_decode_attention(q_cat: torch.Tensor, latent_cache: torch.Tensor, block_tables: torch.Tensor,
                         context_lens: torch.Tensor, block_size: int, scale: float, holder=None) -> torch.Tensor:
    """``q_cat [B, heads, 576]`` (absorbed query ‖ rope query) against the paged latent cache
    ``[num_blocks, block_size, (1,) 576]`` → latent-space output ``[B, heads, 512]``; ``context_lens`` counts the
    tokens in the cache, the current one included. ``holder`` keeps the scratch buffer between calls."""
    B, nh, dim = q_cat.shape
    if dim != 576 or q_cat.dtype != torch.bfloat16 or latent_cache.dtype != torch.bfloat16:
        raise ValueError("mla_decode_attention: bf16 tensors with a latent width of 512 + 64 are required")
    lib = _lib.get_lib()
    max_blocks = block_tables.shape[1]
    splits = lib.mfb_mla_decode_splits(B, nh, max_blocks * block_size)
    need = lib.mfb_mla_decode_scratch_bytes(B, nh, splits)
    scratch = getattr(holder, "_mla_scratch", None) if holder is not None else None
    if scratch is None or scratch.numel() * 4 < need:
        scratch = torch.empty((need + 3) // 4, dtype=torch.float32, device=q_cat.device)
        if holder is not None:
            holder._mla_scratch = scratch
    out = torch.empty((B, nh, 512), dtype=torch.bfloat16, device=q_cat.device)
    num_blocks = latent_cache.shape[0]
    rc = lib.mfb_mla_decode_attention(q_cat.data_ptr(), latent_cache.data_ptr(), block_tables.data_ptr(),
                                      context_lens.data_ptr(), out.data_ptr(), scratch.data_ptr(), splits, B, nh,
                                      num_blocks, block_size, max_blocks, float(scale),
                                      _lib.status_word(q_cat.device).data_ptr(), _lib.stream_ptr())
    _lib.check(rc, "mfb_mla_decode_attention")
    _lib.count_launch(2)
    return out


_EXPANDED_BYTES = 2 << 30        # of expanded keys and values at a time; more heads than that take turns


def _latent_prefill(attn, q_nope, q_pe, cache, layer: int):
    """Multi-latent attention of a step's new rows (any lengths, with or without history) over keys and values expanded from the
    cached latents once per call. Expanded numbers are kept as the sum of two bf16 numbers and the softmax weights likewise, so that
    nothing between query and result is rounded to 16 bits. None where the kernel does not take the call or too few rows ask for it."""
    T, nh, nope = q_nope.shape
    rope_d, vd, rank = attn.rope_d, attn.vd, attn.kv_rank
    w, rows = attn.linear_kvb.weight, cache.key_cache[layer]
    if not (q_nope.is_cuda and q_nope.dtype == q_pe.dtype == rows.dtype == w.dtype == torch.bfloat16 and (nope, rope_d, vd) == (128, 64, 128)
            and rank % 8 == 0 and T and w.is_contiguous() and rows.is_contiguous() and Fn.get_gemm_backend() == "tcgen05") or _needs_graph(q_nope, q_pe, w):
        return None
    plan = _prefill_plan(cache, T, latent=True)
    if not plan.ok or plan.n_past_rows >= 1 << 31 or plan.longest * (rank + rope_d) >= 1 << 34 or not plan.expands(nh):
        return None
    q_pe = q_pe.reshape(T, nh, rope_d)
    q_nope, q_pe = _strided(q_nope), _strided(q_pe)
    lib, dev = _lib.get_lib(), q_nope.device
    out = torch.empty((plan.rows, nh * vd), dtype=torch.bfloat16, device=dev)
    groups = plan.copied(max(1, _COPIED_BYTES // (2 * (rank + rope_d))))
    latent = torch.empty((max(g[2] for g in groups), rank + rope_d), dtype=torch.bfloat16, device=dev)
    for work, first, n in groups:
        _gather_rows(cache, [latent], [rows], [None], first, plan.longest)
        step = max(1, min(nh, _EXPANDED_BYTES // (n * 256 * 8)))
        for h in range(0, nh, step):
            heads = min(step, nh - h)
            kv = Fn.gemm(latent[:n, :rank], w[h * 256:(h + heads) * 256], out_dtype=torch.float32)
            parts = torch.empty((2,) + kv.shape, dtype=torch.bfloat16, device=dev)
            hi, lo = parts.data_ptr(), parts.data_ptr() + 2 * kv.numel()
            rc = lib.mfb_split_f32(kv.data_ptr(), hi, lo, kv.numel(), _lib.stream_ptr())
            _lib.check(rc, "mfb_split_f32")
            rc = lib.mfb_latent_prefill_tc(
                q_nope.data_ptr() + 2 * h * q_nope.stride(1), q_nope.stride(0), q_nope.stride(1), q_pe.data_ptr() + 2 * h * q_pe.stride(1),
                q_pe.stride(0), q_pe.stride(1), hi, lo, latent.data_ptr() + 2 * rank, rank + rope_d, n, first.data_ptr(),
                work[0].data_ptr(), work[1], out.data_ptr() + 2 * h * vd, out.stride(0), T, heads, float(attn.scale),
                _lib.status_word(dev).data_ptr(), _lib.stream_ptr())
            _lib.check(rc, "mfb_latent_prefill_tc")
            _lib.count_launch(2)
            del kv, parts                # before the next ones are allocated
    return out


def _write_latents(cache, layer: int, kv_c: torch.Tensor, k_pe: torch.Tensor):
    """New latents ``[T, rank]`` and rotated key parts ``[T, rope]``, side by side, into the layer's cache."""
    rows, (T, rank), rope = cache.key_cache[layer], kv_c.shape, k_pe.shape[1]
    if kv_c.is_cuda and kv_c.dtype == k_pe.dtype == rows.dtype == torch.bfloat16 and rank % 8 == rope % 8 == 0 and T \
            and all(t.stride(1) == 1 and t.stride(0) % 8 == 0 and t.data_ptr() % 16 == 0 for t in (kv_c, k_pe)) \
            and rows.is_contiguous() and rows.shape[-1] == rank + rope:
        rc = _lib.get_lib().mfb_latent_to_cache(kv_c.data_ptr(), kv_c.stride(0), k_pe.data_ptr(), k_pe.stride(0), rows.data_ptr(),
                                                cache._slot_mapping.data_ptr(), T, rank, rope, _lib.stream_ptr())
        _lib.check(rc, "mfb_latent_to_cache")
        _lib.count_launch()
        return
    _write_cache(cache, layer, torch.cat((kv_c, k_pe), dim=-1).unsqueeze(1).contiguous(), None)


def mla_paged_attention_forward(attn, q_nope, q_pe, kv_c, k_pe, meta):
    """Multi-latent attention with a latent cache ``[kv_lora ‖ k_pe]``.

    Prefill expands K/V from the latent with ``linear_kvb``; decode absorbs the up-projections: queries are
    mapped into the latent space (``q_nope @ W_UK``), attention runs against the cached latents, and the result is
    mapped back with ``W_UV`` (reference ``multi_latent_attention.py:219-231,434-448``).
    """
    cache: KVCacheContext = meta.cache
    cache._in_order()
    layer = attn.layer_number - 1 - cache.layer_offset
    T = q_nope.shape[0]
    _write_latents(cache, layer, kv_c, k_pe.reshape(T, -1))
    nh, nope, rope_d, vd, rank = attn.nh, attn.nope, attn.rope_d, attn.vd, attn.kv_rank
    w = attn.linear_kvb.weight.view(nh, nope + vd, rank)
    w_uk, w_uv = w[:, :nope], w[:, nope:]                                      # [nh, nope, rank], [nh, vd, rank]
    B = cache._context_lens.shape[0]
    if (not cache.is_prefill and T == B and q_nope.is_cuda and q_nope.dtype == torch.bfloat16 and rank == 512
            and rope_d == 64 and cache.block_size in (16, 32, 64, 128)):
        # decode: absorbed queries against the latent cache in one tcgen05 kernel (ops/csrc/mla_decode.cu)
        q_lat = torch.einsum("bhn,hnr->bhr", q_nope, w_uk)
        q_cat = torch.cat((q_lat, q_pe.reshape(B, nh, rope_d)), dim=-1).contiguous()
        o_lat = mla_decode_attention(q_cat, cache.key_cache[layer], cache._block_tables, cache._context_lens,
                                     cache.block_size, attn.scale, cache)
        return torch.einsum("bhr,hvr->bhv", o_lat, w_uv).reshape(B, nh * vd)
    lens = _host_lens(cache)
    q_lens = [cache.cu_q[b + 1] - cache.cu_q[b] for b in range(B)]
    if (cache.is_prefill and q_nope.is_cuda and q_nope.dtype == torch.bfloat16 and nope == 128 and rope_d == 64
            and vd == 128 and all(ql == n and ql % 128 == 0 and ql > 0 for ql, n in zip(q_lens, lens))):
        # prefill without history: expand K / V from the latents and run the flash-attention kernel (192 / 128 heads)
        from ..ops import attention as native
        kv = attn._col_nosp(attn.linear_kvb, kv_c).view(T, nh, nope + vd)
        k = torch.cat((kv[..., :nope], k_pe.reshape(T, 1, rope_d).expand(T, nh, rope_d)), dim=-1)
        v = kv[..., nope:]
        qf = torch.cat((q_nope, q_pe), dim=-1)
        if len(set(q_lens)) == 1:
            S = q_lens[0]
            o = native.mla_forward(qf.view(B, S, nh, -1), k.view(B, S, nh, -1), v.reshape(B, S, nh, vd), True, attn.scale)
            return o.reshape(T, nh * vd)
        outs = []
        for b in range(B):
            a, e = cache.cu_q[b], cache.cu_q[b + 1]
            o = native.mla_forward(qf[a:e].unsqueeze(0), k[a:e].unsqueeze(0), v[a:e].unsqueeze(0), True, attn.scale)
            outs.append(o.reshape(e - a, nh * vd))
        return torch.cat(outs, dim=0)
    out = _latent_prefill(attn, q_nope, q_pe, cache, layer)
    if out is not None:
        return out
    outs = []
    for b in range(B):
        a, e = cache.cu_q[b], cache.cu_q[b + 1]
        if e == a:
            continue
        lat = _gather(cache.key_cache[layer], cache._block_tables[b], lens[b], cache.block_size)[:, 0]  # [L, rank+rope]
        c, pe = lat[:, :rank].float(), lat[:, rank:].float()
        q_lat = torch.einsum("thn,hnr->thr", q_nope[a:e].float(), w_uk.float())    # absorbed query
        s = (torch.einsum("thr,lr->htl", q_lat, c) + torch.einsum("thd,ld->htl", q_pe[a:e].float(), pe)) * attn.scale
        nq_tok, L = e - a, lens[b]
        qi = torch.arange(nq_tok, device=s.device).unsqueeze(-1) + (L - nq_tok)
        ki = torch.arange(L, device=s.device).unsqueeze(0)
        s = s.masked_fill((ki > qi).unsqueeze(0), float("-inf"))
        p = torch.softmax(s, dim=-1)
        o_lat = torch.einsum("htl,lr->thr", p, c)
        o = torch.einsum("thr,hvr->thv", o_lat, w_uv.float())
        outs.append(o.reshape(nq_tok, nh * vd).to(q_nope.dtype))
    return torch.cat(outs, dim=0)
