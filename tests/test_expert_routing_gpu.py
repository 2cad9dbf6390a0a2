"""Stable ranks of token copies within their experts (lists that end inside a thread, a warp and a round); the gate in 32-bit precision;
products of a few rows per expert."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("n", [1, 5, 4095, 4096, 4097, 13000])
@pytest.mark.parametrize("E", [1, 7, 512])
def test_expert_ranks(n, E):
    from mindformers_b200.ops import _lib
    torch.manual_seed(n)
    ids = torch.randint(0, E + 1, (n,), device=DEV)              # E itself: a copy without an expert
    rank, counts = torch.full((n,), -1, dtype=torch.int32, device=DEV), torch.zeros(E, dtype=torch.int32, device=DEV)
    _lib.check(_lib.get_lib().mfb_moe_rank(ids.data_ptr(), n, E, rank.data_ptr(), counts.data_ptr(), _lib.stream_ptr()), "rank")
    hot = torch.nn.functional.one_hot(ids, E + 1)[:, :E]
    assert torch.equal(counts.long(), hot.sum(0))
    want = ((hot.cumsum(0) - 1) * hot).sum(1)
    assert torch.equal(rank.long(), torch.where(ids < E, want, -1))


# rows on both sides of the CUDA-core kernel's limit, of its eight-row and the products' 128- and 256-row tiles; experts short of a tile
@pytest.mark.parametrize("T", [1, 9, 192, 193, 300, 1000])
@pytest.mark.parametrize("E,H", [(8, 64), (128, 2048), (264, 1088)])
def test_gate(T, E, H):
    from mindformers_b200.ops import functional as Fn
    torch.manual_seed(T)
    x = torch.randn(T, H, device=DEV).to(torch.bfloat16).requires_grad_()
    w = (torch.randn(E, H, device=DEV) * 0.02).requires_grad_()
    dy = torch.randn(T, E, device=DEV)
    assert Fn.gate_supported(x, w)
    y = Fn.gate_logits(x, w)
    y.backward(dy)
    x64, w64 = x.detach().double(), w.detach().double()
    rel = lambda got, want: float((got.double() - want).norm() / want.norm())
    # sums of up to 2048 products in 32 bits, each off by 2^-24 of its sum: 2^-24 sqrt(2048) / 2 if they are rounded one by one; a
    # dropped third part of an operand would show as 2^-17
    assert rel(y.detach(), x64 @ w64.t()) < 1.4e-6
    assert rel(w.grad, dy.double().t() @ x64) < 1.4e-6
    assert rel(x.grad, dy.double() @ w64) < 4e-3                   # rounded to bf16, at most 2^-8 of every number
    with torch.no_grad():
        assert torch.equal(Fn.gate_logits(x, w), y)
    assert Fn._lib.read_status() == 0


# experts without rows, with one, a whole short tile, one more, a whole block and several blocks; widths short of a tile
@pytest.mark.parametrize("fills", [[0, 1, 32, 0, 33], [128, 5, 0, 64, 96], [300, 2, 31, 1, 0], [1] * 40])
@pytest.mark.parametrize("N,K", [(1536, 2048), (200, 64), (136, 768)])
def test_grouped_short_tiles(fills, N, K):
    from mindformers_b200.ops import functional as Fn
    from mindformers_b200.ops import _lib
    torch.manual_seed(N)
    G = len(fills)
    offsets = [0]
    for n in fills:
        offsets.append(offsets[-1] + -(-n // 128) * 128)
    blocks = [g for g in range(G) for _ in range((offsets[g + 1] - offsets[g]) // 128)]
    R = offsets[-1] + 128
    a = torch.full((R, K), float("nan"), device=DEV).to(torch.bfloat16)        # padding rows may hold anything
    b = (torch.randn(G, K, N, device=DEV) * K ** -0.5).to(torch.bfloat16)
    for g, n in enumerate(fills):
        a[offsets[g]:offsets[g] + n] = torch.randn(n, K, device=DEV).to(torch.bfloat16)
    dev = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    out = torch.empty((R, N), dtype=torch.bfloat16, device=DEV)
    plan = [dev(v) for v in (blocks + [G - 1], [len(blocks)], offsets, fills)]
    rc = _lib.get_lib().mfb_gemm_bf16_grouped_short(
        a.data_ptr(), b.data_ptr(), out.data_ptr(), R, N, K, K, N, N, G, *(t.data_ptr() for t in plan),
        _lib.status_word(DEV).data_ptr(), _lib.stream_ptr())
    _lib.check(rc, "mfb_gemm_bf16_grouped_short")
    for g, n in enumerate(fills):
        if n:
            rows = slice(offsets[g], offsets[g] + n)
            want = a[rows].double() @ b[g].double()
            assert float((out[rows].double() - want).norm() / want.norm()) < 4e-3       # one rounding, at most 2^-8
    assert _lib.read_status() == 0


def test_gate_backward_in_a_graph():
    """The backward pass of a token count that was not there before can be captured."""
    from mindformers_b200.ops import functional as Fn
    torch.manual_seed(0)
    x = torch.randn(700, 256, device=DEV).to(torch.bfloat16).requires_grad_()
    w = torch.randn(128, 256, device=DEV).requires_grad_()
    dy = torch.randn(700, 128, device=DEV)

    def step(n):
        return torch.autograd.grad(Fn.gate_logits(x[:n], w), (x, w), dy[:n])
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step(700)
        step(700)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = step(513)
    for t in got:
        t.zero_()
    graph.replay()
    assert all(torch.equal(a, b) for a, b in zip(got, step(513)))
    assert Fn._lib.read_status() == 0


def _gate(x, w):
    """The router's logits, by the kernels where they take the call."""
    from mindformers_b200.ops import functional as Fn
    return Fn.gate_logits(x, w) if Fn.gate_supported(x, w) else torch.nn.functional.linear(x.float(), w)


@pytest.mark.parametrize("T", [40, 300])
def test_gate_under_transforms(T):
    """Second derivatives, forward mode, vmap and traces of the gate are those of the plain product."""
    import torch.autograd.forward_ad as fwd
    torch.manual_seed(T)
    x = torch.randn(T, 64, device=DEV).to(torch.bfloat16).requires_grad_()
    w = torch.randn(8, 64, device=DEV).requires_grad_()
    seconds = []
    for gate in (_gate, lambda x, w: torch.nn.functional.linear(x.float(), w)):
        gx, gw = torch.autograd.grad(gate(x, w).pow(3).sum(), (x, w), create_graph=True)
        seconds.append(torch.autograd.grad(gx.float().pow(2).sum() + gw.pow(2).sum(), (x, w)))
    for a, b in zip(*seconds):
        # the first pass adds up in another order (1e-6) and its gradient of x is rounded to bf16, at most 2^-8
        assert (a.float() - b.float()).norm() / b.float().norm() < 8e-3
    with torch.no_grad():
        plain, xd, wd = torch.nn.functional.linear(x.float(), w), x.detach(), w.detach()
        with fwd.dual_level():
            out = fwd.unpack_dual(_gate(fwd.make_dual(xd, torch.ones_like(xd)), wd))
        want = wd.sum(1).expand_as(out.tangent)
        assert (out.tangent - want).norm() / want.norm() < 1e-5
        both = torch.func.vmap(_gate, (0, None))(torch.stack((xd, xd)), wd)
        assert (both[1] - plain).norm() / plain.norm() < 1e-5
        traced = torch.jit.trace(_gate, (xd, wd), check_trace=False)
        assert (traced(2 * xd, wd) - 2 * plain).norm() / plain.norm() < 1e-5


def test_gate_on_views():
    """A gradient that starts between two 16-byte boundaries; rows that are one row repeated."""
    from mindformers_b200.ops import functional as Fn
    torch.manual_seed(0)
    T, E, H = 300, 128, 64
    x = torch.randn(T, H, device=DEV).to(torch.bfloat16).requires_grad_()
    w = torch.randn(E, H, device=DEV).requires_grad_()
    dy = torch.randn(T * E + 1, device=DEV)[1:].view(T, E)
    got = torch.autograd.grad(Fn.gate_logits(x, w), (x, w), dy)
    want = torch.autograd.grad(Fn.gate_logits(x, w), (x, w), dy.clone())
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    row = x.detach()[:1].expand(T, H).requires_grad_()
    logits = _gate(row, w)
    grads = torch.autograd.grad(logits, (row, w), dy)
    plain = torch.nn.functional.linear(row.float(), w)
    for a, b in zip((logits, *grads), (plain, *torch.autograd.grad(plain, (row, w), dy))):
        assert (a.float() - b.float()).norm() / b.float().norm() < 8e-3          # bf16 gradients, at most 2^-8 on either side


def test_gate_gradient_in_turns(monkeypatch):
    """The sums of blocks of rows that the weight's gradient is made of stay within their bytes, whatever the number of rows."""
    from mindformers_b200.ops import functional as Fn
    torch.manual_seed(0)
    T, E, H = 5000, 128, 512
    x = torch.randn(T, H, device=DEV).to(torch.bfloat16)
    w = (torch.randn(E, H, device=DEV) * 0.02).requires_grad_()
    dy = torch.randn(T, E, device=DEV)
    want = dy.double().t() @ x.double()
    taken = []
    for limit in (Fn._GATE_BYTES, 3 * 12 * E * H):                        # three blocks of 256 rows at a time
        monkeypatch.setattr(Fn, "_GATE_BYTES", limit, raising=False)
        y = Fn.gate_logits(x, w)
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        got = torch.autograd.grad(y, w, dy)[0]
        taken.append(torch.cuda.max_memory_allocated() - before)
        assert float((got.double() - want).norm() / want.norm()) < 1.4e-6         # as in test_gate
    assert taken[1] < taken[0] - 16 * 12 * E * H
    assert Fn._lib.read_status() == 0
