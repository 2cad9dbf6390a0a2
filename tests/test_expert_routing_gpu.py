"""Stable ranks of token copies within their experts (lists that end inside a thread, a warp and a round); the gate in 32-bit precision."""
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
