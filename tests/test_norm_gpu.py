"""Norms of narrow rows and of packed query / key heads: sizes at which their kernels change form."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _rms(x, w, eps):
    x = x.double()
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w.double()


def _close(got, want, rel):
    err = (got.double() - want).norm() / want.norm().clamp_min(1e-30)
    assert err < rel, float(err)


# rows of 8 .. 32 lanes, of one to four vectors per lane, the first size of the CTA-wide form; rows that do not fill a warp or a CTA
@pytest.mark.parametrize("H", [8, 64, 72, 128, 136, 256, 264, 512, 520, 1024, 1032])
@pytest.mark.parametrize("T", [1, 7, 33, 20000])
@pytest.mark.parametrize("residual", [False, True])
def test_rmsnorm_rows(H, T, residual):
    from mindformers_b200.ops import functional as Fn
    torch.manual_seed(H)
    x, r = (torch.randn(T, H, device=DEV).to(torch.bfloat16).requires_grad_() for _ in range(2))
    w = (1 + 0.1 * torch.randn(H, device=DEV)).to(torch.bfloat16).requires_grad_()
    dy, dh = (torch.randn(T, H, device=DEV).to(torch.bfloat16) for _ in range(2))
    y, h = Fn.rmsnorm(x, w, 1e-5, r if residual else None)
    torch.autograd.backward([y, h] if residual else [y], [dy, dh] if residual else [dy])
    h64 = (x + r if residual else x).detach().double().requires_grad_()
    w64 = w.detach().double().requires_grad_()
    want = _rms(h64, w64, 1e-5)
    want.backward(dy.double())
    # results are sums in 32 bits, rounded once: at most 2^-8 of every number
    _close(y, want.detach(), 4e-3)
    _close(x.grad, h64.grad + (dh.double() if residual else 0), 4e-3)
    _close(w.grad, w64.grad, 4e-3)


@pytest.mark.parametrize("T,nq,nkv,hd", [(1, 1, 1, 8), (5, 4, 2, 64), (130, 32, 8, 128), (2048, 7, 1, 128), (33, 3, 3, 200), (64, 4, 1, 256)])
@pytest.mark.parametrize("buffers", [False, True])
def test_qk_norm(T, nq, nkv, hd, buffers):
    """``buffers``: gradients go into the weights' fp32 buffers, which hold earlier ones."""
    from mindformers_b200.ops import functional as Fn
    torch.manual_seed(T)
    x = torch.randn(T, nq + 2 * nkv, hd, device=DEV).to(torch.bfloat16).requires_grad_()
    ws = [(1 + 0.1 * torch.randn(hd, device=DEV)).to(torch.bfloat16).requires_grad_() for _ in range(2)]
    dy = torch.randn(T, nq + 2 * nkv, hd, device=DEV).to(torch.bfloat16)
    if buffers:
        for w in ws:
            w.main_grad = torch.full((hd,), 3.0, device=DEV)
    assert Fn.qk_norm_supported(x, *ws)
    y = Fn.qk_norm(x, *ws, nq, nkv, 1e-6, 1e-5)
    y.backward(dy)
    x64 = x.detach().double().requires_grad_()
    w64 = [w.detach().double().requires_grad_() for w in ws]
    want = torch.cat((_rms(x64[:, :nq], w64[0], 1e-6), _rms(x64[:, nq:nq + nkv], w64[1], 1e-5), x64[:, nq + nkv:]), 1)
    want.backward(dy.double())
    _close(y, want.detach(), 4e-3)
    _close(x.grad, x64.grad, 4e-3)
    assert torch.equal(y[:, nq + nkv:], x[:, nq + nkv:]) and torch.equal(x.grad[:, nq + nkv:], dy[:, nq + nkv:])
    for w, ref in zip(ws, w64):
        if buffers:
            assert w.grad is None
        _close(w.main_grad - 3.0 if buffers else w.grad, ref.grad, 4e-3)


def test_swiglu_in_several_launches():
    """Rows so wide that the vector indexes of a launch would pass 2^31 with more than one of them."""
    from mindformers_b200.ops import functional as Fn
    torch.manual_seed(0)
    T, F = 3, 1 << 24
    x = torch.randn(T, 2 * F, device=DEV, dtype=torch.bfloat16).requires_grad_()
    dy = torch.randn(T, F, device=DEV, dtype=torch.bfloat16)
    y = Fn.swiglu(x)
    dx = torch.autograd.grad(y, x, dy)[0]
    for t in range(T):
        row = x.detach()[t].float().requires_grad_()
        want = torch.nn.functional.silu(row[:F]) * row[F:]
        _close(y[t].detach(), want.detach().double(), 4e-3)              # rounded once, at most 2^-8 of every number
        _close(dx[t], torch.autograd.grad(want, row, dy[t].float())[0].double(), 4e-3)
