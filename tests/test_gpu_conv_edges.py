"""Causal convolution at the edges of its stretches of 32 steps and 64 channels, with odd channel counts and starts (one
channel per thread) and column slices (two)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

TOL = 4e-3          # one rounding to bf16 (1.7e-3 in the 2-norm) and 32-bit sums


@pytest.mark.parametrize("B,S,C,act,off", [(1, 1, 2, True, 0), (2, 31, 66, True, 0), (1, 33, 64, False, 8), (2, 259, 130, True, 2),
                                           (1, 35, 7, True, 0), (3, 256, 33, True, 1), (1, 700, 128, True, 0)])
def test_conv(B, S, C, act, off):
    from kolmogorov_moe_architecture_b200.ops import cuda_ops, eager
    torch.manual_seed(S)
    wide = torch.randn(B, S, 2 * C + 16 + (-(2 * C)) % 8, device="cuda").to(torch.bfloat16)
    x = wide[..., off:off + C].detach().requires_grad_(True)
    w, b = (torch.randn(C, 4, device="cuda", requires_grad=True), torch.randn(C, device="cuda", requires_grad=True))
    go = torch.randn(B, S, C, device="cuda").to(torch.bfloat16)
    y = cuda_ops.causal_conv1d(x, w, b, act)
    got = (y, *torch.autograd.grad(y, (x, w, b), go))
    xr, wr, br = (t.detach().double().requires_grad_(True) for t in (x, w, b))
    yr = eager.causal_conv1d(xr, wr, br, act)
    want = (yr, *torch.autograd.grad(yr, (xr, wr, br), go.double()))
    for g, r in zip(got, want):
        assert ((g.double() - r).norm() / r.norm().clamp(min=1e-30)).item() < TOL


@pytest.mark.parametrize("T,d", [(1, 256), (7, 768), (33, 1280), (4097, 1536), (130, 1792), (3000, 2048), (5, 1600)])
@pytest.mark.parametrize("residual", [False, True])
def test_norm_rows(T, d, residual):
    """RMSNorm at every register-resident width, a generic one, few and many rows (one, some and all blocks)."""
    from kolmogorov_moe_architecture_b200 import ops
    torch.manual_seed(T)
    mk = lambda: torch.randn(T, d, device="cuda").to(torch.bfloat16)
    x, a, g, gh = mk().requires_grad_(True), mk(), mk(), mk()
    w = torch.randn(d, device="cuda").to(torch.bfloat16).requires_grad_(True)
    h, y = ops.residual_rmsnorm(x, a if residual else None, w, 1e-5)
    got = (h, y, *torch.autograd.grad((h, y), (x, w), (gh, g)))
    xr, wr = x.detach().double().requires_grad_(True), w.detach().double().requires_grad_(True)
    hr = xr + a.double() if residual else xr * 1
    hr = hr + (h.detach().double() - hr.detach())                         # the norm works on the rounded sum
    yr = wr * hr * torch.rsqrt(hr.square().mean(-1, keepdim=True) + 1e-5)
    want = (hr, yr, *torch.autograd.grad((hr, yr), (xr, wr), (gh.double(), g.double())))
    for u, v in zip(got, want):
        assert ((u.double() - v).norm() / v.norm()).item() < TOL
