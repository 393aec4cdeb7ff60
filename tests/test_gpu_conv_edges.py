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
