"""The mixer as one pass against the composition of the single ops and against 64 bits: odd token counts, narrow dt ranks,
several segments, small parameters in bf16 and fp32."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm().clamp(min=1e-30)).item()


@pytest.mark.parametrize("B,S,d,small", [(1, 7, 128, "bf16"), (2, 33, 256, "bf16"), (3, 24, 384, "fp32"), (1, 333, 768, "bf16"),
                                         (2, 72, 1024, "bf16")])
def test_one_pass_equals_single_ops(B, S, d, small, monkeypatch):
    from kolmogorov_moe_architecture_b200 import ops
    from kolmogorov_moe_architecture_b200.models.mamba import Mamba
    from kolmogorov_moe_architecture_b200.ops import cuda_ops
    torch.manual_seed(S)
    with torch.device("cuda"):
        m = Mamba(d).to(torch.bfloat16)
        if small == "fp32":
            for p in (m.conv1d.weight, m.conv1d.bias, m.dt_proj.bias, m.A_log, m.D):
                p.data = p.data.float()
    x = torch.randn(B, S, d, device="cuda").to(torch.bfloat16).requires_grad_(True)
    go = torch.randn(B, S, d, device="cuda").to(torch.bfloat16)
    leaves = [x, *m.parameters()]

    def run():
        y = m(x)
        return (y, *torch.autograd.grad(y, leaves, go))
    one = run()
    with torch.no_grad():
        assert torch.equal(m(x), one[0])
    monkeypatch.setattr(ops, "mamba_inner", lambda *a: None)
    many = run()
    cuda_ops.check_status()
    # the same quantities with fewer roundings to bf16 in between (1.7e-3 each): a handful of them in quadrature
    for a, b in zip(one, many):
        assert a.shape == b.shape and a.dtype == b.dtype and _rel(a, b) < 1e-2
