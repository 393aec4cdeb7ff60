"""The mixer as one pass against the composition of the single ops and against plain torch in 64 bits: odd token counts,
narrow dt ranks, several segments, small parameters in bf16 and fp32."""
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


def _mixer64(m, x, p):
    """The mixer's definition in plain torch; ``p`` holds the parameters by name."""
    B, S, _ = x.shape
    F, R = torch.nn.functional, m.dt_rank
    u, z = F.linear(x, p["in_proj.weight"]).chunk(2, dim=-1)
    u = F.silu(F.conv1d(u.transpose(1, 2), p["conv1d.weight"], p["conv1d.bias"], padding=3, groups=u.shape[-1])[..., :S].transpose(1, 2))
    dt, Bm, Cm = F.linear(u, p["x_proj.weight"]).split([R, 16, 16], dim=-1)
    dt = F.softplus(F.linear(dt, p["dt_proj.weight"], p["dt_proj.bias"]))
    A, h, ys = -torch.exp(p["A_log"]), u.new_zeros(B, u.shape[-1], 16), []
    for t in range(S):
        h = torch.exp(dt[:, t, :, None] * A) * h + (dt[:, t] * u[:, t])[..., None] * Bm[:, t, None, :]
        ys.append((h * Cm[:, t, None, :]).sum(-1))
    return F.linear((torch.stack(ys, 1) + u * p["D"]) * F.silu(z), p["out_proj.weight"])


@pytest.mark.parametrize("B,S,d", [(1, 7, 128), (2, 72, 256), (1, 333, 768)])
def test_one_pass_against_64_bits(B, S, d):
    """A dozen bf16 roundings (1.7e-3 each) lie on the longest way from an input to a gradient; in quadrature 6e-3, and the
    gradients of dt's side are sums of mixed signs, hence three times that."""
    from kolmogorov_moe_architecture_b200.models.mamba import Mamba
    from kolmogorov_moe_architecture_b200.ops import cuda_ops
    torch.manual_seed(S)
    with torch.device("cuda"):
        m = Mamba(d).to(torch.bfloat16)
    x = torch.randn(B, S, d, device="cuda").to(torch.bfloat16).requires_grad_(True)
    go = torch.randn(B, S, d, device="cuda").to(torch.bfloat16)
    names = [n for n, _ in m.named_parameters()]
    y = m(x)
    got = (y, *torch.autograd.grad(y, [x, *m.parameters()], go))
    cuda_ops.check_status()
    leaves = [t.detach().double().requires_grad_() for t in (x, *m.parameters())]
    ref = _mixer64(m, leaves[0], dict(zip(names, leaves[1:])))
    for n, a, b in zip(["y", "x", *names], got, (ref, *torch.autograd.grad(ref, leaves, go.double()))):
        assert _rel(a, b) < 1.8e-2, n


@pytest.mark.parametrize("frozen", ["x_proj", "dt_proj"])
def test_a_frozen_projection_gets_no_gradient(frozen):
    """With destinations registered for both weights, only the trained one's is written and committed."""
    from kolmogorov_moe_architecture_b200.models.mamba import Mamba
    from kolmogorov_moe_architecture_b200.ops import cuda_ops
    torch.manual_seed(0)
    with torch.device("cuda"):
        m = Mamba(128).to(torch.bfloat16)
    views, done = {}, []
    ws = {"x_proj": m.x_proj.weight, "dt_proj": m.dt_proj.weight}
    try:
        for n, w in ws.items():
            views[n] = torch.full_like(w, 7.0)
            cuda_ops.register_grad_sink(w, views[n], lambda p, n=n: done.append(n))
        ws[frozen].requires_grad_(False)
        x = torch.randn(2, 24, 128, device="cuda").to(torch.bfloat16)
        m(x).float().square().mean().backward()
    finally:
        for w in ws.values():
            cuda_ops._GRAD_SINKS.pop(w.data_ptr(), None)
    (trained,) = set(ws) - {frozen}
    assert done == [trained]
    assert (views[frozen] == 7.0).all() and not (views[trained] == 7.0).any()


@pytest.mark.parametrize("which", ["x_proj", "dt_proj"])
def test_a_projection_off_the_16_byte_grid(which, monkeypatch):
    """A weight that TMA cannot address is left to the single ops, which take it at an odd token count."""
    monkeypatch.setenv("KMOE_STRICT", "0")
    from kolmogorov_moe_architecture_b200.models.mamba import Mamba
    torch.manual_seed(0)
    with torch.device("cuda"):
        m = Mamba(128).to(torch.bfloat16)
    x = torch.randn(1, 13, 128, device="cuda").to(torch.bfloat16)
    with torch.no_grad():
        want = m(x)
        w = getattr(m, which).weight
        w.data = torch.cat([w.data.new_zeros(1), w.data.flatten()])[1:].view_as(w)
        assert w.data_ptr() % 16 == 2
        assert _rel(m(x), want) < 1e-2            # as the two routes differ in test_one_pass_equals_single_ops
