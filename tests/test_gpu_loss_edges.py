"""Output-head loss: wide rows of cross-entropy, the bookkeeping kernels around the rows, and who owns the gradients."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm().clamp(min=1e-30)).item()


# one bf16 rounding (8 significant bits) of the result
ONE_ROUNDING = 2.0 ** -8


@pytest.mark.parametrize("R,V", [(1, 16384), (300, 16391), (149, 20000), (5, 57600), (3, 57601)])
def test_wide_rows(R, V):
    """More rows than CTAs run at once, a tail, labels in the tail and the last vector, ignored rows, minus infinity and the
    type's lowest value among the entries."""
    from kolmogorov_moe_architecture_b200.ops import cuda_ops as c
    torch.manual_seed(V)
    pitch = -(-V // 64) * 64
    buf = torch.full((R, pitch), float("nan"), dtype=torch.bfloat16, device="cuda")
    buf[:, :V] = (torch.randn(R, V, device="cuda") * 3).to(torch.bfloat16)
    buf[:, 7] = float("-inf")
    buf[:, V // 2] = torch.finfo(torch.bfloat16).min
    buf[0, 0] = 60.0
    lab = torch.randint(8, V // 3, (R,), device="cuda")
    lab[0] = V - 1
    if R > 2:
        lab[1], lab[2] = -100, V // 8 * 8 - 1
    lg = buf[:, :V].double()
    ref = torch.nn.functional.cross_entropy(lg, lab, ignore_index=-100, reduction="none")
    p = (torch.softmax(lg, -1) - torch.nn.functional.one_hot(lab.clamp(min=0), V)) * 0.37
    p[lab == -100] = 0
    gs = torch.full((1,), 0.37, device="cuda")
    only = c.K.ce_fwd_bwd(buf[:, :V], lab, gs, -100, False)
    assert torch.equal(buf[:, :V].double(), lg)
    rows = c.K.ce_fwd_bwd(buf[:, :V], lab, gs, -100, True)
    assert torch.equal(only, rows)
    assert (rows.double() - ref).abs().max() < 2.0 ** -18 * ref.abs().max().clamp(min=1)     # 32-bit sums
    assert _rel(buf[:, :V], p) < ONE_ROUNDING
    assert buf[:, V:].isnan().all()


def test_rows_not_finite():
    """Rows of minus infinity only, with a NaN, with plus infinity: no number, as in torch, and the rows beside them unharmed."""
    from kolmogorov_moe_architecture_b200.ops import cuda_ops as c
    V = 16400
    buf = torch.zeros(4, -(-V // 64) * 64, dtype=torch.bfloat16, device="cuda")
    buf[0], buf[1, 5], buf[2, 6] = float("-inf"), float("nan"), float("inf")
    rows = c.K.ce_fwd_bwd(buf[:, :V], torch.tensor([3, 4, 5, 6], device="cuda"), torch.ones(1, device="cuda"), -100, True)
    assert rows[:3].isnan().all() and abs(rows[3].item() - torch.tensor(float(V)).log().item()) < 1e-5


@pytest.mark.parametrize("B,S,n", [(3, 1, 2), (2, 3, 4), (1, 70, 2), (2, 129, 3)])
@pytest.mark.parametrize("dtype", [torch.long, torch.int32])
def test_heads_and_labels(B, S, n, dtype):
    """Sequences shorter than the heads reach, every label ignored for one head, labels of another integer type."""
    from kolmogorov_moe_architecture_b200.ops import cuda_ops as c
    torch.manual_seed(S)
    V, d = 200, 64
    h = torch.randn(B, S, d, device="cuda").bfloat16().requires_grad_(True)
    Ws = [(torch.randn(V, d, device="cuda") * 0.2).bfloat16().requires_grad_(True) for _ in range(n)]
    lab = torch.randint(0, V, (B, S), device="cuda")
    lab[:, S // 2:] = -100
    w = tuple(1.0 / (i + 1) for i in range(n))
    total, per = c.mtp_cross_entropy(h, Ws, lab.to(dtype), w)
    hd, Wd = h.detach().double().requires_grad_(True), [W.detach().double().requires_grad_(True) for W in Ws]
    want = 0.0
    for i, W in enumerate(Wd):
        tgt = lab[:, i + 1:].reshape(-1)
        lg = (hd[:, :max(S - i - 1, 0)] @ W.t()).reshape(-1, V)
        ce = torch.nn.functional.cross_entropy(lg, tgt, ignore_index=-100, reduction="sum") / max(1, int((tgt != -100).sum()))
        assert abs(per[i].item() - ce.item()) < 0.01          # logits are rounded to bf16: 2^-8 of values up to 5
        want = want + w[i] * ce
    assert abs(total.item() - want.item()) < 0.02
    assert torch.allclose(total, (per * torch.tensor(w, device="cuda")).sum(), rtol=1e-6)
    got = torch.autograd.grad(total, [h, *Ws], allow_unused=True)
    assert [g is None for g in got] == [False] + [i + 1 >= S for i in range(n)]
    for g, r in zip(got, torch.autograd.grad(want, [hd, *Wd])):
        if g is not None:
            assert (g.double() - r).norm() <= 0.02 * r.norm()  # probabilities from rounded logits, two bf16 roundings


def test_label_shapes():
    """One row of labels serves every sequence; labels without a batch dimension, of one column or of another length are
    refused, and none are looked at where no head has anything to predict."""
    from kolmogorov_moe_architecture_b200.ops import cuda_ops as c
    torch.manual_seed(0)
    B, S, V, d = 3, 9, 96, 64
    h = torch.randn(B, S, d, device="cuda").bfloat16()
    Ws = [(torch.randn(V, d, device="cuda") * 0.2).bfloat16() for _ in range(2)]
    row = torch.randint(0, V, (1, S), device="cuda")
    run = lambda lab, n=2, x=h: c.mtp_cross_entropy(x, Ws[:n], lab, (1.0, 0.5)[:n])
    assert all(torch.equal(a, b) for a, b in zip(run(row), run(row.repeat(B, 1))))
    assert all(torch.equal(a, b) for a, b in zip(run(row.cpu().float()), run(row)))
    for shape in [(S,), (B, 1), (1, 1), (B, S - 1), (B, S + 1), (2, S), (B, S, 1)]:
        with pytest.raises((IndexError, RuntimeError)):
            run(torch.zeros(shape, dtype=torch.long, device="cuda"))
    assert run(torch.zeros(4, dtype=torch.long, device="cuda"), 1, h[:, :1])[0].item() == 0.0


@pytest.mark.parametrize("how", ["retain", "hooks", "scaled"])
def test_gradients_are_nobody_elses(how):
    """The forward pass's buffers become the gradients only in the graph's last pass; a retained graph and saved-tensor hooks
    get copies, whatever the caller does with the first pass's gradients."""
    from kolmogorov_moe_architecture_b200.ops import cuda_ops as c
    torch.manual_seed(0)
    h = torch.randn(2, 40, 64, device="cuda").bfloat16().requires_grad_(True)
    W = (torch.randn(96, 64, device="cuda") * 0.2).bfloat16().requires_grad_(True)
    lab = torch.randint(0, 96, (2, 40), device="cuda")
    one = torch.autograd.grad(c.mtp_cross_entropy(h, [W], lab, (1.0,))[0], [h, W])
    if how == "scaled":
        got = torch.autograd.grad(c.mtp_cross_entropy(h, [W], lab, (1.0,))[0] * 4.0, [h, W])
        assert all(torch.equal(g, 4.0 * o) for g, o in zip(got, one))
    elif how == "retain":
        total = c.mtp_cross_entropy(h, [W], lab, (1.0,))[0]
        first = torch.autograd.grad(total, [h, W], retain_graph=True)
        for g in first:
            g.zero_()
        got = torch.autograd.grad(total, [h, W])
        assert all(torch.equal(g, o) for g, o in zip(got, one)) and not any(g.any() for g in first)
    else:
        held = []
        with torch.autograd.graph.saved_tensors_hooks(lambda t: held.append(t) or t, lambda t: t):
            total = c.mtp_cross_entropy(h, [W], lab, (1.0,))[0]
        before = [t.clone() for t in held]
        got = torch.autograd.grad(total * 2.0, [h, W])
        assert all(torch.equal(a, b) for a, b in zip(held, before))
        assert all(torch.equal(g, 2.0 * o) for g, o in zip(got, one))
