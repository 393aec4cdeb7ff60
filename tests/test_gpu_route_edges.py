"""Routing at its edges: one token, odd counts, all expert widths of a warp, bf16 and fp32 logits with ties; the plan with
empty experts, dropped assignments and several warps' stretches; the combine with long, mostly empty slot lists."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,E,k", [(1, 1, 1), (3, 4, 2), (97, 33, 3), (2500, 64, 2), (4097, 16, 8), (130, 128, 4)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_route(T, E, k, dtype):
    from kolmogorov_moe_architecture_b200.ops import cuda_ops
    torch.manual_seed(T)
    logits = torch.randn(T, E, device="cuda").to(dtype)
    logits[::3] = logits[::3].round()                                     # many ties
    x = logits.clone().requires_grad_(True)
    w, idx, aux, counts = cuda_ops.route_topk(x, k, 0.3, 0.1)
    r = logits.double().requires_grad_(True)
    ridx = torch.sort(r, dim=-1, descending=True, stable=True).indices[:, :k]
    p = torch.softmax(r, -1)
    rw = p.gather(1, ridx)
    rw = rw / rw.sum(-1, keepdim=True)
    rc = torch.bincount(ridx.reshape(-1), minlength=E)
    raux = 0.3 * E * (rc / (T * k) * p.mean(0)).sum() + 0.1 * torch.logsumexp(r, -1).square().mean()
    assert torch.equal(idx, ridx) and torch.equal(counts.long(), rc)       # whole numbers; the lower index wins a tie
    gw = torch.randn(T, k, device="cuda").to(dtype)
    got = torch.autograd.grad((w, aux), x, (gw, torch.ones_like(aux)))[0]
    want = torch.autograd.grad((rw, raux), r, (gw.double(), torch.ones_like(raux)))[0]
    tol = 4e-3 if dtype == torch.bfloat16 else 1e-5                        # one rounding of the result / 32-bit sums
    assert (w.double() - rw).norm() <= tol * rw.norm()
    assert abs(aux.item() - raux.item()) <= 1e-5 * abs(raux.item()) + 1e-12
    # k = E: the weights are the softmax itself and its gradient cancels to the auxiliary part, hence the floor
    assert (got.double() - want).norm() <= tol * want.norm() + 1e-6 * gw.double().norm()


@pytest.mark.parametrize("n,E", [(1, 3), (31, 1), (1024, 16), (1025, 64), (12289, 33), (5000, 164)])
@pytest.mark.parametrize("drop", [False, True])
def test_plan(n, E, drop):
    from kolmogorov_moe_architecture_b200.ops import cuda_ops
    torch.manual_seed(n)
    idx = torch.randint(0, max(1, E - 1), (n,), device="cuda")             # the last expert stays empty
    keep = torch.rand(n, device="cuda") < 0.7 if drop else None
    pos, row_src, counts, offsets, tile_group, meta = [t.cpu() for t in cuda_ops.K.moe_plan(idx, keep, E, 0)]
    ids, kp = idx.cpu(), keep.cpu() if drop else torch.ones(n, dtype=torch.bool)
    run, tiles = 0, []
    want_rows = torch.full_like(row_src, -1)
    want_pos = torch.full_like(pos, -1)
    for e in range(E):
        a = ((ids == e) & kp).nonzero().flatten()
        assert counts[e] == a.numel() and offsets[e] == run
        want_rows[run:run + a.numel()] = a.int()
        want_pos[a] = torch.arange(run, run + a.numel(), dtype=torch.int32)
        nt = -(-a.numel() // 128)
        tiles += [e] * nt
        run += nt * 128
    assert offsets[E] == run and meta.tolist() == [len(tiles), run]
    assert torch.equal(row_src, want_rows) and torch.equal(pos, want_pos)
    assert tile_group.tolist() == tiles + [0] * (tile_group.numel() - len(tiles))


@pytest.mark.parametrize("T,k,d", [(1, 1, 8), (37, 2, 264), (300, 16, 2048), (9, 40, 1096)])
@pytest.mark.parametrize("weighted", [False, True])
def test_combine(T, k, d, weighted):
    from kolmogorov_moe_architecture_b200.ops import cuda_ops
    torch.manual_seed(k)
    rows = max(1, T * k // 3)
    Y = torch.randn(rows, d, device="cuda").to(torch.bfloat16)
    pos = torch.full((T * k,), -1, dtype=torch.int32, device="cuda")
    at = torch.randperm(T * k, device="cuda")[:rows]
    pos[at] = torch.arange(rows, dtype=torch.int32, device="cuda")
    w = torch.rand(T * k, device="cuda") if weighted else None
    out = cuda_ops.K.moe_combine(Y, pos, w, T, k)
    scale = (w if weighted else torch.ones(T * k, device="cuda")).double()
    ref = torch.zeros(T, d, dtype=torch.double, device="cuda")
    ref.index_add_(0, at // k, Y.double() * scale[at, None])
    assert (out.double() - ref).norm() <= 4e-3 * ref.norm()


@pytest.mark.parametrize("S,k", [(1, 1), (2, 1), (33, 33), (64, 5), (65, 64), (129, 17), (1536, 96), (16384, 700)])
def test_softmax_topk(S, k):
    """Order and positions are exact: larger first, lower position first among equals, -0 equal to +0."""
    from kolmogorov_moe_architecture_b200.ops import cuda_ops
    torch.manual_seed(S)
    B, E = 2, 3
    logits = torch.randn(B, S, E, device="cuda")
    logits[0, :, 0] = (logits[0, :, 0] * 2).round() / 2                    # ties, both zeros
    logits[0, ::2, 1] = float("-inf")                                      # masked positions (the last expert has none)
    if S > 2:
        logits[1, :, 2] = torch.tensor([0.0, -0.0], device="cuda").repeat(S)[:S]
    w, tok = cuda_ops.expert_choice_route(logits, k)
    x = logits.transpose(1, 2).double()
    order = torch.sort(x, dim=-1, descending=True, stable=True).indices[..., :k]
    assert torch.equal(tok, order)
    p = torch.softmax(x, -1).gather(-1, order)
    ref = p / (p.sum(-1, keepdim=True) + 1e-9)
    ok = torch.isfinite(ref).all(-1)                                       # S = 1: a row of -inf alone has no softmax
    # 32-bit sums of at most 16384 exponentials with a relative error of 2^-21 each (the fast exponential at |x| < 20)
    assert ((w.double() - ref).abs() <= 1e-5 * ref + 1e-30)[ok].all()


@pytest.mark.parametrize("at", [0, 40])
def test_softmax_topk_keeps_positions_valid_with_nan(at):
    from kolmogorov_moe_architecture_b200.ops import cuda_ops
    logits = torch.randn(1, 50, 1, device="cuda")
    logits[0, at, 0] = -float("nan")
    _, tok = cuda_ops.expert_choice_route(logits, 50)
    assert tok[0, 0, 0] == at and torch.equal(tok.sort(dim=-1).values[0, 0], torch.arange(50, device="cuda"))


@pytest.mark.parametrize("T,k,d", [(1, 1, 8), (37, 2, 264), (200, 4, 2048), (65, 3, 1032)])
def test_gather_with_weight_gradient(T, k, d):
    from kolmogorov_moe_architecture_b200.ops import cuda_ops
    torch.manual_seed(d)
    E = 5
    idx = torch.randint(0, E, (T * k,), device="cuda")
    keep = torch.rand(T * k, device="cuda") < 0.7
    pos, row_src, _, _, _, meta = cuda_ops.K.moe_plan(idx, keep, E, 0)
    rows = row_src.numel()
    Y = torch.randn(rows, d, device="cuda").bfloat16()
    Y[row_src < 0] = float("nan")                                          # never read
    dout, w = torch.randn(T, d, device="cuda").bfloat16(), torch.rand(T * k, device="cuda")
    dY, dw = cuda_ops.K.moe_gather_dw(dout, row_src, w, Y, meta, pos, k, 0, 0)
    live = int(meta[1])
    a = row_src[:live].long()
    ref = torch.where((a >= 0)[:, None], dout[a.clamp(min=0) // k].float() * w[a.clamp(min=0), None], 0.0).bfloat16()
    assert torch.equal(dY[:live], ref)                                     # one product, one rounding
    p = pos.long()
    prod = torch.where((p >= 0)[:, None], dout.double().repeat_interleave(k, 0) * Y[p.clamp(min=0)].double(), 0.0)
    # products of bf16 are exact in 32 bits; a sum of d of them
    assert ((dw.double() - prod.sum(-1)).abs() <= d * 2.0 ** -24 * prod.abs().sum(-1)).all()


@pytest.mark.parametrize("B,S,E,C,d", [(1, 1, 1, 1, 8), (3, 50, 4, 13, 264), (2, 300, 33, 300, 136)])
def test_choice_bookkeeping(B, S, E, C, d):
    from kolmogorov_moe_architecture_b200.ops import cuda_ops
    torch.manual_seed(S)
    T = B * S
    tok = torch.stack([torch.randperm(S, device="cuda")[:C] for _ in range(B * E)]).view(B, E, C)
    wts = torch.rand(B, C, E, device="cuda").transpose(1, 2)               # strided
    status = cuda_ops.status_tensor(tok.device)
    row_src, pos, weight, meta = cuda_ops.K.moe_choice_plan(tok.int(), wts, S, T, status)
    a = ((tok + torch.arange(B, device="cuda").view(B, 1, 1) * S) * E + torch.arange(E, device="cuda").view(1, E, 1))
    rows = a.permute(1, 0, 2).reshape(-1)
    want = torch.full((T * E,), -1, dtype=torch.int32, device="cuda")
    want[rows] = torch.arange(rows.numel(), dtype=torch.int32, device="cuda")
    assert torch.equal(row_src.long(), rows) and torch.equal(pos, want) and meta.tolist() == [rows.numel()] * 2
    assert torch.equal(weight[a], wts)
    Y, dout = torch.randn(rows.numel(), d, device="cuda").bfloat16(), torch.randn(T, d, device="cuda").bfloat16()
    _, dw = cuda_ops.K.moe_gather_dw(dout, row_src, weight, Y, meta, pos, E, B, C)
    prod = dout[rows // E].double() * Y.double()
    bound = (d * 2.0 ** -24 * prod.abs().sum(-1)).view(E, B, C).transpose(0, 1)
    assert ((dw.view(B, E, C).double() - prod.sum(-1).view(E, B, C).transpose(0, 1)).abs() <= bound).all()
    tok[0, 0, 0] = T + 7                                                   # outside: an empty row and an error
    row_src, *_ = cuda_ops.K.moe_choice_plan(tok, wts, S, T, status)
    assert row_src[0] == -1
    with pytest.raises(RuntimeError, match="status 31"):
        cuda_ops.check_status()


@pytest.mark.parametrize("bad", [-1, 20, 45])
def test_a_token_outside_its_sequence_is_an_error(bad):
    """Also in the first sequence of a batch, where the index would name a row of the next one."""
    from kolmogorov_moe_architecture_b200.ops import cuda_ops
    B, S, E, C = 2, 20, 2, 3
    tok = torch.arange(C, device="cuda").repeat(B, E, 1)
    tok[0, 1, 2] = bad
    status = cuda_ops.status_tensor(tok.device)
    row_src, pos, *_ = cuda_ops.K.moe_choice_plan(tok, torch.ones(B, E, C, device="cuda"), S, B * S, status)
    assert row_src[B * C + 2] == -1 and (row_src >= 0).sum() == B * E * C - 1 and (pos >= 0).sum() == B * E * C - 1
    with pytest.raises(RuntimeError, match="token index outside its sequence"):
        cuda_ops.check_status()


def test_expert_choice_keeps_nothing_without_gradients():
    """Under no_grad the pre-activations (two rows x f bf16 buffers) are neither formed nor kept."""
    from kolmogorov_moe_architecture_b200 import ops
    torch.manual_seed(0)
    B, S, d, f, E, C = 2, 256, 64, 1024, 4, 128
    x = torch.randn(B, S, d, device="cuda").bfloat16()
    ws = [torch.nn.Parameter((torch.randn(*s, device="cuda") * 0.1).bfloat16()) for s in ((E, d, f), (E, d, f), (E, f, d))]
    w, tok = ops.expert_choice_route(torch.randn(B, S, E, device="cuda"), C)
    got = []
    for enabled in (False, True):
        with torch.set_grad_enabled(enabled):
            for _ in range(2):
                out = None
                torch.cuda.synchronize()
                held = torch.cuda.memory_allocated()
                torch.cuda.reset_peak_memory_stats()
                out = ops.expert_choice_swiglu(x, *ws, w, tok)
                peak = torch.cuda.max_memory_allocated() - held
        got.append((peak, out.detach().clone()))
    assert torch.equal(got[0][1], got[1][1])
    assert got[0][0] <= got[1][0] - 2 * (E * B * C * f * 2)
