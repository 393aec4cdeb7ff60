"""Sizes that are no whole number of 64-element blocks on the GEMM paths: operand rows read in single boxes, padded
split reductions, odd vocabularies."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(out, ref):
    return ((out.double() - ref.double()).norm() / ref.double().norm().clamp(min=1e-30)).item()


def _rand(*shape, scale=1.0):
    return (torch.randn(*shape, device="cuda") * scale).to(torch.bfloat16)


# One rounding of the result to bf16 is 2^-9 at most and about 1.7e-3 in the 2-norm; the sums are in 32 bits.
ONE_ROUNDING = 4e-3


@pytest.mark.parametrize("M,N,K", [(72, 72, 64), (136, 200, 72), (264, 328, 8), (2464, 1000, 192), (1000, 2464, 640)])
def test_mn_major_rows_in_boxes(M, N, K):
    from kolmogorov_moe_architecture_b200.ops import cuda_ops as c
    a, b = _rand(K, M), _rand(K, N)
    out = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device="cuda")
    c.mm_tn(a, b, out=out)                                     # both operands MN-major
    c.check_status()
    assert _rel(out, a.double().t() @ b.double()) < ONE_ROUNDING
    x = _rand(M, K)
    assert _rel(c.mm_nn(x, b), x.double() @ b.double()) < ONE_ROUNDING
    c.check_status()


@pytest.mark.parametrize("rows,V,d", [(128, 65, 64), (300, 50257 % 1000 + 1000, 192), (136, 127, 128)])
def test_odd_row_count_and_odd_reduction(rows, V, d):
    """The three products of an output head whose vocabulary is odd; guard bands around every operand hold NaN."""
    from kolmogorov_moe_architecture_b200.ops import cuda_ops as c
    pitch = -(-V // 64) * 64
    guard = torch.full((V + 64, d), float("nan"), dtype=torch.bfloat16, device="cuda")
    W = guard[:V]
    W.copy_(_rand(V, d))
    h = _rand(rows, d)
    buf = torch.full((rows, pitch), float("nan"), dtype=torch.bfloat16, device="cuda")
    c.gemm(h, W, buf, M=rows, N=-(-V // 8) * 8, Kd=d, lda=d, ldb=d, ldc=pitch, b_rows=V)
    assert _rel(buf[:, :V], h.double() @ W.double().t()) < ONE_ROUNDING
    dh = torch.empty(rows, d, dtype=torch.bfloat16, device="cuda")
    c.gemm(buf, W, dh, M=rows, N=d, Kd=V, b_major=c.MAJ_MN, lda=pitch, ldb=d, ldc=d)
    assert _rel(dh, buf[:, :V].double() @ W.double()) < ONE_ROUNDING
    dW = torch.full((V + 8, d), 7.0, dtype=torch.bfloat16, device="cuda")
    c.gemm(buf, h, dW, M=V, N=d, Kd=rows, a_major=c.MAJ_MN, b_major=c.MAJ_MN, lda=pitch, ldb=d, ldc=d)
    c.check_status()
    assert _rel(dW[:V], buf[:, :V].double().t() @ h.double()) < ONE_ROUNDING
    assert (dW[V:] == 7.0).all()


# Rounded to bf16 on the way: gate, up, hidden, the rows and dH, dG, dU - seven roundings of about 1.7e-3 that add in
# quadrature to 4.5e-3 at most; twice that.
EXPERT_TOL = 9e-3


def _expert_case(E, d, f):
    return [_rand(E, d, f, scale=d ** -0.5), _rand(E, d, f, scale=d ** -0.5), _rand(E, f, d, scale=f ** -0.5)]


@pytest.mark.parametrize("T,d,f,E,k", [(1, 64, 72, 3, 2), (200, 192, 88, 4, 2), (333, 72, 2464, 5, 1), (515, 1792, 136, 64, 2)])
def test_expert_widths(T, d, f, E, k):
    from kolmogorov_moe_architecture_b200 import ops
    from kolmogorov_moe_architecture_b200.ops import cuda_ops, eager
    torch.manual_seed(T)
    ws = _expert_case(E, d, f)
    x = _rand(T, d)
    wts, idx = eager.topk_softmax_route(torch.randn(T, E, device="cuda"), k)
    wts = wts.to(torch.bfloat16)
    go = _rand(T, d)
    leaves = [t.clone().requires_grad_() for t in (x, *ws, wts)]
    out = ops.grouped_swiglu(*leaves[:4], idx, leaves[4])
    got = (out, *torch.autograd.grad(out, leaves, go))
    cuda_ops.check_status()
    ref_leaves = [t.double().requires_grad_() for t in (x, *ws, wts)]
    ref = eager.grouped_swiglu(*ref_leaves[:4], idx, ref_leaves[4])
    want = (ref, *torch.autograd.grad(ref, ref_leaves, go.double()))
    for g, w in zip(got, want):
        if w.norm() > 0:
            assert _rel(g, w) < EXPERT_TOL


@pytest.mark.parametrize("B,S,d,f,E", [(1, 65, 64, 72, 3), (2, 130, 136, 200, 4)])
def test_expert_choice_widths(B, S, d, f, E):
    from kolmogorov_moe_architecture_b200 import ops
    from kolmogorov_moe_architecture_b200.ops import cuda_ops, eager
    torch.manual_seed(S)
    ws = _expert_case(E, d, f)
    x = _rand(B, S, d)
    wts, tok = eager.expert_choice_route(torch.randn(B, S, E, device="cuda"), -(-S // E))
    go = _rand(B, S, d)
    leaves = [t.clone().requires_grad_() for t in (x, *ws, wts)]
    out = ops.expert_choice_swiglu(*leaves, tok)
    got = (out, *torch.autograd.grad(out, leaves, go))
    cuda_ops.check_status()
    ref_leaves = [t.double().requires_grad_() for t in (x, *ws, wts)]
    ref = eager.expert_choice_swiglu(*ref_leaves, tok)
    want = (ref, *torch.autograd.grad(ref, ref_leaves, go.double()))
    for g, w in zip(got, want):
        assert _rel(g, w) < EXPERT_TOL


@pytest.mark.parametrize("B,S,d,V,chunk", [(1, 9, 64, 65, 8192), (2, 70, 128, 1001, 64), (2, 33, 64, 131, 8192)])
def test_loss_vocabulary(B, S, d, V, chunk):
    from kolmogorov_moe_architecture_b200.ops import cuda_ops, eager
    torch.manual_seed(V)
    h = _rand(B, S, d)
    Ws = [_rand(V, d, scale=0.1) for _ in range(3)]
    labels = torch.randint(0, V, (B, S), device="cuda")
    labels[:, ::7] = -100
    wts = (0.5, 0.3, 0.2)
    leaves = [t.clone().requires_grad_() for t in (h, *Ws)]
    total, _ = cuda_ops.mtp_cross_entropy(leaves[0], leaves[1:], labels, wts, chunk_rows=chunk)
    got = torch.autograd.grad(total, leaves)
    cuda_ops.check_status()
    ref_leaves = [t.double().requires_grad_() for t in (h, *Ws)]
    ref = 0.0
    for i, W in enumerate(ref_leaves[1:]):
        lg = ref_leaves[0][:, : S - i - 1] @ W.t()
        ref = ref + wts[i] * torch.nn.functional.cross_entropy(lg.reshape(-1, V), labels[:, i + 1:].reshape(-1), ignore_index=-100)
    want = torch.autograd.grad(ref, ref_leaves)
    # logits and their gradients are rounded to bf16, and dH / dW to bf16 once per head / row chunk
    assert abs(total.item() - ref.item()) < 2e-3 * abs(ref.item())
    for g, w in zip(got, want):
        assert _rel(g, w) < EXPERT_TOL


@pytest.mark.parametrize("M,N,G", [(1, 8, 1), (33, 72, 2), (130, 72, 3), (257, 264, 2), (300, 520, 2)])
@pytest.mark.parametrize("addends", [0, 1, 2])
def test_output_edges_stay_inside(M, N, G, addends):
    """Results leave by TMA stores of 32 x 64 blocks: nothing past column N, row M or between the groups is written."""
    from kolmogorov_moe_architecture_b200.ops import cuda_ops as c
    if addends == 2 and M <= 128:
        pytest.skip("the second addend exists in the CTA-pair kernel only")
    K, pitch = 96, N + 24
    a, b = _rand(G, M, K), _rand(G, N, K)
    D, D2 = _rand(G, M + 5, pitch), _rand(G, M + 5, pitch)
    out = torch.full((G, M + 5, pitch), 3.0, dtype=torch.bfloat16, device="cuda")
    kw = {}
    if addends:
        kw.update(D=D, beta=0.5, ldd=pitch)
    if addends == 2:
        kw.update(D2=D2, beta2=-1.5)
    c.gemm(a, b, out, mode=c.BATCHED, groups=G, M=M, N=N, Kd=K, lda=K, ldb=K, ldc=pitch, a_gs=M * K, b_gs=N * K,
           c_gs=(M + 5) * pitch, **kw)
    c.check_status()
    ref = torch.bmm(a.double(), b.double().transpose(1, 2))
    if addends:
        ref = ref + 0.5 * D[:, :M, :N].double()
    if addends == 2:
        ref = ref - 1.5 * D2[:, :M, :N].double()
    assert _rel(out[:, :M, :N], ref) < ONE_ROUNDING
    assert (out[:, M:] == 3.0).all() and (out[:, :, N:] == 3.0).all()


@pytest.mark.parametrize("R,V", [(3, 65), (5, 8), (7, 50257), (2, 114000), (2, 116000)])
@pytest.mark.parametrize("grad", [True, False])
def test_cross_entropy_rows(R, V, grad):
    """Rows that fit shared memory and rows that do not (from 115200 entries), with a tail, ignored and large entries."""
    from kolmogorov_moe_architecture_b200.ops import cuda_ops as c
    torch.manual_seed(V)
    pitch = -(-V // 64) * 64
    buf = torch.full((R, pitch), float("nan"), dtype=torch.bfloat16, device="cuda")
    buf[:, :V] = (torch.randn(R, V, device="cuda") * 3).to(torch.bfloat16)
    buf[0, V - 1] = 80.0
    lab = torch.randint(0, V, (R,), device="cuda")
    lab[1] = -100
    lg = buf[:, :V].double()
    ref = torch.nn.functional.cross_entropy(lg, lab, ignore_index=-100, reduction="none")
    p = (torch.softmax(lg, -1) - torch.nn.functional.one_hot(lab.clamp(min=0), V)) * 0.37
    p[1] = 0
    rows = c.K.ce_fwd_bwd(buf[:, :V], lab, torch.full((1,), 0.37, device="cuda"), -100, grad)
    assert (rows.double() - ref).abs().max() < 2e-5 * ref.abs().max()        # 32-bit sums
    if grad:
        assert _rel(buf[:, :V], p) < ONE_ROUNDING
    else:
        assert torch.equal(buf[:, :V].double(), lg)
    assert buf[:, V:].isnan().all()


@pytest.mark.parametrize("V", [32000, 50257, 131075])
def test_row_losses_have_no_bias(V):
    """The loss value: per row one rounding to fp32 (2^-21 at values of 8 to 16) plus the relative error of a 32-bit sum of
    exponentials, below 2^-21 together; both signs, so the mean over many rows stays below 2^-23."""
    from kolmogorov_moe_architecture_b200.ops import cuda_ops as c
    torch.manual_seed(V)
    R = 1024
    buf = torch.zeros(R, -(-V // 64) * 64, dtype=torch.bfloat16, device="cuda")
    buf[:, :V] = torch.randn(R, V, device="cuda").mul(0.8).bfloat16()
    lab = torch.randint(0, V, (R,), device="cuda")
    rows = c.K.ce_fwd_bwd(buf[:, :V], lab, torch.ones(1, device="cuda"), -100, False)
    err = rows.double() - torch.nn.functional.cross_entropy(buf[:, :V].double(), lab, reduction="none")
    assert err.abs().max() < 2.0 ** -20 and err.mean().abs() < 2.0 ** -23


@pytest.mark.parametrize("parts", [1, 2, 3])
def test_loss_vocabulary_slices(parts, monkeypatch):
    """The hidden states' gradient accumulated in vocabulary slices, several row chunks and heads."""
    from kolmogorov_moe_architecture_b200.ops import cuda_ops
    monkeypatch.setattr(cuda_ops, "_loss_split", lambda *a: parts)
    torch.manual_seed(parts)
    B, S, d, V = 2, 90, 128, 1003
    h = _rand(B, S, d)
    Ws = [_rand(V, d, scale=0.1) for _ in range(3)]
    labels = torch.randint(0, V, (B, S), device="cuda")
    leaves = [t.clone().requires_grad_() for t in (h, *Ws)]
    total, _ = cuda_ops.mtp_cross_entropy(leaves[0], leaves[1:], labels, (0.5, 0.3, 0.2), chunk_rows=64)
    got = torch.autograd.grad(total, leaves)
    cuda_ops.check_status()
    rl = [t.double().requires_grad_() for t in (h, *Ws)]
    ref = sum(w * torch.nn.functional.cross_entropy((rl[0][:, : S - i - 1] @ W.t()).reshape(-1, V), labels[:, i + 1:].reshape(-1))
              for i, (W, w) in enumerate(zip(rl[1:], (0.5, 0.3, 0.2))))
    for g, w in zip(got, torch.autograd.grad(ref, rl)):
        assert _rel(g, w) < EXPERT_TOL


@pytest.mark.parametrize("blocks,spare,d,f,swiglu", [
    ((8, 7, 6), 0, 256, 384, True),           # 21 blocks for 3 experts: the first count that takes CTA pairs
    ((14, 1, 0, 11), 2, 192, 328, True),      # one-block and empty experts, odd ends, spare blocks after the live ones
    ((33, 2, 94), 3, 128, 264, False),        # runs across the 32- and 128-block steps of the tile list
    ((0, 0), 16, 128, 256, False),            # nothing routed here
    ((500, 267), 1, 64, 64, False),           # the longest list
    ((500, 268), 1, 64, 64, False),           # one more: single CTAs
])
def test_expert_blocks_in_pairs(blocks, spare, d, f, swiglu):
    """256-row tiles over 128-row expert blocks: each expert's blocks in twos, an odd last one alone.  The products have
    one bf16 rounding on fp32 sums of at most 2 * 256 terms: |error| <= 2^-8 |y| + 512 * 2^-24 * sum |terms|; the SwiGLU
    value adds the rounding of nothing else (it is formed from the fp32 accumulators)."""
    from kolmogorov_moe_architecture_b200.ops import cuda_ops as c
    torch.manual_seed(5)
    E, live = len(blocks), sum(blocks)
    rows = (live + spare) * 128
    group = [e for e, n in enumerate(blocks) for _ in range(n)]
    tiles = torch.tensor(group + [0] * spare, dtype=torch.int32, device="cuda")
    nmt = torch.tensor([live], dtype=torch.int32, device="cuda")
    x = torch.randn(rows, d, device="cuda").bfloat16()
    x[live * 128:] = float("nan")                                    # never part of a live result
    w1, w2 = (torch.randn(E, d, f, device="cuda").mul(d ** -0.5).bfloat16() for _ in range(2))
    out = torch.full((rows, f), 7.0, dtype=torch.bfloat16, device="cuda")
    kw = dict(mode=c.GROUPED_M, M=rows, N=f, groups=E, b_major=c.MAJ_MN, ldb=f, ldc=f, b_gs=d * f, tile_group=tiles,
              num_m_tiles=nmt)
    if swiglu:
        c.gemm(x, w1, out, B2=w2, epi=c.EPI_SWIGLU, Kd=d, lda=d, **kw)
    else:
        xx = torch.cat([x, x], dim=1)                                # [x | x] [w1 ; w2] as one split reduction
        c.gemm(xx, w1, out, B2=w2, k_split=d, Kd=2 * d, lda=2 * d, **kw)
    c.check_status()
    assert bool((out[live * 128:] == 7.0).all())
    first = 0
    for e, n in enumerate(blocks):
        xs, o = x[first * 128:(first + n) * 128].double(), out[first * 128:(first + n) * 128].double()
        first += n
        g, u = xs @ w1[e].double(), xs @ w2[e].double()
        mag = xs.abs() @ w1[e].double().abs(), xs.abs() @ w2[e].double().abs()
        if swiglu:
            y = torch.nn.functional.silu(g) * u
            slack = 512 * 2.0 ** -24 * (1.1 * mag[0] * u.abs() + mag[1] * g.abs()) + 2.0 ** -20 * y.abs()   # fast exp
        else:
            y, slack = g + u, 512 * 2.0 ** -24 * (mag[0] + mag[1])
        assert bool(((o - y).abs() <= 2.0 ** -8 * y.abs() + slack + 1e-30).all())


@pytest.mark.parametrize("V", [1003, 1024])
def test_loss_without_gradients_makes_none(V):
    """An evaluation pass: per head the logits' product and the row kernel, and no gradient buffers."""
    from kolmogorov_moe_architecture_b200.ops import cuda_ops as c
    torch.manual_seed(V)
    h = _rand(2, 40, 128).requires_grad_()
    Ws = [torch.nn.Parameter(_rand(V, 128, scale=0.1)) for _ in range(3)]
    labels = torch.randint(0, V, (2, 40), device="cuda")

    def run():
        n = c.LAUNCHES["count"]
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        held = torch.cuda.memory_allocated()
        total, per = c.mtp_cross_entropy(h, Ws, labels, (0.5, 0.3, 0.2))
        return total, c.LAUNCHES["count"] - n, torch.cuda.max_memory_allocated() - held
    with torch.no_grad():
        run()
        total, launches, peak = run()
    assert launches == 6 and not total.requires_grad
    assert peak < 2 * 80 * (V + 64) * 2            # two logits buffers at most; the heads' dW alone are more than that
    with_grad, launches, _ = run()
    assert launches > 6 and torch.equal(with_grad.detach(), total)


def test_loss_memory_is_bounded_by_the_row_chunk(monkeypatch):
    """Beside the gradients themselves the loss holds one chunk's logits and fp32 accumulators, whatever the row count."""
    from kolmogorov_moe_architecture_b200.ops import cuda_ops as c
    monkeypatch.setattr(c, "_loss_split", lambda *a: 3)
    torch.manual_seed(0)
    B, S, d, V, chunk = 4, 4096, 256, 1003, 512
    h = _rand(B, S, d).requires_grad_()
    Ws = [_rand(V, d, scale=0.1).requires_grad_() for _ in range(2)]
    labels = torch.randint(0, V, (B, S), device="cuda")
    for _ in range(2):
        total = None
        torch.cuda.synchronize()
        held = torch.cuda.memory_allocated()
        torch.cuda.reset_peak_memory_stats()
        total, _ = c.mtp_cross_entropy(h, Ws, labels, (0.5, 0.5), chunk_rows=chunk)
        peak = torch.cuda.max_memory_allocated() - held
    results = 2 * B * S * d + 2 * 2 * V * d                          # dH and the dW
    small = 2 * 2 * chunk * (V + 64) + 4 * 3 * chunk * d             # two logits buffers, three slices of a chunk
    assert peak < results + small + 4 * 8 * B * S + (1 << 20)        # label copies


def _off(t):
    """The same values at an address that is a multiple of 2 bytes only."""
    buf = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    v = buf[1:].view(t.shape)
    v.copy_(t)
    assert v.data_ptr() % 4 == 2
    return v


@pytest.mark.parametrize("f", [72, 128])
@pytest.mark.parametrize("which", ["tokens", "experts"])
def test_expert_operands_off_the_16_byte_grid(which, f):
    """Inputs, weights and the incoming gradient as views that start anywhere: the same bits as aligned copies give."""
    from kolmogorov_moe_architecture_b200 import ops
    from kolmogorov_moe_architecture_b200.ops import eager
    torch.manual_seed(f)
    B, S, d, E, k = 1, 40, 64, 3, 2
    x, ws, go = _rand(B, S, d), _expert_case(E, d, f), _rand(B, S, d)
    if which == "tokens":
        wts, idx = eager.topk_softmax_route(torch.randn(S, E, device="cuda"), k)
        run = lambda x, *w: ops.grouped_swiglu(x.view(S, d), *w, idx, wts).view(B, S, d)
    else:
        wts, tok = eager.expert_choice_route(torch.randn(B, S, E, device="cuda"), 14)
        run = lambda x, *w: ops.expert_choice_swiglu(x, *w, wts, tok)

    def results(move):
        leaves = [move(t).requires_grad_() for t in (x, *ws)]
        out = run(*leaves)
        return (out, *torch.autograd.grad(out, leaves, move(go)))
    for a, b in zip(results(lambda t: t.clone()), results(_off)):
        assert torch.equal(a, b)


def test_loss_operands_off_the_16_byte_grid():
    from kolmogorov_moe_architecture_b200.ops import cuda_ops as c
    torch.manual_seed(0)
    h, W = _rand(2, 20, 64), _rand(131, 64, scale=0.1)
    labels = torch.randint(0, 131, (2, 20), device="cuda")

    def results(move):
        leaves = [move(t).requires_grad_() for t in (h, W)]
        total, _ = c.mtp_cross_entropy(leaves[0], [leaves[1]], labels, (1.0,))
        return (total, *torch.autograd.grad(total, leaves))
    for a, b in zip(results(lambda t: t.clone()), results(_off)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("which", ["loss", "tokens", "experts"])
def test_a_second_derivative_is_refused(which):
    """The kernels' gradients carry no graph.  A penalty on them raises instead of quietly leaving out its own gradient."""
    from kolmogorov_moe_architecture_b200 import ops
    from kolmogorov_moe_architecture_b200.ops import cuda_ops as c, eager
    torch.manual_seed(0)
    x = _rand(1, 24, 64).requires_grad_()
    if which == "loss":
        y, _ = c.mtp_cross_entropy(x, [_rand(131, 64, scale=0.1)], torch.randint(0, 131, (1, 24), device="cuda"), (1.0,))
    elif which == "tokens":
        wts, idx = eager.topk_softmax_route(torch.randn(24, 3, device="cuda"), 2)
        y = ops.grouped_swiglu(x.view(24, 64), *_expert_case(3, 64, 72), idx, wts).float().sum()
    else:
        wts, tok = eager.expert_choice_route(torch.randn(1, 24, 3, device="cuda"), 8)
        y = ops.expert_choice_swiglu(x, *_expert_case(3, 64, 72), wts, tok).float().sum()
    (g,) = torch.autograd.grad(y, x, create_graph=True)
    with pytest.raises(RuntimeError, match="no second derivative"):
        (x.float().square().sum() + g.float().square().sum()).backward()


@pytest.mark.parametrize("blocks,spare,d,f,P,split", [
    ((8, 7, 6), 0, 256, 384, 384, False),     # as dH: one reduction over K-major rows of the weight
    ((14, 1, 0, 11), 2, 328, 192, 192, False),
    ((8, 7, 6), 1, 192, 384, 384, True),      # as dX: [dG | dU] against two weights, widths of whole 64-element blocks
    ((7, 9, 5), 0, 192, 328, 384, True),      # the reduction of each weight ends inside a block, the operand's is padded
    ((2, 20), 3, 264, 72, 128, True),
])
def test_expert_blocks_in_pairs_k_major(blocks, spare, d, f, P, split):
    """The backward products of the pair schedule: weights [d, f] read along f.  Tolerances as in
    test_expert_blocks_in_pairs: one rounding to bf16 on fp32 sums of at most 2 * 384 terms."""
    from kolmogorov_moe_architecture_b200.ops import cuda_ops as c
    torch.manual_seed(6)
    E, live = len(blocks), sum(blocks)
    rows = (live + spare) * 128
    tiles = torch.tensor([e for e, n in enumerate(blocks) for _ in range(n)] + [0] * spare, dtype=torch.int32, device="cuda")
    nmt = torch.tensor([live], dtype=torch.int32, device="cuda")
    w1, w2 = (torch.randn(E, d, f, device="cuda").mul(f ** -0.5).bfloat16() for _ in range(2))
    parts = 2 if split else 1
    x = torch.zeros(rows, parts * P, device="cuda", dtype=torch.bfloat16)      # zeros between f and P, as the kernels pad
    for j in range(parts):
        x[:, j * P:j * P + f] = torch.randn(rows, f, device="cuda").bfloat16()
    x[live * 128:] = float("nan")
    out = torch.full((rows, d), 7.0, dtype=torch.bfloat16, device="cuda")
    kw = dict(B2=w2, k_split=P, b_klen=f) if split else {}
    c.gemm(x, w1, out, mode=c.GROUPED_M, M=rows, N=d, Kd=parts * P, groups=E, lda=parts * P, ldb=f, ldc=d, b_gs=d * f,
           tile_group=tiles, num_m_tiles=nmt, **kw)
    c.check_status()
    assert bool((out[live * 128:] == 7.0).all())
    first = 0
    for e, n in enumerate(blocks):
        xs, o = x[first * 128:(first + n) * 128].double(), out[first * 128:(first + n) * 128].double()
        first += n
        y, mag = 0.0, 0.0
        for j, w in enumerate((w1, w2)[:parts]):
            a, b = xs[:, j * P:j * P + f], w[e].double().t()
            y, mag = y + a @ b, mag + a.abs() @ b.abs()
        assert bool(((o - y).abs() <= 2.0 ** -8 * y.abs() + 768 * 2.0 ** -24 * mag + 1e-30).all())


@pytest.mark.parametrize("T,d,f,E,k", [(2000, 192, 328, 3, 2), (2700, 256, 384, 3, 1)])
def test_expert_layer_in_pairs(T, d, f, E, k):
    """Token choice with enough row blocks per expert that every grouped product of both passes runs on CTA pairs."""
    from kolmogorov_moe_architecture_b200 import ops
    from kolmogorov_moe_architecture_b200.ops import cuda_ops, eager
    assert cuda_ops.K.moe_plan(torch.zeros(T * k, dtype=torch.long, device="cuda"), None, E, 0)[1].numel() >= 7 * 128 * E
    torch.manual_seed(T)
    ws, x, go = _expert_case(E, d, f), _rand(T, d), _rand(T, d)
    wts, idx = eager.topk_softmax_route(torch.randn(T, E, device="cuda"), k)
    wts = wts.to(torch.bfloat16)
    leaves = [t.clone().requires_grad_() for t in (x, *ws, wts)]
    out = ops.grouped_swiglu(*leaves[:4], idx, leaves[4])
    got = (out, *torch.autograd.grad(out, leaves, go))
    cuda_ops.check_status()
    rl = [t.double().requires_grad_() for t in (x, *ws, wts)]
    ref = eager.grouped_swiglu(*rl[:4], idx, rl[4])
    for g, w in zip(got, (ref, *torch.autograd.grad(ref, rl, go.double()))):
        if w.norm() > 0:
            assert _rel(g, w) < EXPERT_TOL


@pytest.mark.parametrize("out_f", [24, 64])
def test_linear_gradient_off_the_16_byte_grid(out_f):
    from kolmogorov_moe_architecture_b200 import ops
    torch.manual_seed(out_f)
    x, w, go = _rand(40, 128), _rand(out_f, 128).requires_grad_(), _rand(40, out_f)
    y = ops.linear(x, w)
    (a,), (b,) = (torch.autograd.grad(y, w, g, retain_graph=True) for g in (go, _off(go)))
    assert torch.equal(a, b)
