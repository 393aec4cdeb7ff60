"""Selective scan where its schedule changes: one and several segments, chunks and channel blocks that end early, B and C as
column slices of a projection (bf16) and as fp32, with and without gate, bias and skip."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# Results and activation gradients are rounded to bf16 once (1.7e-3 in the 2-norm); ex2.approx and the 32-bit sums add less.
TOL = 4e-3


def _rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm().clamp(min=1e-30)).item()


def _ref(u, dt, A, Bm, Cm, D, z, bias, softplus):
    d = dt if bias is None else dt + bias
    d = torch.nn.functional.softplus(d) if softplus else d
    h = torch.zeros(u.shape[0], u.shape[2], 16, dtype=u.dtype, device=u.device)
    ys = []
    for t in range(u.shape[1]):
        h = torch.exp(d[:, t, :, None] * A) * h + (d[:, t] * u[:, t])[..., None] * Bm[:, t, None, :]
        ys.append((h * Cm[:, t, None, :]).sum(-1))
    y = torch.stack(ys, 1)
    y = y if D is None else y + u * D
    return y if z is None else y * torch.nn.functional.silu(z)


@pytest.mark.parametrize("B,S,C,form,gate", [
    (1, 1, 8, "slice", True), (2, 7, 72, "float", True), (1, 8, 64, "slice", False), (3, 9, 136, "slice", True),
    (1, 65, 200, "slice", True), (1, 333, 1536, "slice", True), (2, 517, 64, "float", False), (4, 130, 4096, "slice", True),
    (1, 333, 72, "slice", True), (2, 517, 200, "float", False), (1, 130, 8, "slice", True)])
def test_segments_chunks_layouts(B, S, C, form, gate):
    from kolmogorov_moe_architecture_b200 import ops
    torch.manual_seed(S + C)
    bf = lambda *s: torch.randn(*s, device="cuda").to(torch.bfloat16)
    u, dt, xz = bf(B, S, C), bf(B, S, C) * 0.5, bf(B, S, 2 * C)
    proj = bf(B, S, 24 + 32)
    Bm, Cm = proj[..., 24:40], proj[..., 40:]
    if form == "float":
        Bm, Cm = Bm.float(), Cm.float()
    A = -torch.exp(torch.randn(C, 16, device="cuda") * 0.5)
    D = torch.randn(C, device="cuda") if gate else None
    bias = torch.randn(C, device="cuda") if gate else None
    z = xz[..., C:] if gate else None
    dt = dt if gate else dt.abs()
    go = bf(B, S, C)
    args = [u, dt, A, Bm, Cm, D, z, bias]
    on = [t for t in args if t is not None]
    for t in on:
        t.requires_grad_(True)
    y = ops.selective_scan(*args, gate)
    got = (y, *torch.autograd.grad(y, on, go))
    with torch.no_grad():
        assert torch.equal(ops.selective_scan(*args, gate), y)
    ref_args = [None if t is None else t.detach().double().requires_grad_(True) for t in args]
    yr = _ref(*ref_args, gate)
    want = (yr, *torch.autograd.grad(yr, [t for t in ref_args if t is not None], go.double()))
    for g, w in zip(got, want):
        assert _rel(g, w) < TOL


@pytest.mark.parametrize("B,S,C", [(1, 333, 72), (2, 517, 200), (1, 130, 8)])
def test_half_filled_channel_blocks_in_segments(B, S, C):
    """What the sizes above with C % 16 == 8 are for: their last channel block is half empty and there are several segments."""
    from kolmogorov_moe_architecture_b200.ops import cuda_ops as c
    u, bc = torch.ones(B, S, C, dtype=torch.bfloat16, device="cuda"), torch.ones(B, S, 16, dtype=torch.bfloat16, device="cuda")
    seg = c.K.scan_fwd(u, u, None, -torch.ones(C, 16, device="cuda"), bc, bc, None, None, True, False)[2]
    assert C % 16 == 8 and seg.numel() >= 2 * B * 17 * C


@pytest.mark.parametrize("B,S,C", [(1, 0, 64), (1, 0, 8), (0, 5, 64)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_nothing_to_scan(B, S, C, dtype):
    """An empty sequence or batch: an empty result, empty or zero gradients, no kernel."""
    from kolmogorov_moe_architecture_b200 import ops
    mk = lambda *s, t=torch.bfloat16: torch.ones(*s, dtype=t, device="cuda").requires_grad_(True)
    args = [mk(B, S, C), mk(B, S, C), mk(C, 16, t=torch.float32), mk(B, S, 16, t=dtype), mk(B, S, 16, t=dtype),
            mk(C, t=torch.float32), mk(B, S, C), mk(C, t=torch.float32)]
    y = ops.selective_scan(*args)
    assert y.shape == (B, S, C)
    for g, t in zip(torch.autograd.grad(y, args, torch.ones_like(y)), args):
        assert g.shape == t.shape and not g.any()


def test_backward_takes_its_own_checkpoints_only():
    """Checkpoints are whole 16-channel blocks; those of a pass without gradients (none) or of the bare channels are refused by
    the single op and by the mixer."""
    from kolmogorov_moe_architecture_b200.ops import cuda_ops as c
    K, st = c.K, c.status_tensor(torch.device("cuda", torch.cuda.current_device()))
    B, S, C, R = 1, 24, 72, 8
    mk = lambda *s: torch.ones(*s, dtype=torch.bfloat16, device="cuda")
    u, A, bc = mk(B, S, C), -torch.ones(C, 16, device="cuda"), mk(B, S, 16)
    _, ckpt, seg = K.scan_fwd(u, u, None, A, bc, bc, None, None, True, True)
    assert ckpt.numel() == 3 * 80 * 16 and seg.numel() == 0
    scan = lambda ck: K.scan_bwd(u, u, None, A, bc, bc, None, None, u, ck, seg, True)
    W = 64                                    # the mixer's width
    p = [mk(W, 4), mk(W), mk(R + 32, W), mk(W, R), mk(W), mk(W, 16), mk(W)]
    xz = mk(B, S, 2 * W)
    y, x, x_dbl, delta, params, ckpt2, seg2 = K.mamba_inner_fwd(xz, *p, True, st)
    mixer = lambda ck: K.mamba_inner_bwd(y, xz, x, x_dbl, delta, params, ck, seg2, p[2], p[3], True, False, None, None, None,
                                         False, None, None, None, st)
    for bwd, own in ((scan, ckpt), (mixer, ckpt2)):
        bwd(own)
        for other in (own[:0], own[:-3 * 8 * 16], own.double()):
            with pytest.raises(RuntimeError, match="ckpt|checkpoints"):
                bwd(other)
    c.check_status()


def test_no_checkpoints_without_gradients():
    """Under no_grad the state before every chunk (16 fp32 values per channel and 8 steps, four times the output) is not kept."""
    from kolmogorov_moe_architecture_b200 import ops
    torch.manual_seed(0)
    B, S, C = 2, 512, 1024
    mk = lambda *s: torch.randn(*s, device="cuda").to(torch.bfloat16)
    u, dt, z, Bm, Cm = mk(B, S, C), mk(B, S, C), mk(B, S, C), mk(B, S, 16), mk(B, S, 16)
    A = torch.nn.Parameter(-torch.rand(C, 16, device="cuda") - 0.5)
    D, bias = (torch.nn.Parameter(torch.randn(C, device="cuda")) for _ in range(2))
    peaks = []
    for enabled in (False, True):
        with torch.set_grad_enabled(enabled):
            for _ in range(2):
                out = None
                torch.cuda.synchronize()
                held = torch.cuda.memory_allocated()
                torch.cuda.reset_peak_memory_stats()
                out = ops.selective_scan(u, dt, A, Bm, Cm, D, z, bias)
                peak = torch.cuda.max_memory_allocated() - held
        peaks.append((peak, out.detach().clone()))
    checkpoints = 4 * B * (S // 8) * C * 16
    assert torch.equal(peaks[0][1], peaks[1][1])
    assert peaks[0][0] < peaks[1][0] - checkpoints // 2
