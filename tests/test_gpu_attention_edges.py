"""Attention at the sizes where its schedules change: partial and single blocks, head groups that one CTA, two or four CTAs
of a cluster share in the backward pass, documents that end inside a block; both head widths."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# P, dS and the results are rounded to bf16 (about 1.7e-3 each in the 2-norm), sums are in 32 bits: three roundings in
# quadrature, and a quarter of the exponentials carries 1e-4.
TOL = 6e-3


def _ref(q, k, v, doc_start):
    from kolmogorov_moe_architecture_b200.ops import eager
    B, S, H, D = q.shape
    g = H // k.shape[2]
    kh, vh = k.repeat_interleave(g, dim=2), v.repeat_interleave(g, dim=2)
    s = torch.einsum("bqhd,bkhd->bhqk", q, kh) / D ** 0.5
    s = s.masked_fill(torch.triu(torch.ones(S, S, dtype=torch.bool, device=q.device), 1), float("-inf"))
    if doc_start is not None:
        s = s + eager.doc_start_to_mask(doc_start, s.dtype)
    return torch.einsum("bhqk,bkhd->bqhd", torch.softmax(s, -1), vh)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,S,H,Hkv,docs", [
    (1, 1, 2, 2, 0), (1, 33, 4, 1, 0), (2, 128, 6, 3, 0), (1, 129, 8, 2, 3), (2, 257, 14, 2, 0), (1, 640, 12, 3, 5),
    (3, 511, 4, 4, 2), (8, 900, 16, 4, 4), (1, 1500, 8, 1, 0)])
def test_blocks_groups_documents(B, S, H, Hkv, docs, D):
    from kolmogorov_moe_architecture_b200 import ops
    from kolmogorov_moe_architecture_b200.ops import cuda_ops, eager
    torch.manual_seed(S + H)
    mk = lambda n: torch.randn(B, S, n, D, device="cuda").to(torch.bfloat16)
    q, k, v, go = mk(H), mk(Hkv), mk(Hkv), mk(H)
    ds = None
    if docs:
        ids = torch.sort(torch.randint(0, docs, (B, S), device="cuda"), dim=1).values
        ds = eager.doc_start_from_ids(ids)
    leaves = [t.clone().requires_grad_() for t in (q, k, v)]
    out = ops.attention(*leaves, doc_start=ds)
    got = (out, *torch.autograd.grad(out, leaves, go))
    again = torch.autograd.grad(ops.attention(*leaves, doc_start=ds), leaves, go)
    cuda_ops.check_status()
    rl = [t.double().requires_grad_() for t in (q, k, v)]
    ref = _ref(*rl, ds)
    want = (ref, *torch.autograd.grad(ref, rl, go.double()))
    for g, w in zip(got, want):
        scale = w.norm().item()
        assert (g.double() - w).norm().item() <= TOL * max(scale, 1e-3 * w.numel() ** 0.5)
    for g, h in zip(got[1:], again):
        assert torch.equal(g, h)                       # fixed order of every sum


@pytest.mark.parametrize("B,S,H,Hkv,docs", [
    (1, 1, 1, 1, 0), (1, 1152, 16, 4, 0), (1, 1200, 16, 4, 3), (1, 1281, 18, 6, 0),   # one wave of single tiles and beyond it
    (8, 300, 16, 4, 0), (3, 700, 16, 4, 4), (25, 640, 2, 1, 0)])                   # pairs, an odd last tile
@pytest.mark.parametrize("D", [64, 128])
def test_query_tiles_per_cta(B, S, H, Hkv, docs, D):
    from kolmogorov_moe_architecture_b200 import ops
    from kolmogorov_moe_architecture_b200.ops import cuda_ops, eager
    torch.manual_seed(S)
    q, k, v = (torch.randn(B, S, n, D, device="cuda").to(torch.bfloat16) for n in (H, Hkv, Hkv))
    ds = None
    if docs:
        ds = eager.doc_start_from_ids(torch.sort(torch.randint(0, docs, (B, S), device="cuda"), dim=1).values)
    out = ops.attention(q, k, v, doc_start=ds)
    cuda_ops.check_status()
    ref = _ref(q.float(), k.float(), v.float(), ds)
    assert ((out.float() - ref).norm() / ref.norm()).item() < TOL


@pytest.mark.parametrize("S,H", [(256, 2), (1021, 4)])
def test_row_sums_of_64_wide_heads_are_32_bit(S, H):
    """The saved log-sum-exp: scores of 64 bf16 products each summed in fp32 (below 64 * 2^-24 * 8 for scores below 8) and
    exponentials within 2^-21, the sum in fp32 - 2^-15 covers all of it ten times over; the mean is ten times closer."""
    from kolmogorov_moe_architecture_b200.ops import cuda_ops as c
    torch.manual_seed(S)
    q, k, v = (torch.randn(1, S, H, 64, device="cuda").bfloat16() for _ in range(3))
    _, lse = c.K.attn_fwd(q, k, v, 0.125, None, c.status_tensor(q.device))
    s = torch.einsum("bqhd,bkhd->bhqk", q.double(), k.double()) * 0.125
    s = s.masked_fill(torch.triu(torch.ones(S, S, dtype=torch.bool, device="cuda"), 1), float("-inf"))
    err = lse.double() - torch.logsumexp(s, -1)
    assert err.abs().max() < 2.0 ** -15 and err.mean().abs() < 2.0 ** -18
