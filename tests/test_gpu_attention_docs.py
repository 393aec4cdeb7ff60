"""Packed documents whose ends fall on, just before and just behind the borders of 128-row blocks, and documents of one token:
every query sees its own document up to itself, forward and backward."""
import pytest
import torch

pytestmark = pytest.mark.gpu

TOL = 6e-3      # three bf16 roundings in quadrature, as in the other attention tests


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("S,starts", [
    (256, (0, 127)), (256, (0, 128)), (257, (0, 129, 256)), (513, (0, 1, 2, 255, 256, 511)), (400, (0, 384)),
    (700, (0, 64, 65, 300, 640, 699)), (129, tuple(range(129)))])
def test_documents_at_block_borders(S, starts, D):
    from kolmogorov_moe_architecture_b200 import ops
    from kolmogorov_moe_architecture_b200.ops import cuda_ops
    torch.manual_seed(S + D)
    B, H, Hkv = 2, 4, 2
    ds = torch.zeros(B, S, dtype=torch.int32, device="cuda")
    for s in starts:
        ds[0, s:] = s                                   # the second sequence is one document
    mk = lambda n: torch.randn(B, S, n, D, device="cuda").to(torch.bfloat16)
    leaves, go = [mk(n).requires_grad_() for n in (H, Hkv, Hkv)], mk(H)
    out = ops.attention(*leaves, doc_start=ds)
    got = (out, *torch.autograd.grad(out, leaves, go))
    cuda_ops.check_status()
    q, k, v = (t.detach().double().requires_grad_() for t in leaves)
    pos = torch.arange(S, device="cuda")
    hidden = (pos[None, None, :] > pos[None, :, None]) | (pos[None, None, :] < ds.long()[:, :, None])
    s = torch.einsum("bqhd,bkhd->bhqk", q, k.repeat_interleave(2, 2)) / D ** 0.5
    p = torch.softmax(s.masked_fill(hidden[:, None], float("-inf")), -1)
    ref = torch.einsum("bhqk,bkhd->bqhd", p, v.repeat_interleave(2, 2))
    for g, w in zip(got, (ref, *torch.autograd.grad(ref, (q, k, v), go.double()))):
        assert (g.double() - w).norm().item() <= TOL * max(w.norm().item(), 1e-3 * w.numel() ** 0.5)
