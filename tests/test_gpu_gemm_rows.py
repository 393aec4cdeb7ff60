"""Products whose rows go to individual addresses (the expert-parallel return), here all on one GPU."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(1, 64, 64), (130, 200, 72), (300, 264, 200), (257, 1032, 64)])
@pytest.mark.parametrize("addend", [False, True])
def test_rows_at_addresses(M, N, K, addend):
    """Rows in another order, every seventh skipped, columns beside them and rows without a sender untouched; tiles that end
    early in both directions, with and without an addend."""
    from kolmogorov_moe_architecture_b200.ops import cuda_ops as c
    torch.manual_seed(M)
    a, b, d = (torch.randn(*s, device="cuda").bfloat16() for s in ((M, K), (N, K), (M, N)))
    out = torch.full((M + 3, N + 8), 7.0, dtype=torch.bfloat16, device="cuda")
    to = torch.randperm(M + 3, device="cuda")[:M]
    keep = torch.arange(M, device="cuda") % 7 != 3
    addr = torch.where(keep, out.data_ptr() + to * out.stride(0) * 2, 0)
    kw = dict(D=d, beta=0.5, ldd=N) if addend else {}
    c.gemm(a, b, torch.empty(0, dtype=torch.bfloat16, device="cuda"), M=M, N=N, Kd=K, lda=K, ldb=K, ldc=N, row_ptr=addr, **kw)
    c.check_status()
    want = a.double() @ b.double().t() + (0.5 * d.double() if addend else 0.0)
    # exact products, sums of K + 1 values in 32 bits, one rounding to bf16
    size = a.double().abs() @ b.double().abs().t() + (0.5 * d.double().abs() if addend else 0.0)
    bound = 2.0 ** -8 * want.abs() + 1.01 * (K + 1) * 2.0 ** -23 * size
    assert ((out[to, :N].double() - want).abs() <= bound)[keep].all()
    untouched = torch.ones_like(out, dtype=torch.bool)
    untouched[to[keep], :N] = False
    assert (out[untouched] == 7.0).all()
