"""Batched products over many reduction ranges: more groups than the table in shared memory holds, empty ones among them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("groups", [1, 127, 128, 131])
@pytest.mark.parametrize("m,n", [(128, 192), (264, 520)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_many_ranges(groups, m, n, dtype):
    from kolmogorov_moe_architecture_b200.ops import cuda_ops as c
    torch.manual_seed(groups)
    blocks = [(3 * g) % 4 for g in range(groups)]              # 0 to 3 blocks of 64 rows
    blocks[-1] = 2
    kl = torch.tensor(blocks, dtype=torch.int32) * 64
    kb = kl.cumsum(0) - kl
    rows = int(kl.sum())
    X = torch.randn(rows, m, device="cuda").bfloat16()
    Y = torch.randn(rows, n, device="cuda").bfloat16()
    out = torch.full((groups, m, n), 7.0, dtype=dtype, device="cuda")
    c.gemm(X, Y, out, mode=c.BATCHED, groups=groups, a_major=c.MAJ_MN, b_major=c.MAJ_MN, M=m, N=n, Kd=rows, lda=m, ldb=n,
           ldc=n, c_gs=m * n, k_begin=kb.int().cuda(), k_len=kl.cuda())
    c.check_status()
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 0.0        # one rounding of the result
    for g, (s, l) in enumerate(zip(kb.tolist(), kl.tolist())):
        x, y = X[s:s + l].double(), Y[s:s + l].double()
        # products of bf16 are exact in 32 bits; a sum of l of them is off by at most l * 2^-23 of the sum of their sizes
        bound = eps * (x.t() @ y).abs() + (1 + eps) * l * 2.0 ** -23 * (x.abs().t() @ y.abs())
        assert ((out[g].double() - x.t() @ y).abs() <= bound).all(), (g, l)
