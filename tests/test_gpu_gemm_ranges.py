"""Schedules read from the device: batched products over many reduction ranges (more groups than the table in shared memory
holds, empty ones among them), row blocks of groups of which few or none are live; reductions on either side of the lengths
where the epilogue changes its number of warps."""
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


@pytest.mark.parametrize("groups", [2, 16])                   # on CTA pairs, on single CTAs
@pytest.mark.parametrize("live", [0, 1, 3])
def test_most_ctas_have_no_tile(groups, live):
    """The grid follows from the padded row count, the tiles from the live one.  Many launches: a CTA without a tile ends
    while its neighbours still work."""
    from kolmogorov_moe_architecture_b200.ops import cuda_ops as c
    torch.manual_seed(live)
    M, N, K = 2048, 1024, 128
    a, b = torch.randn(M, K, device="cuda").bfloat16(), torch.randn(groups, N, K, device="cuda").bfloat16()
    owner = (torch.arange(M // 128, device="cuda") * groups // (M // 128)).int()
    n = torch.tensor([live], dtype=torch.int32, device="cuda")
    out = torch.full((M, N), 7.0, dtype=torch.bfloat16, device="cuda")
    for _ in range(200):
        c.gemm(a, b, out, mode=c.GROUPED_M, groups=groups, M=M, N=N, Kd=K, lda=K, ldb=K, ldc=N, b_gs=N * K, tile_group=owner,
               num_m_tiles=n)
    c.check_status()
    for t in range(live):
        x, y = a[t * 128:(t + 1) * 128].double(), b[int(owner[t])].double()
        bound = 2.0 ** -8 * (x @ y.t()).abs() + 1.01 * K * 2.0 ** -23 * (x.abs() @ y.abs().t())    # exact products, one rounding
        assert ((out[t * 128:(t + 1) * 128].double() - x @ y.t()).abs() <= bound).all()
    assert (out[live * 128:] == 7.0).all()


@pytest.mark.parametrize("form,K", [("plain", 8), ("plain", 384), ("plain", 392), ("addend", 2048), ("addend", 2056),
                                    ("fp32", 128), ("swiglu", 512), ("swiglu", 520)])
@pytest.mark.parametrize("M,N", [(2600, 2072), (300, 136)])   # more tiles than pairs, one round
def test_epilogue_warps(form, K, M, N):
    from kolmogorov_moe_architecture_b200.ops import cuda_ops as c
    torch.manual_seed(K)
    a, b, b2 = (torch.randn(r, K, device="cuda").bfloat16() for r in (M, N, N))
    x, y = a.double(), b.double()
    if form == "swiglu":
        h, g, u = (torch.empty(M, N, dtype=torch.bfloat16, device="cuda") for _ in range(3))
        b, b2 = b / 8, b2 / 8
        c.gemm(a, b, h, B2=b2, G=g, U=u, epi=c.EPI_SWIGLU, M=M, N=N, Kd=K, lda=K, ldb=K, ldc=N)
        c.check_status()
        gate, up = x @ b.double().t(), x @ b2.double().t()
        for got, want in ((g, gate), (u, up), (h, torch.nn.functional.silu(gate) * up)):
            assert (got.double() - want).norm() <= 2.0 ** -8 * want.norm()      # one rounding to 8 bits
        return
    d = torch.randn(M, N, device="cuda").bfloat16() if form == "addend" else None
    out = c.mm_nt(a, b, out_dtype=torch.float32 if form == "fp32" else None, D=d, beta=0.5)
    c.check_status()
    more = 0.0 if d is None else 0.5 * d.double()
    want = x @ y.t() + more
    # exact products, sums of K + 1 values in 32 bits, one rounding of bf16 results
    bound = 1.01 * (K + 1) * 2.0 ** -23 * (x.abs() @ y.abs().t() + (more if d is None else more.abs()))
    bound += 0.0 if form == "fp32" else 2.0 ** -8 * want.abs()
    assert ((out.double() - want).abs() <= bound).all()
