"""Stores of the split-precision GEMM: whole tiles, ragged ones, odd row strides and bases, columns that
are not neighbours in memory, every N tile and mode."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _bound(a, b, K):
    # operands to 2^-22 of each element (hi + lo TF32), FP32 sums of chunks of 32 products: K / 32 + 12 roundings
    return (K / 32 + 16) * 2.0 ** -22 * (a.abs() @ b.abs().t())


@pytest.mark.parametrize("M,N,K", [(128, 128, 32), (256, 384, 70), (129, 127, 33), (60, 33, 28), (130, 64, 64), (3, 31, 200)])
@pytest.mark.parametrize("bn", [128, 32])
@pytest.mark.parametrize("ldc_extra,base", [(0, 0), (1, 0), (2, 1)])
@pytest.mark.parametrize("mode", [0, 1])
def test_plain_stores(M, N, K, bn, ldc_extra, base, mode):
    from qodeapplications_gb300.gemm import SplitRegistry, TCGroupedGemm
    g = torch.Generator().manual_seed(M + N + K)
    a, b = (torch.randn(r, K, generator=g, dtype=torch.float64).cuda() for r in (M, N))
    ldc = N + ldc_extra
    C = torch.full((base + M * ldc + 8,), 0.5, dtype=torch.float64, device="cuda")
    reg = SplitRegistry("tf32x3", "cuda")
    gg = TCGroupedGemm(reg)
    gg.add(M, N, [(a, K, b, K, K, -1.0)], C[base:], ldc, mode=mode)
    reg.upload()
    gg.finalize((bn, 16))
    reg.split("in")
    gg.run()
    gg.check()
    view = C[base:base + M * ldc].view(M, ldc)
    ref = -(a @ b.t()) + (0.5 if mode == 1 else 0.0)
    assert bool(((view[:, :N] - ref).abs() <= _bound(a, b, K)).all())
    assert bool((view[:, N:] == 0.5).all()) and bool((C[:base] == 0.5).all()) and bool((C[base + M * ldc:] == 0.5).all())


@pytest.mark.parametrize("ni,nj", [(3, 10), (5, 13), (16, 16)])
@pytest.mark.parametrize("shuffled", [False, True])
def test_scattered_stores(ni, nj, shuffled):
    from qodeapplications_gb300.gemm import SplitRegistry, TCGroupedGemm
    g = torch.Generator().manual_seed(ni * nj)
    n, K = ni * nj, 90                                 # (I, J) pairs on either side
    a, b = (torch.randn(n, K, generator=g, dtype=torch.float64).cuda() for _ in range(2))
    order = torch.randperm(n, generator=g) if shuffled else torch.arange(n)
    i, j = order // nj, order % nj
    i32 = lambda x: x.to(torch.int32).cuda()
    dim = (ni * ni, nj * nj)
    maps = (i32(i * ni), i32(j * nj), i32(i), i32(j), (i == j).to(torch.uint8).cuda(), (i == j).to(torch.uint8).cuda())
    DA, DB = (torch.randn(n, generator=g, dtype=torch.float64).cuda() for _ in range(2))
    H = torch.zeros(dim, dtype=torch.float64, device="cuda")
    reg = SplitRegistry("tf32x3", "cuda")
    gg = TCGroupedGemm(reg)
    gg.add(n, n, [(a, K, b, K, K, 1.0)], H, dim[1], mode=2, maps=maps, DA=DA, DB=DB)
    reg.upload()
    gg.finalize()
    reg.split("in")
    gg.run()
    gg.check()
    diag = maps[4].bool()
    x = a @ b.t() + torch.where(diag[None, :], DA[:, None], 0.0) + torch.where(diag[:, None], DB[None, :], 0.0)
    rows = (maps[0].long()[:, None] + maps[2].long()[None, :]), (maps[1].long()[:, None] + maps[3].long()[None, :])
    assert bool(((H[rows] - x).abs() <= _bound(a, b, K) + 2.0 ** -50 * x.abs()).all())
