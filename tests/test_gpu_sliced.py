"""The FP64 grouped GEMM on the tensor cores (digit slices) against FP64 matmul.

Bound per element: the reference's own K additions, 2 (K + 4) 2^-53 sum |a||b|, plus the
fixed-point resolution of the digits, K 2^-60 max|a| max|b| (rows and columns scaled by their
largest element)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture
def sliced(monkeypatch):
    """Every FP64 task goes to the sliced kernel."""
    from qodeapplications_gb300 import gemm
    monkeypatch.setattr(gemm, "SLICED_MIN_CHAIN", 0)
    monkeypatch.setattr(gemm, "SLICED_MIN_K", 1)
    return gemm


def _operand(g, batch, rows, K, trans, kind):
    x = torch.randn(batch, rows, K, generator=g, dtype=torch.float64)
    if kind == "wide":
        x *= 10.0 ** (-14.0 * torch.rand(batch, rows, K, generator=g, dtype=torch.float64))
    if kind == "sparse":
        x *= (torch.rand(batch, rows, K, generator=g) < 0.2)
    if kind == "tiny":
        x *= 1e-290
    if kind == "huge":
        x *= 1e150
    x = x.cuda()
    return (x.transpose(1, 2).contiguous() if trans else x), x


def _bound(a, b, alpha):
    K = a.shape[-1]
    mag = a.abs() @ b.abs().transpose(1, 2)
    top = a.abs().amax(2, keepdim=True) * b.abs().amax(2, keepdim=True).transpose(1, 2)
    return abs(alpha) * (2 * (K + 4) * 2.0 ** -53 * mag + K * 2.0 ** -60 * top)


@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (127, 63, 31), (128, 64, 32), (129, 65, 33), (128, 32, 128), (130, 33, 129),
                                   (60, 28, 1100), (5, 200, 4000)])
@pytest.mark.parametrize("flags,batch,mode,kind", [(0, 1, 0, "normal"), (1, 3, 1, "wide"), (2, 1, 1, "sparse"),
                                                   (3, 3, 0, "tiny"), (0, 2, 1, "huge")])
def test_shapes_layouts_and_ranges(sliced, M, N, K, flags, batch, mode, kind):
    g = torch.Generator().manual_seed(M * 1000 + N * 10 + K)
    C = torch.zeros(batch, M, N, dtype=torch.float64, device="cuda")
    segs, ref, tol = [], torch.zeros_like(C), torch.zeros_like(C)
    for k, alpha in ((K, 1.0), (7, -0.3)):
        A, a = _operand(g, batch, M, k, flags & 1, kind)
        B, b = _operand(g, 1, N, k, flags & 2, "normal")
        segs.append((A, A.shape[2], B, B.shape[2], k, alpha, flags, M * k, 0))
        ref += alpha * (a @ b.transpose(1, 2))
        tol += _bound(a, b, alpha)
    gg = sliced.GroupedGemm()
    gg.add(M, N, segs, C, N, mode=mode, batch=batch, sC=M * N)
    gg.finalize()
    assert gg.sliced is not None and gg.n_tasks == 0
    gg.run()
    gg.check()
    tol += 2.0 ** -52 * ref.abs() + 5e-324
    assert bool(((C - ref).abs() <= tol).all()), float(((C - ref).abs() / tol).max())


def test_mixed_tile_widths_scatter_and_panels(sliced, monkeypatch):
    """Many tiles of both widths per CTA, the scatter epilogue with its delta terms, and operands in
    several workspace waves."""
    from qodeapplications_gb300 import sliced as plan
    monkeypatch.setattr(plan, "WORKSPACE_LIMIT", 3 << 20)
    g = torch.Generator().manual_seed(5)
    gg = sliced.GroupedGemm()
    checks = []
    for batch, M, N, K in ((400, 18, 20, 18), (1, 300, 400, 100), (300, 20, 50, 40)):
        A, a = _operand(g, batch, M, K, False, "normal")
        B, b = _operand(g, 1, N, K, False, "normal")
        C = torch.zeros(batch, M, N, dtype=torch.float64, device="cuda")
        gg.add(M, N, [(A, K, B, K, K, 1.0, 0, M * K, 0)], C, N, mode=0, batch=batch, sC=M * N)
        checks.append((C, a @ b.transpose(1, 2), _bound(a, b, 1.0)))
    M, N, K = 200, 150, 90
    A, a = _operand(g, 1, M, K, False, "normal")
    B, b = _operand(g, 1, N, K, False, "normal")
    i32 = dict(dtype=torch.int32, device="cuda")
    perm = torch.randperm(M, generator=g).to(**i32)
    DA, DB = torch.randn(M, dtype=torch.float64).cuda(), torch.randn(N, dtype=torch.float64).cuda()
    dA, dB = torch.arange(M).cuda() % 3 == 0, torch.arange(N).cuda() % 4 == 0
    C = torch.full((M, N), 7.0, dtype=torch.float64, device="cuda")
    gg.add(M, N, [(A, K, B, K, K, 2.0)], C, N, mode=2,
           maps=(perm, torch.zeros(M, **i32), torch.zeros(N, **i32), torch.arange(N, **i32), dA.to(torch.uint8),
                 dB.to(torch.uint8)), DA=DA, DB=DB)
    ref = 2.0 * (a @ b.transpose(1, 2))[0] + DA[:, None] * dB[None, :] + DB[None, :] * dA[:, None]
    out = torch.empty_like(ref)
    out[perm.long()] = ref
    tol = torch.empty_like(ref)
    tol[perm.long()] = _bound(a, b, 2.0)[0] + 2.0 ** -51 * (ref.abs() + DA.abs()[:, None] + DB.abs()[None, :])
    checks.append((C, out, tol))
    gg.finalize()
    assert len(gg.sliced.waves) > 3
    for _ in range(2):                   # stored results: a second run gives the same
        gg.run()
    gg.check()
    for got, want, t in checks:
        assert bool(((got - want).abs() <= t + 2.0 ** -52 * want.abs()).all())


def test_infinities_and_nan_as_in_fp64(sliced):
    """Rows and columns with non-finite elements: finite, infinite and NaN results where FP64 has
    them; the other elements are untouched."""
    g = torch.Generator().manual_seed(6)
    M, N, K = 140, 70, 50
    A, B = (torch.randn(n, K, generator=g, dtype=torch.float64) for n in (M, N))
    A[3, 5], A[131, 0], B[66, 49] = float("inf"), float("nan"), -float("inf")
    A[:, 49] += 10.0
    B[10, 5] = 0.0                       # inf * 0
    A, B = A.cuda(), B.cuda()
    C = torch.zeros(M, N, dtype=torch.float64, device="cuda")
    gg = sliced.GroupedGemm()
    gg.add(M, N, [(A, K, B, K, K, -2.0)], C, N)
    gg.finalize().run()
    gg.check()
    want = -2.0 * (A @ B.t())
    assert torch.equal(C.isnan(), want.isnan()) and torch.equal(C.isinf(), want.isinf())
    assert torch.equal(C[C.isinf()], want[C.isinf()])
    ok = want.isfinite()
    assert bool(((C - want).abs()[ok] <= 1e-12).all())
