"""Layout passes of the three-index density blocks, and the split of operands stored transposed: copies
and sign changes (and one FP64 addition), so the results are equal, not close."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [1, 2, 7, 18, 28, 29, 30, 33, 41])
@pytest.mark.parametrize("nb,nk", [(1, 1), (3, 5), (4, 4), (5, 7)])
def test_expand_and_collect(N, nb, nk):
    from qodeapplications_gb300 import _lib
    g = torch.Generator().manual_seed(100 * N + nb)
    K, R = N ** 3, nb * nk
    rows = torch.randn(K, R, generator=g, dtype=torch.float64)
    p, q, r = (x.reshape(-1) for x in torch.meshgrid(*[torch.arange(N)] * 3, indexing="ij"))
    full = rows.clone()
    full[q > r] = -rows[((p * N + r) * N + q)[q > r]]
    for anti, want in ((False, rows), (True, full)):
        rho_ref = want.t().reshape(nb, nk, N, N, N)
        mir_ref = rho_ref.permute(1, 0, 4, 3, 2).contiguous()
        src = rows.clone()
        if anti:
            src[q > r] = float("nan")                  # not read
        src = src.cuda()
        for mirror in (False, True):
            rho = torch.full((nb, nk, N, N, N), float("nan"), dtype=torch.float64, device="cuda")
            mir = torch.full((nk, nb, N, N, N), float("nan"), dtype=torch.float64, device="cuda")
            _lib.DensityLayout([(src, rho, mir if mirror else None, nb, nk, anti)], N, "cuda").run()
            assert torch.equal(rho.cpu(), rho_ref)
            assert torch.equal(mir.cpu(), mir_ref) if mirror else bool(torch.isnan(mir).all())
    grho, gmir = (torch.randn(s + (N, N, N), generator=g, dtype=torch.float64) for s in ((nb, nk), (nk, nb)))
    for mirror in (False, True):
        out = torch.full((K, R), float("nan"), dtype=torch.float64, device="cuda")
        _lib.DensityLayout([(out, grho.cuda(), gmir.cuda() if mirror else None, nb, nk, False)], N, "cuda", collect=True).run()
        ref = grho + gmir.permute(1, 0, 4, 3, 2) if mirror else grho
        assert torch.equal(out.cpu(), ref.reshape(R, K).t())


def test_expand_blocks_of_one_launch():
    """Blocks of different state counts share a launch; a mirrored block may be missing."""
    from qodeapplications_gb300 import _lib
    N, items, refs = 6, [], []
    for nb, nk, mirror in ((2, 3, True), (17, 1, False), (4, 9, True)):
        rows = torch.randn(N ** 3, nb * nk, dtype=torch.float64)
        rho = torch.empty((nb, nk, N, N, N), dtype=torch.float64, device="cuda")
        mir = torch.empty((nk, nb, N, N, N), dtype=torch.float64, device="cuda") if mirror else None
        items.append((rows.cuda(), rho, mir, nb, nk, False))
        refs.append(rows.t().reshape(nb, nk, N, N, N))
    _lib.DensityLayout(items, N, "cuda").run()
    for (_r, rho, mir, _nb, _nk, _a), ref in zip(items, refs):
        assert torch.equal(rho.cpu(), ref)
        assert mir is None or torch.equal(mir.cpu(), ref.permute(1, 0, 4, 3, 2))


@pytest.mark.parametrize("precision", ["tf32x3", "bf16x3"])
@pytest.mark.parametrize("rows,K,ld", [(1, 1, 1), (31, 63, 40), (32, 64, 32), (33, 65, 33), (100, 200, 128)])
def test_split_of_transposed_operands(precision, rows, K, ld):
    from qodeapplications_gb300.gemm import SplitRegistry, Transposed
    g = torch.Generator().manual_seed(rows + K)
    x = (torch.randn(K, ld, generator=g, dtype=torch.float64) * 10.0 ** torch.randint(-30, 30, (K, ld), generator=g)).cuda()
    y = x[:, :rows].t().contiguous()
    reg = SplitRegistry(precision, "cuda")
    a, b = reg.operand(Transposed(x), rows, K, ld, "x"), reg.operand(y, rows, K, K, "x")
    for op in (a, b):
        op["hi"].fill_(7), op["lo"].fill_(7)
    reg.split("x")
    assert torch.equal(a["hi"], b["hi"]) and torch.equal(a["lo"], b["lo"])
    other = torch.zeros((K + 1, ld + 1), dtype=torch.float64, device="cuda")
    with pytest.raises(ValueError):                    # rows apart in memory
        reg.operand(Transposed(other[:, :ld]), rows, K + 1, ld, "x")
