"""FP64 products of rows whose elements differ by many orders of magnitude: every element of the grouped
GEMM keeps the bound of an FP64 sum, (K + 4) 2^-53 sum |a||b|, also where that is far below the
product of the largest elements of its row and column.  The reference is an extended-precision sum."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _graded(rng, rows, K, kind, side):
    x = rng.standard_normal((rows, K))
    k = np.arange(K) / max(K - 1, 1)
    if kind == "random":                              # every element of its own size
        x *= 10.0 ** rng.uniform(-16, 0, (rows, K))
    elif kind == "opposed":                           # large elements meet small ones only
        x *= 10.0 ** (-24.0 * (k if side == 0 else 1.0 - k))
    elif kind == "masked":                            # the largest elements meet zeros
        x *= np.where(k < 0.5, 1.0 if side == 0 else 0.0, 1e-11)
    elif kind == "rows":                              # some rows flat, some not
        x *= np.where((np.arange(rows) % 3 == 0)[:, None], 10.0 ** rng.uniform(-12, 0, (rows, K)), 1.0)
    elif kind == "subnormal":
        x *= (10.0 ** (-24.0 * k) * 1e-300 if side == 0 else 1e200)
    return x


def _reference(a, b):
    a, b = a.astype(np.longdouble), b.astype(np.longdouble)
    return a @ b.T, np.abs(a) @ np.abs(b).T


def _run(monkeypatch, M, N, segs, mode, splitk):
    from qodeapplications_gb300 import gemm
    monkeypatch.setattr(gemm, "SLICED_MIN_CHAIN", 0)
    monkeypatch.setattr(gemm, "SLICED_MIN_K", 1)
    C = torch.zeros(M, N, dtype=torch.float64, device="cuda")
    g = gemm.GroupedGemm()
    g.add(M, N, segs, C, N, mode=mode, splitk=splitk)
    g.finalize()
    assert g.sliced is not None and g.n_tasks == 0
    g.run()
    g.check()
    return C.cpu().numpy()


# tiles of both widths with ragged edges; K inside one stage, several groups, and (split) several tiles
@pytest.mark.parametrize("M,N,K,mode", [(1, 1, 2, 0), (130, 33, 31, 0), (129, 65, 300, 0), (40, 20, 1300, 1)])
@pytest.mark.parametrize("flags", [0, 3])
@pytest.mark.parametrize("kind", ["random", "opposed", "masked", "rows", "subnormal"])
def test_error_relative_to_the_products(monkeypatch, M, N, K, mode, flags, kind):
    rng = np.random.default_rng(M + N + K)
    alpha = (1.0, -0.375)                             # (exact factors)
    segs, ref, mag = [], 0, 0
    for k, al in zip((K, 9), alpha):
        a, b = _graded(rng, M, k, kind, 0), _graded(rng, N, k, kind, 1)
        r, s = _reference(a, b)
        ref, mag = ref + al * r, mag + abs(al) * s
        A = torch.as_tensor(np.ascontiguousarray(a.T if flags & 1 else a), device="cuda")
        B = torch.as_tensor(np.ascontiguousarray(b.T if flags & 2 else b), device="cuda")
        segs.append((A, A.shape[1], B, B.shape[1], k, al, flags, 0, 0))
    C = _run(monkeypatch, M, N, segs, mode, 4 if mode == 1 else 1)
    # (5e-324: products that leave the range of FP64)
    tol = (K + 9 + 4) * 2.0 ** -53 * mag + (K + 9) * 5e-324
    bad = np.abs(C - ref) > tol
    assert not bad.any(), (int(bad.sum()), float((np.abs(C - ref) / np.maximum(mag, 1e-320)).max()))


@pytest.mark.parametrize("n", [28, 70])
def test_identity_returns_the_elements(monkeypatch, n):
    """A product with the identity is a copy, small elements included."""
    rng = np.random.default_rng(n)
    a = rng.standard_normal((150, n)) * 10.0 ** rng.uniform(-200, 0, (150, n))
    A, eye = torch.as_tensor(a, device="cuda"), torch.eye(n, dtype=torch.float64, device="cuda")
    C = _run(monkeypatch, 150, n, [(A, n, eye, n, n, 1.0)], 0, 1)
    assert np.array_equal(C, a)


def test_leading_identity_of_a_transformation():
    from qodeapplications_gb300.orbitals import transform_indices
    rng = np.random.default_rng(7)
    x = rng.standard_normal((40, 40)) * 10.0 ** rng.uniform(-30, 0, (40, 40))
    perm = np.eye(40)[rng.permutation(40)]
    got = transform_indices(torch.as_tensor(x, device="cuda"), [None, torch.as_tensor(perm, device="cuda")])
    assert np.array_equal(got.cpu().numpy(), x @ perm)
