"""FP64 densities of states in classes (as Sz classes after a rounded state update): large coefficients on
the determinants of the own class, tiny ones on the rest, so that whole classes of elements are formed
beside the digits, by tiles of rows with the same marked columns.  Bound as in test_gpu_graded_densities.py:
2 (count + 4) 2^-53 sum |z_b||z_k|."""
import numpy as np
import pytest

from qodeapplications_gb300 import synthetic as S
from test_gpu_graded_densities import CHG, _reference

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


# classes of 1 (all marked or none), 2, 3 rows that do not fill tiles of 4 x 2; 64 is a whole block
@pytest.mark.parametrize("classes", [2, 3, 64])
@pytest.mark.parametrize("n_orb,n", [(4, 5), (7, 16), (6, 21), (6, 64), (5, 70)])
def test_error_relative_to_the_products(n_orb, n, classes):
    from qodeapplications_gb300.densities import DensityBuilder, FragmentSpace
    space = FragmentSpace({c: S.sector_configs(n_orb, 0, 4 - c, (0,) if c == 0 else (-1, 1)) for c in CHG}, n_orb, 0, 4)
    b = DensityBuilder(space, {c: n for c in CHG}, mirror=False, antisym=False)
    assert b.sliced is not None
    rng = np.random.default_rng(n_orb * 100 + n + classes)
    z = {}
    for c in CHG:
        x = rng.standard_normal((n, space.n_conf[c]))
        own = np.arange(n)[:, None] % classes == np.arange(space.n_conf[c])[None, :] % classes
        z[c] = torch.as_tensor(np.where(own, x, 1e-11 * x), device="cuda")
    b.build(z)
    b.check()
    for (op, bc, kc), cp in space.couplings.items():
        ref, mag, cnt = _reference(cp, z[bc].t().contiguous(), z[kc].t().contiguous())
        got = b._tmp[(op, bc, kc)].view(cp.K, n, n)
        bad = (got - ref).abs() > 2 * (cnt + 4) * 2.0 ** -53 * mag
        assert not bool(bad.any()), (op, bc, kc, int(bad.sum()), float(((got - ref).abs() / mag.clamp_min(1e-300)).max()))
