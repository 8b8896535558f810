"""FP64 densities of states whose coefficients differ by many orders of magnitude: every element keeps the
bound of an FP64 sum over its couplings, (count + 4) 2^-53 sum |z_b||z_k| on either side, also where
no coupling holds a large coefficient."""
import numpy as np
import pytest

from qodeapplications_gb300 import synthetic as S

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
CHG = (+1, 0, -1)


def _reference(cp, zb, zk):
    """(sums over the couplings, sums of absolute values, couplings of the index) [K, nb, nk] in FP64."""
    idx = torch.repeat_interleave(torch.arange(cp.K, device=zb.device), cp.idx_ptr[1:] - cp.idx_ptr[:-1])
    ref = torch.zeros((cp.K, zb.shape[1], zk.shape[1]), dtype=torch.float64, device=zb.device)
    mag = torch.zeros_like(ref)
    for a in range(0, len(idx), 4096):
        s = slice(a, a + 4096)
        p = cp.sign[s].double()[:, None, None] * zb[cp.P[s].long()][:, :, None] * zk[cp.Q[s].long()][:, None, :]
        ref.index_add_(0, idx[s], p)
        mag.index_add_(0, idx[s], p.abs())
    return ref, mag, (cp.idx_ptr[1:] - cp.idx_ptr[:-1]).double()[:, None, None]


# pad widths 16, 32, 64 and blocks of 64; "dominant": one determinant near 1, tails down to 1e-12;
# "states": sizes of their own for every state and determinant
@pytest.mark.parametrize("kind", ["dominant", "states"])
@pytest.mark.parametrize("n_orb,n", [(4, 3), (8, 16), (5, 17), (6, 33), (4, 65)])
def test_error_relative_to_the_products(n_orb, n, kind):
    from qodeapplications_gb300.densities import DensityBuilder, FragmentSpace
    space = FragmentSpace({c: S.sector_configs(n_orb, 0, 4 - c, (0,) if c == 0 else (-1, 1)) for c in CHG}, n_orb, 0, 4)
    ns = {c: n for c in CHG}
    b = DensityBuilder(space, ns, mirror=False, antisym=False)
    assert b.sliced is not None
    rng = np.random.default_rng(n_orb * 100 + n)
    z = {}
    for c in CHG:
        x = rng.standard_normal((n, space.n_conf[c]))
        if kind == "dominant":
            x *= 10.0 ** rng.uniform(-12, -3, (1, space.n_conf[c]))
            x[:, rng.integers(space.n_conf[c])] = 1.0
        else:
            x *= 10.0 ** rng.uniform(-14, 0, x.shape)
        z[c] = torch.as_tensor(x, device="cuda")
    b.build(z)
    b.check()
    for (op, bc, kc), cp in space.couplings.items():
        ref, mag, cnt = _reference(cp, z[bc].t().contiguous(), z[kc].t().contiguous())
        got = b._tmp[(op, bc, kc)].view(cp.K, n, n)
        bad = (got - ref).abs() > 2 * (cnt + 4) * 2.0 ** -53 * mag
        assert not bool(bad.any()), (op, bc, kc, int(bad.sum()), float(((got - ref).abs() / mag.clamp_min(1e-300)).max()))
