"""The density adjoint on the tensor cores (digit slices) against FP64 PyTorch products.

A gradient row is a sum over couplings c of products with |z| <= 1 (normalised states): every
rounding is relative to S = sum_c sum |z||G|, formed beside the reference.  FP64: one rounding per
product and at most `count` atomic additions, (count + 4) 2^-52 S, plus the 62-bit resolution of digits
(states and columns scaled by their largest element), 2^-58 max|z| sum_c max|G|.  FP32: the same with
2^-23 and the 46-bit resolution 2^-42."""
import numpy as np
import pytest

from qodeapplications_gb300 import synthetic as S

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _space(n_orb):
    from qodeapplications_gb300.densities import FragmentSpace
    return FragmentSpace({c: S.sector_configs(n_orb, 0, 4 - c, (0,) if c == 0 else (-1, 1)) for c in (0, -1)}, n_orb, 0, 4)


def _run(space, cp, precision, nb, nk, zb, zk, G):
    """(gzb, gzk) of the sliced kernel for one caa block (bra charge 0, ket charge -1)."""
    from qodeapplications_gb300 import _lib
    from qodeapplications_gb300.densities import CoeffDigits, SlicedDensityAdjoint
    dt = torch.float64 if precision == "fp64" else torch.float32
    coeff = CoeffDigits({"bra": {0: zb}, "ket": {-1: zk}}, zb.device, slices=8 if precision == "fp64" else 6)
    gb, gk = (torch.zeros(z.shape, dtype=dt, device=zb.device) for z in (zb, zk))
    adj = SlicedDensityAdjoint([(cp, coeff, ("bra", 0), ("ket", -1), G, gb, gk)],
                               _lib.FP64 if precision == "fp64" else _lib.FP32, [coeff], zb.device)
    adj.run(_lib.stream_ptr())
    adj.check()
    return gb.double(), gk.double()


def _reference(cp, zb, zk, G):
    """The two products per coupling and the sums of their absolute values, in FP64."""
    idx = torch.repeat_interleave(torch.arange(cp.K, device=zb.device), cp.idx_ptr[1:] - cp.idx_ptr[:-1])
    P, Q, s = cp.P.long(), cp.Q.long(), cp.sign.double()
    out = []
    for z, rows, dst, tr, n_dst in ((zk, Q, P, True, zb.shape[0]), (zb, P, Q, False, zk.shape[0])):
        ref = torch.zeros((n_dst, G.shape[1] if tr else G.shape[2]), dtype=torch.float64, device=zb.device)
        mag, cnt, top = torch.zeros_like(ref), torch.zeros(n_dst, dtype=torch.float64, device=zb.device), torch.zeros_like(ref)
        for a in range(0, len(idx), 4096):
            g = G[idx[a:a + 4096]]
            g = g if tr else g.transpose(1, 2)
            x = z[rows[a:a + 4096]]
            ref.index_add_(0, dst[a:a + 4096], s[a:a + 4096, None] * torch.einsum("cok,ck->co", g, x))
            mag.index_add_(0, dst[a:a + 4096], torch.einsum("cok,ck->co", g.abs(), x.abs()))
            top.index_add_(0, dst[a:a + 4096], g.abs().amax(2) * z.abs().max())
            cnt.index_add_(0, dst[a:a + 4096], torch.ones(len(x), dtype=torch.float64, device=zb.device))
        out.append((ref, mag, top, cnt[:, None]))
    return out


# state counts at the edges of the pad widths and blocks; n_orb so that indices have less than one
# tile of 128 couplings, and several
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("n_orb,nb,nk", [(3, 1, 1), (4, 3, 16), (6, 17, 5), (6, 32, 32), (4, 33, 64), (5, 65, 7), (4, 70, 66)])
def test_matches_fp64_products(precision, n_orb, nb, nk):
    space = _space(n_orb)
    cp = space.couplings[("caa", 0, -1)]
    g = torch.Generator().manual_seed(n_orb * 100 + nb)
    zb, zk = (torch.randn(space.n_conf[c], n, generator=g, dtype=torch.float64) *
              10.0 ** (-4 * torch.rand(space.n_conf[c], n, generator=g, dtype=torch.float64)) for c, n in ((0, nb), (-1, nk)))
    zb, zk = (x.div(x.norm(dim=0)).cuda() for x in (zb, zk))
    G = torch.randn(cp.K, nb, nk, generator=g, dtype=torch.float64).cuda() * 0.01
    got = _run(space, cp, precision, nb, nk, zb, zk, G)
    eps, res = (2.0 ** -52, 2.0 ** -58) if precision == "fp64" else (2.0 ** -23, 2.0 ** -42)
    n = max(nb, nk)
    for x, (ref, mag, top, cnt) in zip(got, _reference(cp, zb, zk, G)):
        tol = (cnt + 4) * eps * mag + n * res * top
        assert bool(((x - ref).abs() <= tol).all()), float(((x - ref).abs() / tol.clamp_min(1e-300)).max())


def test_infinite_gradient_element_stays_in_its_index():
    """An infinite dE/drho element reaches the rows of its own operator index only."""
    space = _space(4)
    cp = space.couplings[("caa", 0, -1)]
    g = torch.Generator().manual_seed(9)
    zb, zk = (torch.randn(space.n_conf[c], 4, generator=g, dtype=torch.float64).cuda() for c in (0, -1))
    G = torch.randn(cp.K, 4, 4, generator=g, dtype=torch.float64).cuda()
    idx = int(cp.ranges()[0][5])
    G[idx, 1, 2] = float("inf")
    gb, gk = _run(space, cp, "fp64", 4, 4, zb, zk, G)
    (rb, _, _, _), (rk, _, _, _) = _reference(cp, zb, zk, G)
    for x, ref in ((gb, rb), (gk, rk)):
        assert torch.equal(x.isfinite(), ref.isfinite())
        ok = ref.isfinite()
        assert float((x - ref)[ok].abs().max()) <= 1e-12 * float(ref[ok].abs().max())
