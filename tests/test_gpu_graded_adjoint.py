"""The density adjoint on determinants and gradients of very different sizes: every element of dE/dz keeps
the bound of sums in the result's type, (couplings + states + 4) eps sum |z||G| (eps = 2^-52 in FP64, 2^-23
in FP32: products, additions, and in FP32 the rounding of the operands)."""
import numpy as np
import pytest

from test_gpu_adjoint_sliced import _reference, _run, _space

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _graded(rng, shape, kind, small):
    x = rng.standard_normal(shape)
    if kind == "determinants":                        # tails of a wave function: rows of one size each
        return x * 10.0 ** rng.uniform(-small, 0, (shape[0],) + (1,) * (len(shape) - 1))
    if kind == "elements":
        return x * 10.0 ** rng.uniform(-small, 0, shape)
    if kind == "opposed":                             # large elements meet small ones only
        k = np.arange(shape[-1]) / max(shape[-1] - 1, 1)
        return x * 10.0 ** (-small * (k if len(shape) == 2 else 1.0 - k))
    raise ValueError(kind)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("kind", ["determinants", "elements", "opposed", "one index"])
@pytest.mark.parametrize("n_orb,nb,nk", [(4, 3, 16), (6, 17, 17), (6, 32, 30), (4, 64, 64), (4, 70, 66)])
def test_error_relative_to_the_products(precision, kind, n_orb, nb, nk):
    space = _space(n_orb)
    cp = space.couplings[("caa", 0, -1)]
    rng = np.random.default_rng(n_orb * 100 + nb)
    small = 14 if precision == "fp64" else 12
    of = "determinants" if kind == "one index" else kind
    zb, zk = (torch.as_tensor(_graded(rng, (space.n_conf[c], n), of, small), device="cuda") for c, n in ((0, nb), (-1, nk)))
    G = _graded(rng, (cp.K, nb, nk), of, small)
    if kind == "one index":                           # nothing but the rows of its own couplings in a sum
        G[np.arange(cp.K) != int(cp.ranges()[0][7])] = 0.0
    if kind == "opposed":                             # along both state indices
        G = G * 10.0 ** (-small * (1.0 - np.arange(nb) / max(nb - 1, 1)))[:, None]
    G = torch.as_tensor(G, device="cuda")
    got = _run(space, cp, precision, nb, nk, zb, zk, G)
    eps = 2.0 ** -52 if precision == "fp64" else 2.0 ** -23
    for x, (ref, mag, _top, cnt) in zip(got, _reference(cp, zb, zk, G)):
        # (1e-37: FP32 results below its normal range)
        tol = (cnt + max(nb, nk) + 4) * eps * mag + (0.0 if precision == "fp64" else 1e-37)
        bad = (x - ref).abs() > tol
        assert not bool(bad.any()), (int(bad.sum()), float(((x - ref).abs() / mag.clamp_min(1e-300)).max()))
