"""FP64 densities on the tensor cores (digit slices) against the CUDA-core FP64 kernel.

States are normalised, so a density element is a sum of at most n_conf products whose absolute
values add up to at most 1 (Cauchy-Schwarz): both sides round at most n_conf times, n_conf 2^-52,
and the digits resolve 2^-61 of a state's largest coefficient, n_conf 2^-60."""
import numpy as np
import pytest

from qodeapplications_gb300 import synthetic as S

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
CHG = (+1, 0, -1)


def _states(space, n, rng):
    out = {}
    for c in space.charges:
        z = rng.standard_normal((n[c], space.n_conf[c])) * 10.0 ** rng.uniform(-8, 0, (1, space.n_conf[c]))
        out[c] = torch.as_tensor(z / np.linalg.norm(z, axis=1, keepdims=True), device="cuda")
    return out


def _space(n_orb):
    from qodeapplications_gb300.densities import FragmentSpace
    return FragmentSpace({c: S.sector_configs(n_orb, 0, 4 - c, (0,) if c == 0 else (-1, 1)) for c in CHG}, n_orb, 0, 4)


def _reference(builder, *args):
    """The same build with xrh_density_accumulate."""
    kept, builder.sliced = builder.sliced, None
    ref = {(op, k): t.clone() for op, blocks in builder.build(*args).items() for k, t in blocks.items()}
    builder.sliced = kept
    return ref


# state counts at the edges of the 16, 32 and 64 wide layouts and of the blocks of 64; orbitals so
# that the longest indices stay inside one exact group, or span several
@pytest.mark.parametrize("n_orb,n", [(4, 1), (4, 3), (5, 16), (9, 16), (5, 17), (6, 32), (8, 32), (5, 33), (8, 64), (5, 65), (6, 70)])
def test_matches_cuda_core_kernel(n_orb, n):
    from qodeapplications_gb300.densities import DensityBuilder
    space = _space(n_orb)
    ns = {+1: n, 0: max(1, n - 2), -1: n}
    b = DensityBuilder(space, ns)
    z = _states(space, ns, np.random.default_rng(n))
    assert b.sliced is not None
    ref = _reference(b, z)
    for t in b._tmp.values():                    # nothing of the reference run may be left to read
        t.zero_()
    rho = b.build(z)
    b.check()
    tol = max(space.n_conf.values()) * (2.0 ** -52 + 2.0 ** -60)
    for (op, k), want in ref.items():
        assert float((rho[op][k] - want).abs().max()) <= tol, (op, k)


def test_separate_bra_states_full_lists_and_new_coefficients():
    from qodeapplications_gb300.densities import DensityBuilder
    space = _space(5)
    nk, nb = {c: 7 for c in CHG}, {c: 19 for c in CHG}
    b = DensityBuilder(space, nk, n_states_bra=nb, mirror=False, antisym=False)
    for seed in (1, 2):
        z, zb = _states(space, nk, np.random.default_rng(seed)), _states(space, nb, np.random.default_rng(10 + seed))
        ref = _reference(b, z, zb)
        rho = b.build(z, zb)
        b.check()
        for (op, k), want in ref.items():
            assert float((rho[op][k] - want).abs().max()) <= max(space.n_conf.values()) * 2.0 ** -51, (op, k)


def test_states_with_infinities_and_nan():
    """Blocks of the other states are untouched; the state's own elements are what FP64 gives."""
    from qodeapplications_gb300.densities import DensityBuilder
    space = _space(4)
    ns = {c: 5 for c in CHG}
    b = DensityBuilder(space, ns, mirror=False, antisym=False)
    z = _states(space, ns, np.random.default_rng(3))
    z[0][2, 4], z[-1][1, 0] = float("inf"), float("nan")
    ref = _reference(b, z)
    rho = b.build(z)
    for (op, k), want in ref.items():
        got = rho[op][k]
        assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf()), (op, k)
        ok = want.isfinite()
        assert float((got - want)[ok].abs().max()) <= max(space.n_conf.values()) * 2.0 ** -51, (op, k)
