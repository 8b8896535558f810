"""Products over the determinants and over t^3 integrals on either side of their dispatch rules: the
tensor-core and the CUDA-core path give the same FP64 results to rounding."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "tf32x3"])
@pytest.mark.parametrize("n_orb,n_states", [(6, 5), (7, 33)])
def test_monomer_products(monkeypatch, precision, n_orb, n_states):
    from perf import cases
    from qodeapplications_gb300 import hamiltonian
    got = []
    for limit in (1 << 60, 0):
        monkeypatch.setattr(hamiltonian, "MONO_SLICED_MIN", limit)
        state = cases.prepare(dict(kind="hbuild", precision=precision, n_orb=n_orb, n_states=n_states), 3)
        assert (state["plan"].mono_abt is None) == (limit == 0)
        H = cases.run(state)
        got.append({k: x.clone() for k, x in (H.items() if isinstance(H, dict) else [("H", H)])})
    # sums over K <= 1 470 determinants, each path within K ulp of sum |z sigma|, H's scale
    for k, a in got[0].items():
        assert float((a - got[1][k]).abs().max()) <= 2 * 1470 * 2.0 ** -53 * max(1.0, float(a.abs().max()))


@pytest.mark.parametrize("n_orb", [3, 7])
def test_orbital_product(monkeypatch, n_orb):
    from perf import cases
    from qodeapplications_gb300 import gradients
    got = []
    for limit in (1000, 0):
        monkeypatch.setattr(gradients, "ORBITAL_SLICED_MIN", limit)
        state = cases.prepare(dict(kind="gradient", precision="fp64", n_orb=n_orb, n_states=3), 3)
        got.append(cases.run(state)["kappa"].clone())
        assert (state["adj"]._orb["VG"] is None) == (limit == 1000)
    # sums of t^3 products, t = 4 n_orb
    tol = 2 * (4 * n_orb) ** 3 * 2.0 ** -53
    assert float((got[0] - got[1]).abs().max()) <= tol * max(1.0, float(got[0].abs().max()))
