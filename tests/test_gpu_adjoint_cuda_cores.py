"""The reverse pass through the density adjoint on the tensor cores against the same pass through the CUDA-core
kernels (xrh_density_adjoint in FP64, xrh_density_adjoint_f32_grouped above 16 states on the split paths).

dE/dz elements are sums over n_conf-long lists of products with |z| <= 1: 1e-12 (FP64) and 2e-5 (FP32, its sums
of some thousand terms) of the largest element."""
import pytest

from qodeapplications_gb300 import synthetic as S

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
CHG = (+1, 0, -1)


def _gradients(precision, n_orb, n_states, cuda_cores, monkeypatch):
    from qodeapplications_gb300.densities import FragmentSpace
    from qodeapplications_gb300.gradients import XRDimerAdjoint
    from qodeapplications_gb300.hamiltonian import DeviceIntegrals, XRDimerPlan
    sysd = S.make_system(n_frag=2, n_orb=n_orb, n_states=n_states, charges=CHG, seed=8)
    spaces = [FragmentSpace({c: sysd["states"][m][c][1] for c in CHG}, n_orb, 0, 4) for m in range(2)]
    plan = XRDimerPlan(spaces, [{c: n_states for c in CHG}] * 2, [list(CHG)] * 2,
                       DeviceIntegrals(h=sysd["h"], V=sysd["V"], Ns=sysd["Ns"]), precision=precision, autotune=False)
    with monkeypatch.context() as m:
        if cuda_cores:
            m.setattr(XRDimerAdjoint, "_setup_sliced", lambda self: setattr(self, "dens_adj_sliced", []))
        adj = XRDimerAdjoint(plan)
    assert bool(adj.dens_adj_sliced) != cuda_cores
    assert bool(adj.dens_adj_groups) == (cuda_cores and precision != "fp64")       # made where they run
    plan.build([{c: torch.as_tensor(sysd["states"][m][c][0], device="cuda") for c in CHG} for m in range(2)])
    g = torch.Generator().manual_seed(1)
    d = torch.randn(plan.tot[0] * plan.tot[1], generator=g, dtype=torch.float64)
    adj.launch((d / d.norm()).cuda())
    out = adj.state_gradient()
    adj.check_status()
    return {(m, c): out[m][c].clone() for m in range(2) for c in CHG}


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("tf32x3", 2e-5)])
@pytest.mark.parametrize("n_orb,n_states", [(4, 17), (5, 33), (6, 64)])
def test_same_gradient(monkeypatch, precision, tol, n_orb, n_states):
    got = _gradients(precision, n_orb, n_states, False, monkeypatch)
    ref = _gradients(precision, n_orb, n_states, True, monkeypatch)
    for k, want in ref.items():
        assert float(want.abs().max()) > 0
        assert float((got[k] - want).abs().max()) <= tol * float(want.abs().max()), k
