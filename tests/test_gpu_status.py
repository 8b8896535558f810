"""A bounded device wait that gave up (its status word is planted on the host: nothing waits here) is
reported by every public FP64 call that hands results to the host or waits for the device, and by
check_status of the objects that do neither."""
import types

import numpy as np
import pytest

import xr_oracle as O
from qodeapplications_gb300 import synthetic as S

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
CHG = [+1, 0, -1]


@pytest.fixture
def gave_up(monkeypatch):
    from qodeapplications_gb300 import _lib

    def plant():
        monkeypatch.setattr(_lib, "status_word",
                            lambda dev: torch.full((1,), _lib.XRH_ERR_TIMEOUT, dtype=torch.int32, device=dev))
        return pytest.raises(_lib.XRHError, match="reported status")
    return plant


def _system(n_frag=2, n_orb=4, n_states=3):
    sysd = S.make_system(n_frag=n_frag, n_orb=n_orb, n_states=n_states, charges=CHG, seed=3)
    oi = O.FragInts(sysd["h"], sysd["V"], sysd["Ns"])
    return sysd, oi


def test_build_density_tensors(gave_up):
    from qodeapplications_gb300.densities import build_density_tensors
    sysd, _ = _system()
    z = {c: types.SimpleNamespace(coeffs=co, configs=np.array([[o for o in range(8) if int(m) >> o & 1] for m in masks]))
         for c, (co, masks) in sysd["states"][0].items()}
    V = np.asarray(sysd["V"])[:8, :8, :8, :8]
    build_density_tensors(z, 4, V, 0)
    with gave_up():
        build_density_tensors(z, 4, V, 0)


def test_monomer_two_electron(gave_up):
    from qodeapplications_gb300.densities import FragmentSpace
    from qodeapplications_gb300.hamiltonian import DeviceIntegrals, monomer_two_electron
    sysd, _ = _system(n_orb=6)                       # (long enough sums for the tensor cores)
    st = sysd["states"][0]
    space = FragmentSpace({c: st[c][1] for c in CHG}, 6, 0, 4)
    z = {0: torch.as_tensor(st[0][0], device="cuda")}
    V = DeviceIntegrals(h=sysd["h"], V=sysd["V"], Ns=sysd["Ns"]).V(0, 0, 0, 0).contiguous()
    monomer_two_electron(space, z, V, 0)
    with gave_up():
        monomer_two_electron(space, z, V, 0)


def test_orbital_transformations(gave_up):
    from qodeapplications_gb300.orbitals import transform_indices, transform_integrals, transform_ints
    x, m = torch.randn(40, 40, dtype=torch.float64, device="cuda"), torch.eye(40, dtype=torch.float64, device="cuda")
    ints = {"S": m.clone(), "T": x, "V": torch.randn((40,) * 4, dtype=torch.float64, device="cuda")}
    U = np.eye(20)
    transform_indices(x, [m, m])
    raises = gave_up()
    with raises:
        transform_indices(x, [m, m])
    with raises:
        transform_integrals(m, ints)
    with raises:
        transform_ints(U, ints, [10, 10])


@pytest.mark.parametrize("device", [False, True])
def test_get_xr_H_and_diagrams(gave_up, device):
    from qodeapplications_gb300 import diagrams
    from qodeapplications_gb300.diagrammatic_expansion import blocks
    from qodeapplications_gb300.get_xr_result import get_xr_H
    sysd, oi = _system()
    dens = [O.build_densities({c: O.Sector(*sysd["states"][m][c]) for c in CHG}, 4, 0, 4) for m in range(2)]
    get_xr_H((oi, oi, None), dens, 0, [CHG, CHG], device=device)
    blocks(dens, oi, diagrams.SV_diagrams)[(0, 1)][((0, 0), (0, 0))]["v0101"]
    raises = gave_up()
    with raises:
        get_xr_H((oi, oi, None), dens, 0, [CHG, CHG], device=device)
    with raises:
        blocks(dens, oi, diagrams.SV_diagrams)[(0, 1)][((0, 0), (0, 0))]["v0101"]


def test_fragment_states(gave_up):
    from qodeapplications_gb300.fragment_states import FragmentHamiltonian, fci_states
    from qodeapplications_gb300.hamiltonian import DeviceIntegrals
    sysd, _ = _system(n_orb=6)
    ints = DeviceIntegrals(h=sysd["h"], V=sysd["V"], Ns=sysd["Ns"])
    masks, h, V = sysd["states"][0][0][1], ints.T(0, 0).contiguous(), ints.V(0, 0, 0, 0).contiguous()
    raises = gave_up()
    with raises:
        fci_states(masks, 6, 0, h, V, 1)
    f = FragmentHamiltonian(masks, 6, 0, h, V)
    f.apply(torch.ones(1, f.n_conf, dtype=torch.float64, device="cuda"))
    with raises:
        f.check_status()
    with raises:
        f.matrix()


def test_trimer_blocks(gave_up):
    from qodeapplications_gb300.densities import DensityBuilder, FragmentSpace
    from qodeapplications_gb300.hamiltonian import DeviceIntegrals
    from qodeapplications_gb300.trimer import XRTrimerPlan
    sysd, _ = _system(n_frag=3, n_orb=3, n_states=2)
    ns = {c: 2 for c in CHG}
    rho = []
    for m in range(3):
        b = DensityBuilder(FragmentSpace({c: sysd["states"][m][c][1] for c in CHG}, 3, 0, 4), ns)
        rho.append(b.build({c: torch.as_tensor(sysd["states"][m][c][0], device="cuda") for c in CHG}))
    raises = gave_up()
    plan = XRTrimerPlan(rho, DeviceIntegrals(h=sysd["h"], V=sysd["V"], Ns=sysd["Ns"]), [4] * 3, [CHG] * 3, [ns] * 3)
    plan.launch()
    with raises:
        plan.check_status()


@pytest.mark.parametrize("use_graphs", [False, True])
def test_optimizer(use_graphs):
    """One word for the launches of an optimizer's plan and reverse pass."""
    from qodeapplications_gb300 import _lib
    from qodeapplications_gb300.iteration import XRStateOptimizer
    sysd, _ = _system()
    opt = XRStateOptimizer(sysd, use_graphs=use_graphs)
    for _ in range(3):
        opt.iterate()
    words = {g.sliced.status.data_ptr() for g in (opt.plan.pre, opt.plan.fin, opt.adj.L1, opt.adj.L2, opt.adj.L3) if g.sliced}
    words |= {b.sliced.status.data_ptr() for b in opt.plan.builders} | {s.status.data_ptr() for s in opt.adj.dens_adj_sliced}
    assert words == {opt.plan.status.data_ptr()}
    opt.plan.status.fill_(_lib.XRH_ERR_TIMEOUT)
    with pytest.raises(_lib.XRHError, match="reported status"):
        opt.iterate()
    with pytest.raises(_lib.XRHError, match="reported status"):
        opt.gradient_norm


def test_differentiable_energy():
    from qodeapplications_gb300 import _lib
    from qodeapplications_gb300.autograd import XRDimerEnergy
    sysd, _ = _system()
    e = XRDimerEnergy.from_system(sysd)
    h, V = (torch.as_tensor(sysd[k], device="cuda").requires_grad_() for k in ("h", "V"))
    z = [{c: torch.as_tensor(sysd["states"][m][c][0], device="cuda") for c in CHG} for m in range(2)]
    E = e(h, V, z)
    e.plan.status.fill_(_lib.XRH_ERR_TIMEOUT)
    with pytest.raises(_lib.XRHError, match="reported status"):
        E.backward()
    with pytest.raises(_lib.XRHError, match="reported status"):
        e(h, V, z)


def test_ring():
    from qodeapplications_gb300 import _lib
    from qodeapplications_gb300.ring import XRRing
    r = XRRing(n_frag=3, n_orb=3, n_states=2, n_elec_ref=3, precision="fp64", graph=False, autotune=False)
    r.iterate(with_triples=False)
    r.plan.status.fill_(_lib.XRH_ERR_TIMEOUT)
    with pytest.raises(_lib.XRHError, match="reported status"):
        r.iterate(with_triples=False)
