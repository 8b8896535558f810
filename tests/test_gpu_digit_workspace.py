"""The digits of the FP64 launches of a plan lie in one workspace, its reverse pass's too (or in a second one
where that needs more); what one launch leaves there does not reach another."""
import pytest

from qodeapplications_gb300 import synthetic as S

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
CHG = (+1, 0, -1)


def _buffers(gemms):
    return {g.sliced.work.data_ptr(): g.sliced.work.numel() for g in gemms if getattr(g, "sliced", None)}


@pytest.mark.parametrize("orbitals", [3, 7])
def test_plan_and_reverse_pass(orbitals):
    from qodeapplications_gb300.iteration import XRStateOptimizer
    sysd = S.make_system(n_frag=2, n_orb=orbitals, n_states=5, charges=CHG, seed=4)
    opt = XRStateOptimizer(sysd, use_graphs=False)
    plan, adj = opt.plan, opt.adj
    forward = [plan.pre, plan.fin, plan.sigma_batch.gemm]
    reverse = [adj.L1, adj.L2, adj.L3, adj.Lgamma]
    used = [g for g in forward + reverse if g.sliced]
    assert len(used) >= 4
    assert len(_buffers(forward)) == 1 and len(_buffers(forward + reverse)) <= 2
    assert max(_buffers(forward + reverse).values()) == max(g.sliced.size for g in used)
    # the same iterations with a workspace per launch (full of the largest doubles at the start)
    energies = [opt.iterate() for _ in range(3)]
    other = XRStateOptimizer(sysd, use_graphs=False)
    for g in [other.plan.pre, other.plan.fin, other.plan.sigma_batch.gemm, other.adj.L1, other.adj.L2, other.adj.L3,
              other.adj.Lgamma]:
        if g.sliced:
            g.sliced.work.fill_(0x7f)
    assert [other.iterate() for _ in range(3)] == pytest.approx(energies, abs=1e-12)


def test_shared_by_the_pairs_of_a_trimer():
    from qodeapplications_gb300.densities import FragmentSpace
    from qodeapplications_gb300.hamiltonian import DeviceIntegrals
    from qodeapplications_gb300.trimer_hv import XRTrimerHamiltonian
    sysd = S.make_system(n_frag=3, n_orb=4, n_states=2, charges=CHG, seed=5)
    spaces = [FragmentSpace({c: sysd["states"][m][c][1] for c in CHG}, 4, 0, 4) for m in range(3)]
    t = XRTrimerHamiltonian(spaces, [{c: 2 for c in CHG}] * 3, [CHG] * 3, DeviceIntegrals(h=sysd["h"], V=sysd["V"], Ns=sysd["Ns"]))
    gemms = [g for p in t.plans for g in (p.pre, p.fin, p.sigma_batch.gemm)] + [t.stage1] + t.simt
    assert sum(1 for g in gemms if g.sliced) >= 6 and len(_buffers(gemms)) == 1


def test_a_launch_without_its_workspace_is_an_error(monkeypatch):
    from qodeapplications_gb300 import gemm
    from qodeapplications_gb300.sliced import Workspace
    monkeypatch.setattr(gemm, "SLICED_MIN_CHAIN", 0)
    a, c = torch.randn(40, 40, dtype=torch.float64, device="cuda"), torch.zeros(40, 40, dtype=torch.float64, device="cuda")
    g = gemm.GroupedGemm()
    g.add(40, 40, [(a, 40, a, 40, 40, 1.0)], c, 40)
    work = Workspace(a.device)
    g.finalize(work=work)
    with pytest.raises(RuntimeError, match="workspace"):
        g.run()
    work.allocate()
    g.run()
    assert float((c - a @ a.t()).abs().max()) < 1e-12
