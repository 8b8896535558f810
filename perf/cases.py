"""Timed cases of the excitonic-Hamiltonian (XR-H) framework, through its public entry points.

Every case is a seeded synthetic system of the kind the repository's tests and benchmark use: fragments
of n_orb spatial orbitals, four electrons when neutral, charges +1, 0, -1, orthonormal Gaussian states of
definite Sz, symmetric Gaussian one-electron integrals and Cholesky-built two-electron integrals (the
distributions of synthetic.make_system, drawn on the GPU).  The kinds of calls:

  densities  DensityBuilder.build: every transition density of one fragment from new states
  hbuild     XRDimerPlan.build: densities of both fragments and the dimer Hamiltonian from new states
  gradient   XRDimerAdjoint.launch, state_gradient and (fp64) orbital_gradient: the reverse pass on a built plan
  iterate    XRStateOptimizer.iterate: one whole optimizer iteration
  hpsi       FragmentHamiltonian.apply: determinant-space H Psi on a block of CI vectors
  orbitals   orbitals.transform_ints: integrals re-transformed to new orbitals, symmetric and biorthogonal
  trimer_hv  XRTrimerHamiltonian.apply: matrix-free H v of three fragments

n_orb 9 with 10 states and n_orb 14 with 40 or 60 states are the sizes of bench.py's configurations; the
FragmentSpace (determinant coupling lists) depends on the sizes alone and is kept as a program keeps it.
Split-precision plans are made with autotune=False: the autotuner picks split-K factors by timing, and with them
the order of FP32 sums, so that two processes would not return the same digits.  The reverse pass has no such
option; there the state gradient, whose FP32 atomics vary by more than that, is returned alone.
"""
import functools
import itertools
import math

import numpy as np
import torch

from qodeapplications_gb300 import synthetic
from qodeapplications_gb300.densities import DensityBuilder, FragmentSpace
from qodeapplications_gb300.fragment_states import FragmentHamiltonian
from qodeapplications_gb300.gradients import XRDimerAdjoint
from qodeapplications_gb300.hamiltonian import DeviceIntegrals, XRDimerPlan
from qodeapplications_gb300.iteration import XRStateOptimizer
from qodeapplications_gb300.orbitals import transform_ints
from qodeapplications_gb300.trimer_hv import XRTrimerHamiltonian

CHARGES = (+1, 0, -1)
N_ELEC = 4          # electrons of a neutral fragment
N_CHOL = 40
STEP = 0.02         # XRStateOptimizer's default step
KRYLOV = 48         # XRStateOptimizer's default Krylov depth of a first iteration
F64 = dict(dtype=torch.float64, device="cuda")


def listed():
    return [
        # the smallest optimizer iteration of the benchmark (config 1), in the default precision: latency and launches
        dict(name="iterate-fp64-9x10", kind="iterate", precision="fp64", n_orb=9, n_states=10),
        # backward of the same small dimer in split precision: state gradient alone, as a state optimisation asks for
        dict(name="gradient-tf32x3-9x10", kind="gradient", precision="tf32x3", n_orb=9, n_states=10),
        # H from new states with the default plan of a small dimer (900 x 900, product order)
        dict(name="hbuild-fp64-9x10", kind="hbuild", precision="fp64", n_orb=9, n_states=10),
        # H from new states at an odd, ragged size between the benchmark's two dimers
        dict(name="hbuild-fp64-11x27", kind="hbuild", precision="fp64", n_orb=11, n_states=27),
        # H of the benchmark's default dimer (2 x 14 orbitals, 60 states), default precision: the largest build
        dict(name="hbuild-fp64-14x60", kind="hbuild", precision="fp64", n_orb=14, n_states=60),
        # the same build in split precision, as in every headline iteration
        dict(name="hbuild-tf32x3-14x60", kind="hbuild", precision="tf32x3", n_orb=14, n_states=60),
        # backward: state and orbital gradient on a built plan, default precision, odd size
        dict(name="gradient-fp64-12x21", kind="gradient", precision="fp64", n_orb=12, n_states=21),
        # state gradient of the headline iteration
        dict(name="gradient-tf32x3-14x60", kind="gradient", precision="tf32x3", n_orb=14, n_states=60),
        # transition densities alone (what build_density_tensors and every sub-cluster of a chain starts with)
        dict(name="densities-fp64-14x40", kind="densities", precision="fp64", n_orb=14, n_states=40),
        # determinant-space H Psi on a block of CI vectors (five electrons in 28 spin orbitals)
        dict(name="hpsi-14x16", kind="hpsi", precision="fp64", n_orb=14, n_states=16),
        # the orbital optimizer's integral re-transformation of a dimer
        dict(name="orbitals-14", kind="orbitals", precision="fp64", n_orb=14, n_states=1),
        # matrix-free H v of the benchmark's trimer (3 x 14 orbitals, 40 states, neutral: 448 000 product states)
        dict(name="trimer_hv-tf32x3-14x40", kind="trimer_hv", precision="tf32x3", n_orb=14, n_states=40),
    ]


def draw(rng):
    kind = rng.choice(["iterate", "hbuild", "hbuild", "gradient", "gradient", "densities", "densities", "hpsi",
                       "orbitals", "trimer_hv"])
    precision = rng.choice(["fp64", "tf32x3"]) if kind in ("hbuild", "gradient") else \
        "tf32x3" if kind == "trimer_hv" else rng.choice(["fp64", "fp32"]) if kind == "densities" else "fp64"
    n_orb = rng.randint(6, 14)
    top = {"trimer_hv": 40, "hpsi": 32}.get(kind, 60)
    n_states = int(round(math.exp(rng.uniform(math.log(4), math.log(top)))))
    if kind in ("gradient", "iterate") and precision == "fp64":
        n_states = min(n_states, 33)     # a reverse pass costs about twice its build
    if kind == "orbitals":
        n_states = 1
    return dict(kind=kind, precision=precision, n_orb=n_orb, n_states=n_states)


# ------------------------------------------------------------------------------------ inputs --
@functools.lru_cache(maxsize=64)
def masks_of(n_orb, n_elec):
    """Determinants of one electron count (Sz = 0, or both of +-1/2) and twice their Sz."""
    want = (0,) if n_elec % 2 == 0 else (-1, 1)
    out, sz = [], []
    for comb in itertools.combinations(range(2 * n_orb), n_elec):
        s = sum(1 if o < n_orb else -1 for o in comb)
        if s in want:
            m = sum(1 << o for o in comb)
            out.append(m)
            sz.append(s)
    return np.array(out, dtype=np.uint64), np.array(sz)


@functools.lru_cache(maxsize=2)
def space_of(n_orb):
    return FragmentSpace({c: masks_of(n_orb, N_ELEC - c)[0] for c in CHARGES}, n_orb, 0, N_ELEC)


def generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def states(g, n_orb, n_states):
    """One fragment's orthonormal states {charge: (n_states, n_conf)}: odd electron counts alternate Sz."""
    out = {}
    for c in CHARGES:
        _, sz = masks_of(n_orb, N_ELEC - c)
        kinds = sorted(set(sz.tolist()), reverse=True)
        z = torch.zeros((n_states, len(sz)), **F64)
        for k, s in enumerate(kinds):
            rows = torch.arange(k, n_states, len(kinds), device="cuda")
            cols = torch.as_tensor(np.nonzero(sz == s)[0], device="cuda")
            q, _ = torch.linalg.qr(torch.randn((len(cols), len(rows)), generator=g, **F64))
            z[rows[:, None], cols[None, :]] = q.t()
        out[c] = z
    return out


def integrals(g, sizes):
    """h (N x N) and antisymmetrised V (N^4) over the spin orbitals of the fragments (alpha then beta in each)."""
    n = sum(sizes)
    a = 0.1 * torch.randn((n, n), generator=g, **F64)
    h = torch.triu(a) + torch.triu(a, 1).t()
    L = 0.05 * torch.randn((N_CHOL, n, n), generator=g, **F64)
    L = 0.5 * (L + L.transpose(1, 2))
    sp = torch.as_tensor(synthetic.spin_orbital_spatial_index(sizes), device="cuda")
    spin = torch.as_tensor(np.concatenate([np.repeat([0, 1], k) for k in sizes]), device="cuda")
    same = (spin[:, None] == spin[None, :]).to(torch.float64)
    h = h[sp][:, sp] * same
    Ls = L[:, sp][:, :, sp] * same
    N = len(sp)
    eri = (Ls.reshape(N_CHOL, -1).t() @ Ls.reshape(N_CHOL, -1)).view(N, N, N, N)     # (pr|qs) at [p, r, q, s]
    phys = eri.permute(0, 2, 1, 3)
    return h, (0.25 * (phys - phys.transpose(2, 3))).contiguous()


def inputs(case, seed, n_frag=2):
    g = generator(seed)
    h, V = integrals(g, [case["n_orb"]] * n_frag)
    zs = [states(g, case["n_orb"], case["n_states"]) for _ in range(n_frag)]
    return g, h, V, zs


def layout_of(case):
    """Small dimers take the plan's default (product order); large ones the per-sector blocks that iterations use."""
    return "product" if case["n_states"] <= 12 else "sectors"


def counts(case):
    return [{c: case["n_states"] for c in CHARGES}] * 2


def orbital_inputs(case, seed):
    """Spatial transformation, and spin-free overlap, T, U, V in spin orbitals."""
    g = generator(seed)
    sizes = [case["n_orb"]] * 2
    n = sum(sizes)
    T, V = integrals(g, sizes)
    sp = torch.as_tensor(synthetic.spin_orbital_spatial_index(sizes), device="cuda")
    spin = torch.as_tensor(np.concatenate([np.repeat([0, 1], k) for k in sizes]), device="cuda")
    same = (spin[:, None] == spin[None, :]).to(torch.float64)

    def sym(scale):
        a = scale * torch.randn((n, n), generator=g, **F64)
        return 0.5 * (a + a.t())

    S = (torch.eye(n, **F64) + sym(0.02))[sp][:, sp] * same
    U = torch.stack([sym(0.05)[sp][:, sp] * same for _ in sizes])
    x = 0.05 * torch.randn((n, n), generator=g, **F64)
    return torch.matrix_exp(x - x.t()), dict(S=S, T=T, U=U, V=V), sizes, sp, same


def ground_like(g, case, sector=0):
    """A normalised product-order vector that lies in one total-charge sector, as a ground state does."""
    n = case["n_states"]
    d = torch.randn((3 * n, 3 * n), generator=g, **F64)
    chg = torch.as_tensor(np.repeat(CHARGES, n), device="cuda")
    d *= (chg[:, None] + chg[None, :] == sector).to(torch.float64)
    return (d / d.norm()).reshape(-1)


def prepare(case, seed):
    kind, n_orb = case["kind"], case["n_orb"]
    if kind == "densities":
        z = states(generator(seed), n_orb, case["n_states"])
        builder = DensityBuilder(space_of(n_orb), {c: case["n_states"] for c in CHARGES}, precision=case["precision"])
        return dict(kind=kind, builder=builder, z=z)
    if kind == "orbitals":
        X, ints, sizes, _, _ = orbital_inputs(case, seed)
        return dict(kind=kind, X=X, ints=ints, sizes=sizes)
    if kind == "hpsi":
        g = generator(seed)
        h, V = integrals(g, [n_orb])
        masks = masks_of(n_orb, N_ELEC + 1)[0]
        H = FragmentHamiltonian(masks, n_orb, 0, h, V, n_vec=case["n_states"])
        psi = torch.randn((case["n_states"], len(masks)), generator=g, **F64)
        return dict(kind=kind, H=H, psi=psi / psi.norm(dim=1, keepdim=True))
    if kind == "trimer_hv":
        g, h, V, zs = inputs(case, seed, 3)
        H = XRTrimerHamiltonian([space_of(n_orb)] * 3, [{c: case["n_states"] for c in CHARGES}] * 3, [list(CHARGES)] * 3,
                                DeviceIntegrals.from_tensors(h, V, [2 * n_orb] * 3), precision=case["precision"],
                                hv_precision=case["precision"], total_charge=0, autotune=False)
        H.build(zs)
        v = torch.randn(H.dim, generator=g, **F64)
        return dict(kind=kind, H=H, v=v / v.norm())
    g, h, V, zs = inputs(case, seed)
    if kind == "iterate":
        host = [{c: (z.cpu().numpy(), masks_of(n_orb, N_ELEC - c)[0]) for c, z in zf.items()} for zf in zs]
        sysd = dict(n_frag=2, n_orb=n_orb, n_core=0, n_elec_ref=N_ELEC, charges=CHARGES, Ns=[2 * n_orb] * 2,
                    h=h.cpu().numpy(), V=V.cpu().numpy(), states=host)
        return dict(kind=kind, opt=XRStateOptimizer(sysd, precision=case["precision"]))
    ints = DeviceIntegrals.from_tensors(h, V, [2 * n_orb] * 2)
    layout = layout_of(case) if kind == "hbuild" else "sectors"
    plan = XRDimerPlan([space_of(n_orb)] * 2, counts(case), [list(CHARGES)] * 2, ints, output="full",
                       precision=case["precision"], layout=layout, autotune=case["precision"] == "fp64")
    if kind == "hbuild":
        return dict(kind=kind, plan=plan, zs=zs, layout=layout)
    plan.build(zs)
    return dict(kind=kind, adj=XRDimerAdjoint(plan), d=ground_like(g, case), orbital=case["precision"] == "fp64", T=h, V=V,
                U=torch.zeros((2,) + h.shape, **F64), index=synthetic.spin_orbital_spatial_index([n_orb] * 2))


# --------------------------------------------------------------------------------------- run --
def run(state):
    kind = state["kind"]
    if kind == "densities":
        return named_blocks(state["builder"].build(state["z"]))
    if kind == "hbuild":
        H = state["plan"].build(state["zs"])
        return H if state["layout"] == "product" else {str(t): s["H"] for t, s in state["plan"].sectors.items()}
    if kind == "gradient":
        adj = state["adj"]
        adj.launch(state["d"])
        if not state["orbital"]:
            return adj.state_gradient()
        return dict(states=adj.state_gradient(), kappa=adj.orbital_gradient(state["T"], state["U"], state["V"], state["index"]))
    if kind == "iterate":
        opt = state["opt"]
        E = opt.iterate()
        return dict(E=E, states=opt.plan.coeffs, kappa=opt.kappa_grad)
    if kind == "hpsi":
        return state["H"].apply(state["psi"])
    if kind == "orbitals":
        symm, bior = transform_ints(state["X"], state["ints"], state["sizes"])
        return dict(symm=symm, bior=bior)
    return state["H"].apply(state["v"])


def named_blocks(rho):
    return {"%s%+d%+d" % (op, b, k): t for op, blocks in rho.items() for (b, k), t in blocks.items()}


# -------------------------------------------------------------------------------------- work --
def conf(case):
    n = case["n_orb"]
    c = math.comb
    return {+1: 2 * c(n, 2) * n, 0: c(n, 2) ** 2, -1: 2 * c(n, 3) * c(n, 2)}


def density_work(case):
    """Bytes of one fragment's states and densities, FLOPs of its couplings (each operator tuple of an
    anticommuting pair once; a creation operator of the spin that leaves the list's Sz: half of the free ones)."""
    n, N, K = case["n_states"], 2 * case["n_orb"], conf(case)
    elems = n * n * (2 * (2 * N + 2 * N ** 3) + 2 * 2 * N * N // 2 + 3 * N * N)
    coup = 0.0
    for c in CHARGES:
        ne = N_ELEC - c
        coup += K[c] * ne * (N - ne + 1) / 4                       # ca (Hermitian half)
        if c < 1:                                                    # a and caa out of this ket
            coup += K[c] * ne / 2 + K[c] * ne * (ne - 1) / 2 * (N - ne + 2) / 2
    coup += K[-1] * 5 * 4 / 4                                        # aa from -1 to +1
    return 8 * (elems + n * sum(K.values())), 2.0 * n * n * coup


def h_work(case):
    """Bytes read (states, integrals) and written (H), FLOPs of the precontractions, final blocks and sigma."""
    n, N, K = case["n_states"], 2 * case["n_orb"], conf(case)
    _, dens = density_work(case)
    pre = 2 * (2 * 2 * n * n * N * (N + 2 * N ** 3) + 2 * n * n * N ** 4) + 3 * 2 * n * n * N ** 4
    blocks = 9 * 2 * n ** 4 * N * N + 8 * 4 * n ** 4 * N + 2 * 2 * n ** 4 * N * N
    sigma = 2 * sum(2.0 * n * K[c] * (N_ELEC - c) * (N_ELEC - c - 1) / 2 * (N * N / 6) for c in CHARGES)
    out = 19 * n ** 4
    return 8 * (2 * n * sum(K.values()) + (2 * N) ** 4 + out), 2 * dens + pre + blocks + sigma


def work(case):
    kind, n, N = case["kind"], case["n_states"], 2 * case["n_orb"]
    if kind == "densities":
        b, f = density_work(case)
    elif kind == "hbuild":
        b, f = h_work(case)
    elif kind == "gradient":        # every product of the build twice in reverse, H not written
        b, f = h_work(case)
        b, f = b - 8 * 19 * n ** 4 + 8 * 2 * n * sum(conf(case).values()), 2 * f
    elif kind == "iterate":
        b, f = h_work(case)
        b, f = b + 8 * 4 * n * sum(conf(case).values()), 3 * f
    elif kind == "hpsi":
        K = conf(case)[-1]
        b, f = 8 * (2 * n * K + N ** 4), 2.0 * n * K * 10 * N * N / 6
    elif kind == "orbitals":
        t = 2 * N
        b, f = 8 * 3 * t ** 4, 2.0 * 6 * t ** 5
    else:                            # trimer_hv: charge blocks through three stages of n^4 N^2
        b, f = 8 * (2 * 7 * n ** 3 + 9 * 3 * n ** 4 + 36 * n * n * N * N), 60 * 2.0 * n ** 4 * N * N + 2.0 * 57 * n ** 5
    return {"bytes": float(b), "flops": float(f)}


# ---------------------------------------------------- the same results in plain 64-bit torch --
@functools.lru_cache(maxsize=4)
def lowered(n_orb, n_elec, k):
    """Annihilation tables of the determinants of `n_elec` electrons after k annihilations: (list, table), the
    list of the next level and [(orbital) -> (source positions, target positions, signs)]."""
    N = 2 * n_orb
    src = masks_of(n_orb, n_elec)[0] if k == 0 else lowered(n_orb, n_elec, k - 1)[0]
    hit = [np.nonzero((src >> np.uint64(p)) & np.uint64(1))[0] for p in range(N)]
    dst = np.unique(np.concatenate([src[hit[p]] ^ np.uint64(1 << p) for p in range(N)]))
    table = []
    for p in range(N):
        above = src[hit[p]] >> np.uint64(p + 1)
        par = np.zeros(len(above), dtype=np.int64)
        for b in range(N):
            par ^= ((above >> np.uint64(b)) & np.uint64(1)).astype(np.int64)
        to = np.searchsorted(dst, src[hit[p]] ^ np.uint64(1 << p))
        table.append(tuple(torch.as_tensor(x, device="cuda") for x in (hit[p], to, 1.0 - 2.0 * par)))
    return dst, table


def lower(z, n_orb, n_elec, k):
    """a_p z for every spin orbital p: (N,) + z.shape[:-1] + (next determinants,)."""
    dst, table = lowered(n_orb, n_elec, k)
    out = []
    for hit, to, sign in table:
        y = torch.zeros(z.shape[:-1] + (len(dst),), **F64)
        out.append(y.index_copy(-1, to, z.index_select(-1, hit) * sign))
    return torch.stack(out)


def embed(z, n_orb, n_elec, other, k):
    """z over the determinants that `other` electrons have after k annihilations."""
    dst = lowered(n_orb, other, k - 1)[0]
    src = masks_of(n_orb, n_elec)[0]
    at = np.searchsorted(dst, src)
    ok = (at < len(dst)) & (dst[np.minimum(at, len(dst) - 1)] == src)
    y = torch.zeros((z.shape[0], len(dst)), **F64)
    return y.index_copy(1, torch.as_tensor(at[ok], device="cuda"), z[:, torch.as_tensor(np.nonzero(ok)[0], device="cuda")])


def common(a, la, b, lb):
    """a and b, last index over determinant lists la and lb, on the determinants that both lists have."""
    both = np.intersect1d(la, lb)
    ia, ib = (torch.as_tensor(np.searchsorted(x, both), device="cuda") for x in (la, lb))
    return a.index_select(-1, ia), b.index_select(-1, ib)


def pairing(a, la, b, lb):
    """sum_X a[.., X] b[.., X] as a (rows of a) x (rows of b) matrix."""
    x, y = common(a, la, b, lb)
    return x.reshape(-1, x.shape[-1]) @ y.reshape(-1, y.shape[-1]).t()


class Fragment:
    """Exact transition densities of one fragment: rho[op][(b, k)] of shape (n, n, N, ..)."""

    def __init__(self, z, n_orb):
        N, n = 2 * n_orb, next(iter(z.values())).shape[0]
        ne = {c: N_ELEC - c for c in CHARGES}
        self.N, self.n = N, n
        L0 = {c: np.sort(masks_of(n_orb, ne[c])[0]) for c in CHARGES}
        order = {c: torch.as_tensor(np.argsort(masks_of(n_orb, ne[c])[0]), device="cuda") for c in CHARGES}
        Z = {c: z[c].index_select(1, order[c]) for c in CHARGES}
        A = {c: lower(z[c], n_orb, ne[c], 0) for c in CHARGES}                        # [p, I, X]
        LA = {c: lowered(n_orb, ne[c], 0)[0] for c in CHARGES}
        B = {c: lower(A[c], n_orb, ne[c], 1) for c in CHARGES}                        # [q, r, J, X] = a_q a_r
        LB = {c: lowered(n_orb, ne[c], 1)[0] for c in CHARGES}
        self.A2 = B
        r = {op: {} for op in ("a", "c", "ca", "aa", "cc", "caa", "cca")}
        for b in CHARGES:
            for k in CHARGES:
                if b == k:
                    r["ca"][(b, k)] = pairing(A[b], LA[b], A[k], LA[k]).view(N, n, N, n).permute(1, 3, 0, 2)
                if b == k + 1:
                    r["a"][(b, k)] = pairing(Z[b], L0[b], A[k], LA[k]).view(n, N, n).permute(0, 2, 1)
                    r["caa"][(b, k)] = pairing(A[b], LA[b], B[k], LB[k]).view(N, n, N, N, n).permute(1, 4, 0, 2, 3)
                if b == k + 2:
                    r["aa"][(b, k)] = pairing(Z[b], L0[b], B[k], LB[k]).view(n, N, N, n).permute(0, 3, 1, 2)
        for (b, k), x in list(r["a"].items()):
            r["c"][(k, b)] = x.permute(1, 0, 2)
        for (b, k), x in list(r["aa"].items()):
            r["cc"][(k, b)] = x.permute(1, 0, 3, 2)
        for (b, k), x in list(r["caa"].items()):
            r["cca"][(k, b)] = x.permute(1, 0, 4, 3, 2)
        self.rho = r

    def monomer(self, c, h, V):
        """H1 of charge c: <I| sum h c+ a + sum V c+_p c+_q a_s a_r |J>."""
        N, n = self.N, self.n
        one = torch.einsum("ijpq,pq->ij", self.rho["ca"][(c, c)], h)
        B = self.A2[c]                                                                # [q, p, I, X] = a_q a_p
        W = V.permute(1, 0, 3, 2).reshape(N * N, N * N)                               # [(q p), (s r)]
        y = (W @ B.reshape(N * N, -1)).view(N * N, n, -1)
        return one + torch.einsum("aix,ajx->ij", B.reshape(N * N, n, -1), y)


def dimer_blocks(frags, h, V):
    """{(ci0, ci1, cj0, cj1): block[(i0, j0), (i1, j1)]} of H2 + H1 x 1 + 1 x H1 (order 0, S = 1, U = 0)."""
    N, n = [f.N for f in frags], [f.n for f in frags]
    sl = [slice(0, N[0]), slice(N[0], N[0] + N[1])]
    rho = [f.rho for f in frags]
    t = [h[sl[m], sl[1 - m]] for m in (0, 1)]

    def Vb(*m):
        return V[sl[m[0]], sl[m[1]], sl[m[2]], sl[m[3]]]

    P1, Pcaa, Pcc, H1 = [{}, {}], [{}, {}], [{}, {}], [{}, {}]
    for m in (0, 1):
        o = 1 - m
        for key, c in rho[m]["c"].items():
            P1[m][key] = torch.einsum("ijp,pq->ijq", c, t[m]) - 2.0 * torch.einsum(
                "ijx,xs->ijs", rho[m]["cca"][key].reshape(n[m], n[m], -1), Vb(m, m, m, o).reshape(-1, N[o]))
        for key, x in rho[m]["caa"].items():
            W = 2.0 * Vb(m, o, m, m).permute(0, 3, 2, 1).reshape(-1, N[o])            # [(p, q, r), s] = V[p, s, r, q]
            Pcaa[m][key] = torch.einsum("ijx,xs->ijs", x.reshape(n[m], n[m], -1), W)
        for key, x in rho[m]["cc"].items():                                            # P[r s] = sum V[p, q, s', r'] rho[p, q]
            Pcc[m][key] = torch.einsum("ijpq,pqsr->ijrs", x, Vb(m, m, o, o))
        for c in CHARGES:
            H1[m][c] = frags[m].monomer(c, h[sl[m], sl[m]], Vb(m, m, m, m))
    out = {}

    def mm(a, b):
        return a.reshape(n[0] * n[0], -1) @ b.reshape(n[1] * n[1], -1).t()

    eye = [torch.eye(k, **F64).reshape(-1) for k in n]
    for ci0, ci1, cj0, cj1 in itertools.product(CHARGES, repeat=4):
        if ci0 + ci1 != cj0 + cj1:
            continue
        d, k0, k1 = ci0 - cj0, (ci0, cj0), (ci1, cj1)
        s = -1.0 if (N_ELEC - cj0) % 2 else 1.0
        if d == 0:
            v = 4.0 * torch.einsum("ijpq,prqs->ijrs", rho[0]["ca"][k0], Vb(0, 1, 0, 1))
            blk = mm(v, rho[1]["ca"][k1]) + torch.outer(H1[0][ci0].reshape(-1), eye[1]) + torch.outer(eye[0], H1[1][ci1].reshape(-1))
        elif d == -1:
            blk = s * (mm(P1[0][k0], rho[1]["a"][k1]) - mm(rho[0]["c"][k0], Pcaa[1][k1]))
        elif d == 1:
            blk = s * (mm(Pcaa[0][k0], rho[1]["c"][k1]) - mm(rho[0]["a"][k0], P1[1][k1]))
        elif d == -2:
            blk = mm(Pcc[0][k0], rho[1]["aa"][k1])
        else:
            blk = mm(rho[0]["aa"][k0], Pcc[1][k1])
        out[(ci0, ci1, cj0, cj1)] = blk
    return out


def sectors_of(blocks, n):
    """{total charge: H}, rows block-major over c0 in the order of CHARGES and row-major (i0, i1) inside."""
    out = {}
    for t in dict.fromkeys(a + b for a in CHARGES for b in CHARGES):
        c0s = [c for c in CHARGES if t - c in CHARGES]
        out[t] = torch.cat([torch.cat([blocks[(a, t - a, b, t - b)].view(n, n, n, n).permute(0, 2, 1, 3).reshape(n * n, n * n)
                                       for b in c0s], 1) for a in c0s], 0)
    return out


def product_of(blocks, n):
    H = torch.zeros((3, n, 3, n, 3, n, 3, n), **F64)
    at = {c: i for i, c in enumerate(CHARGES)}
    for (a, b, c, d), blk in blocks.items():
        H[at[a], :, at[b], :, at[c], :, at[d], :] = blk.view(n, n, n, n).permute(0, 2, 1, 3)
    return H.reshape(9 * n * n, 9 * n * n)


def energy(zs, h, V, d, case):
    n = case["n_states"]
    frags = [Fragment(z, case["n_orb"]) for z in zs]
    D = d.view(3, n, 3, n)
    at = {c: i for i, c in enumerate(CHARGES)}
    E = 0.0
    for (a, b, c, e), blk in dimer_blocks(frags, h, V).items():
        x, y = D[at[a], :, at[b], :], D[at[c], :, at[e], :]
        if float(x.abs().max()) and float(y.abs().max()):
            E = E + torch.einsum("ijkl,ik,jl->", blk.view(n, n, n, n), x, y)
    return E


def gradients(zs, h, V, d, case):
    """dE/dz of both fragments and the antisymmetric spatial dE/dkappa, by reverse differentiation of E."""
    leaf = [{c: z.clone().requires_grad_(True) for c, z in zf.items()} for zf in zs]
    h, V = h.clone().requires_grad_(True), V.clone().requires_grad_(True)
    energy(leaf, h, V, d, case).backward()
    gh, gV = h.grad, V.grad
    t = h.shape[0]
    with torch.no_grad():
        G = h @ gh.t() + h.t() @ gh
        for k in range(4):
            G += V.movedim(k, 0).reshape(t, -1) @ gV.movedim(k, 0).reshape(t, -1).t()
        n = t // 2
        no = case["n_orb"]
        alpha = torch.as_tensor([2 * no * (i // no) + i % no for i in range(n)], device="cuda")
        kappa = torch.zeros((n, n), **F64)
        for so in (alpha, alpha + no):
            g = G[so][:, so]
            kappa += g - g.t()
    return [{c: torch.zeros_like(z) if z.grad is None else z.grad for c, z in zf.items()} for zf in leaf], kappa


def krylov_lowest(H, depth):
    """The lowest Ritz pair after `depth` Lanczos steps from the seeded start vector."""
    n = H.shape[0]
    m = min(depth, n)
    v = torch.randn(n, generator=torch.Generator().manual_seed(7), dtype=torch.float64)
    Q = torch.zeros((m + 1, n), **F64)
    Q[0] = (v / v.norm()).cuda()
    a, b = torch.zeros(m, dtype=torch.float64), torch.zeros(m, dtype=torch.float64)
    for j in range(m):
        w = H @ Q[j]
        a[j] = w @ Q[j]
        for _ in range(2):
            w = w - Q[:j + 1].t() @ (Q[:j + 1] @ w)
        b[j] = w.norm()
        Q[j + 1] = w / w.norm()
    T = torch.diag(a) + torch.diag(b[:m - 1], 1) + torch.diag(b[:m - 1], -1)
    e, Y = torch.linalg.eigh(T)
    return float(e[0]), Q[:m].t() @ Y[:, 0].cuda()


def exact(case, seed):
    kind, n, n_orb = case["kind"], case["n_states"], case["n_orb"]
    if kind == "trimer_hv":
        return None      # the dense operator of the product space takes far longer
    if kind == "densities":
        with torch.no_grad():
            f = Fragment(states(generator(seed), n_orb, n), n_orb)
            return {k: x.contiguous() for k, x in named_blocks(f.rho).items()}
    if kind == "hpsi":
        g = generator(seed)
        h, V = integrals(g, [n_orb])
        masks = masks_of(n_orb, N_ELEC + 1)[0]
        psi = torch.randn((n, len(masks)), generator=g, **F64)
        psi = psi / psi.norm(dim=1, keepdim=True)
        N = 2 * n_orb
        A = lower(psi, n_orb, N_ELEC + 1, 0)
        B = lower(A, n_orb, N_ELEC + 1, 1)
        Ah = (h @ A.reshape(N, -1)).view_as(A)
        Bh = (V.permute(1, 0, 3, 2).reshape(N * N, N * N) @ B.reshape(N * N, -1)).view_as(B)     # [q, p, I, X]

        def raised(Y, k):
            """sum_p c+_p Y[p]: the transpose of lower()."""
            src = masks if k == 0 else lowered(n_orb, N_ELEC + 1, k - 1)[0]
            out = torch.zeros(Y.shape[1:-1] + (len(src),), **F64)
            for p, (hit, to, sign) in enumerate(lowered(n_orb, N_ELEC + 1, k)[1]):
                out.index_add_(-1, hit, Y[p].index_select(-1, to) * sign)
            return out
        return raised(Ah, 0) + raised(raised(Bh, 1), 0)
    if kind == "orbitals":
        X, ints, sizes, sp, same = orbital_inputs(case, seed)
        M = X[sp][:, sp] * same

        def by(x, mats):
            for i, m in enumerate(mats):
                if m is not None:
                    x = torch.tensordot(x, m, dims=([i], [0])).movedim(-1, i)
            return x.contiguous()

        symm = dict(S=by(ints["S"], [M] * 2), T=by(ints["T"], [M] * 2), V=by(ints["V"], [M] * 4),
                    U=torch.stack([by(u, [M] * 2) for u in ints["U"]]))
        inv = torch.linalg.inv(symm["S"])
        it = inv.t()
        bior = dict(Sinv=inv, S=by(symm["S"], [it, None]), T=by(symm["T"], [it, None]),
                    U=torch.stack([by(u, [it, None]) for u in symm["U"]]), V=by(symm["V"], [it, it, None, None]))
        return dict(symm=symm, bior=bior)
    g, h, V, zs = inputs(case, seed)
    if kind == "gradient":
        gz, kappa = gradients(zs, h, V, ground_like(g, case), case)
        return dict(states=gz, kappa=kappa) if case["precision"] == "fp64" else gz
    with torch.no_grad():
        blocks = dimer_blocks([Fragment(z, n_orb) for z in zs], h, V)
        if kind == "hbuild":
            return product_of(blocks, n) if layout_of(case) == "product" else {str(t): H for t, H in sectors_of(blocks, n).items()}
        # iterate: the first iteration looks for the ground state in every sector
        best = None
        for t, H in sectors_of(blocks, n).items():
            e, v = krylov_lowest(H, KRYLOV)
            if best is None or e < best[0]:
                best = (e, t, v)
        del blocks
        E, t, v = best
        d = torch.zeros((3, n, 3, n), **F64)
        at = {c: i for i, c in enumerate(CHARGES)}
        for k, a in enumerate(c for c in CHARGES if t - c in CHARGES):
            d[at[a], :, at[t - a], :] = v[k * n * n:(k + 1) * n * n].view(n, n)
    gz, kappa = gradients(zs, h, V, d.reshape(-1), case)
    new = []
    for zf, gf in zip(zs, gz):
        out = {}
        for c in CHARGES:
            z, g_ = zf[c], gf[c]
            z1 = z - STEP * (g_ - 0.5 * (g_ @ z.t() + z @ g_.t()) @ z)
            e, Q = torch.linalg.eigh(z1 @ z1.t())
            out[c] = (Q * e.rsqrt()) @ Q.t() @ z1
        new.append(out)
    return dict(E=E, states=new, kappa=kappa)
