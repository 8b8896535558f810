"""Orbital transformations of the fragment-blocked integrals on the device.

Replaces the integral re-transformation of the reference's orbital optimizer and its
biorthogonalisation:

* StateSpaceOptimizer/orbital_solver.py:323-413 (transform_ints): the symmetric integrals in
  the new orbitals, every index transformed by the orbital transformation U
  (ket_transformed then bra_transformed with U^T as qode's fragments module applies them),
  then the biorthogonal integrals, the bra indices transformed by S^-1 of the new overlap;
* hermitian-XRCC/get_ints.py:62-66 (direct_Sinv) and :142-143 (bra_transformed(Sinv, ...)).

Here the integrals are supersystem spin-orbital arrays (alpha block then beta block inside
every fragment): S, T (n x n), U (n_frag x n x n), V (n^4), on the device in FP64.  Every index
transformation is one pass of this library's FP64 grouped GEMM kernel:

    pass(X, M):   Y[rest, p] = sum_a X[a, rest] M[a, p]

which transforms the leading index and moves it to the back, so k passes over a k-index
array transform every index once and end in the original index order.  The small matrices
(S^-1, exp(kappa), spin blocking) are one-CTA kernels (csrc/smallmat.cu).

Conventions: X'[p, q, ...] = sum_{a, b, ...} M[a, p] M[b, q] ... X[a, b, ...] for the symmetric
transformation (M = U); the biorthogonal integrals contract S^-1 into the bra indices --
T_b[p, q] = sum_a Sinv[p, a] T[a, q], V_b[p, q, r, s] = sum_ab Sinv[p, a] Sinv[q, b] V[a, b, r, s]
(the first two indices of V_pqrs are the creators, H = sum V_pqrs c+_p c+_q a_s a_r) -- so that
the biorthogonal overlap Sinv S is the identity.
"""
import numpy as np
import torch

from . import _lib
from ._lib import call, ptr, stream_ptr
from .gemm import GroupedGemm
from .synthetic import spin_orbital_spatial_index


def _spin_of(frag_sizes):
    return np.concatenate([np.repeat([0, 1], nf) for nf in frag_sizes]).astype(np.int8)


def _spin_index_tensors(frag_sizes, device):
    """(spatial index int32, spin int8) device arrays of the spin orbitals.  The caller keeps
    both alive until the launch that reads them is enqueued: a temporary freed before the
    call returns its block to the caching allocator, and the next allocation may take it."""
    sidx = spin_orbital_spatial_index(frag_sizes)
    return (torch.as_tensor(np.array(sidx, dtype=np.int32), device=device),
            torch.as_tensor(_spin_of(frag_sizes), device=device))


def _spin_block(src, ld_src, frag_sizes, out):
    """out = spin-orbital form of the spatial matrix src (xrh_spin_block)."""
    sidx_t, spin_t = _spin_index_tensors(frag_sizes, src.device)
    call("xrh_spin_block", sidx_t.numel(), ptr(sidx_t), ptr(spin_t), ptr(src), ld_src, ptr(out), out.shape[1],
         stream_ptr())
    return out


def _transform_all(items, status=None):
    """[(X, batch, mats)] -> transformed arrays: every index of the batch n^k arrays X transformed by
    its matrix (None for the identity).  The i-th passes of all arrays are one grouped GEMM,
        Y[rest, p] = sum_a X[a, rest] M[a, p];
    trailing identities only turn the index order back, one transpose instead of a pass each.  The
    caller checks `status` (_lib.status_word) where it waits for the device; without one it is checked here."""
    own = status is None
    cur, todo = [], []
    if own and items:
        status = _lib.status_word(items[0][0].device)
    for X, batch, mats in items:
        n = X.shape[0 if batch is None else 1]
        if n == 0 or batch == 0:
            raise RuntimeError("an integral array without elements")
        last = max((i + 1 for i, M in enumerate(mats) if M is not None), default=0)
        cur.append(X.contiguous())
        todo.append((n, batch or 1, len(mats) - last,
                     [torch.eye(n, dtype=torch.float64, device=X.device) if M is None else M.contiguous() for M in mats[:last]]))
    for step in range(max((len(t[3]) for t in todo), default=0)):
        g = GroupedGemm(cur[0].device)
        for i, (n, batch, _turn, mats) in enumerate(todo):
            if step >= len(mats):
                continue
            X, nxt = cur[i], torch.empty_like(cur[i])
            size = X.numel() // batch
            # A = X stored [k = a][m = rest] (flag bit 0), B = M stored [k = a][n = p] (flag bit 1)
            g.add(size // n, n, [(X, size // n, mats[step], n, n, 1.0, 3, size if batch > 1 else 0, 0)], nxt, n, mode=0,
                  batch=batch, sC=size if batch > 1 else 0)
            cur[i] = nxt
        g.finalize(status=status).run()
    turns = []
    for i, (n, batch, turn, _mats) in enumerate(todo):
        if turn:
            src, out = cur[i].view(batch, -1), torch.empty_like(cur[i])
            turns += [(x, y, n ** turn, x.numel() // n ** turn) for x, y in zip(src, out.view(batch, -1))]
            cur[i] = out
    if turns:
        _lib.Transposes(turns, cur[0].device).run()
    if own and cur:
        _lib.check_status(status, "integral transformation")
    return cur


def transform_indices(X, mats):
    """Every index of the n^k array X transformed by its matrix (mats[i] for index i, None
    for the identity): X'[p, q, ...] = sum M0[a, p] M1[b, q] ... X[a, b, ...]."""
    return _transform_all([(X, None, mats)])[0]


def transform_integrals(M, ints, status=None):
    """The integrals {S, T, U, V} (any subset) in the orbitals transformed by M (n x n):
    every index transformed (the symmetric integrals of orbital_solver.transform_ints)."""
    return _transform_dict({key: (X, [M] * (X.dim() - (key == "U"))) for key, X in ints.items() if X is not None},
                           ints, status)


def _transform_dict(jobs, like, status=None):
    """{key: (array, mats)} transformed together (U: one matrix per fragment), None for the other keys of like."""
    done = dict(zip(jobs, _transform_all([(X, X.shape[0] if key == "U" else None, mats)
                                          for key, (X, mats) in jobs.items()], status)))
    return {key: done.get(key) for key in like}


def inverse_spin_free(S, frag_sizes):
    """inverse_spin_free_launch, checked (synchronises)."""
    out, status = inverse_spin_free_launch(S, frag_sizes)
    _check_inverse(status)
    return out


def _check_inverse(status):
    if int(status.item()) != 0:
        raise _lib.XRHError("overlap matrix is singular")


def inverse_spin_free_launch(S, frag_sizes):
    """S^-1 of a spin-free spin-orbital overlap (alpha and beta blocks equal, no alpha-beta
    coupling): the inverse of its alpha-alpha block (spatial, <= 64 orbitals), spin-blocked."""
    dev = S.device
    sidx = spin_orbital_spatial_index(frag_sizes)
    spin = _spin_of(frag_sizes)
    n_sp = sum(frag_sizes)
    # the alpha spin orbitals by their spatial index
    alpha = sorted((a for a in range(len(sidx)) if spin[a] == 0), key=lambda a: sidx[a])
    alpha = torch.as_tensor(np.array(alpha, dtype=np.int32), device=dev)
    s_sp = torch.empty((n_sp, n_sp), dtype=torch.float64, device=dev)
    inv_sp = torch.empty_like(s_sp)
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    s = stream_ptr()
    call("xrh_gather_submatrix", n_sp, ptr(alpha), ptr(S), S.shape[1], ptr(s_sp), n_sp, s)
    call("xrh_inverse_small", n_sp, ptr(s_sp), n_sp, ptr(inv_sp), n_sp, ptr(status), s)
    return _spin_block(inv_sp, n_sp, frag_sizes, torch.empty_like(S)), status


def biorthogonal_integrals(symm, frag_sizes, status=None):
    """The biorthogonal integrals from the symmetric ones (get_ints.py:62-66,142-143): S^-1
    of symm['S'] contracted into the bra indices of T, U and V.  Returns a dict with S (the
    biorthogonal overlap, the identity up to rounding), T, U, V and Sinv."""
    Sinv, singular = inverse_spin_free_launch(symm["S"], frag_sizes)
    SinvT = Sinv.t().contiguous()        # pass matrix: M[a, p] = Sinv[p, a]
    if status is None:
        status = _lib.status_word(Sinv.device)
    jobs = {"S": (symm["S"], [SinvT, None]), "T": (symm["T"], [SinvT, None])}
    if symm.get("U") is not None:
        jobs["U"] = (symm["U"], [SinvT, None])
    jobs["V"] = (symm["V"], [SinvT, SinvT, None, None])
    out = {"Sinv": Sinv, **_transform_dict(jobs, jobs, status)}
    _check_inverse(singular)             # one synchronisation, behind everything that was enqueued
    _lib.check_status(status, "integral transformation")
    return out


def rotation_matrix(kappa, frag_sizes):
    """Spin-orbital R = exp(kappa) for antisymmetric spatial kappa (the same rotation for both
    spins), computed by xrh_expm_small and spin-blocked by xrh_spin_block."""
    kappa = kappa.contiguous()
    dev = kappa.device
    n_sp = kappa.shape[0]
    R_sp = torch.empty_like(kappa)
    s = stream_ptr()
    call("xrh_expm_small", n_sp, ptr(kappa), n_sp, ptr(R_sp), n_sp, s)
    n_so = 2 * sum(frag_sizes)
    return _spin_block(R_sp, n_sp, frag_sizes, torch.empty((n_so, n_so), dtype=torch.float64, device=dev))


def transform_ints(U_sp, ints, frag_sizes):
    """orbital_solver.transform_ints (StateSpaceOptimizer/orbital_solver.py:323-413) for
    supersystem arrays: U_sp is the spatial orbital transformation (n_sp x n_sp, e.g. the
    first-order I + s x of :431 or exp(kappa)), ints a dict {S, T, U, V} of spin-orbital
    arrays.  Returns (symmetric, biorthogonal) integral dicts."""
    dev = ints["T"].device
    n_so = 2 * sum(frag_sizes)
    Usp = torch.as_tensor(U_sp, dtype=torch.float64, device=dev).contiguous()
    M = _spin_block(Usp, Usp.shape[0], frag_sizes, torch.empty((n_so, n_so), dtype=torch.float64, device=dev))
    status = _lib.status_word(dev)
    symm = transform_integrals(M, ints, status)
    bior = biorthogonal_integrals(symm, frag_sizes, status)
    return symm, bior
