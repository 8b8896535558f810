"""FP32 densities of blocks of many states: the bits of the general kernel (xrh_density_accumulate_f32)."""
import ctypes
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _list(rng, K, n_conf_b, n_conf_k, counts):
    idx_ptr = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    n = int(idx_ptr[-1])
    sign = np.ones(n, dtype=np.int8)
    n_pos = np.zeros(K, dtype=np.int64)
    for i, c in enumerate(counts):
        n_pos[i] = rng.choice([0, c, rng.integers(0, c + 1)])
        sign[idx_ptr[i] + n_pos[i]:idx_ptr[i + 1]] = -1
    dev = lambda x: torch.as_tensor(x).cuda()
    return [dev(x) for x in (idx_ptr, n_pos, rng.integers(0, n_conf_b, n).astype(np.int32),
                             rng.integers(0, n_conf_k, n).astype(np.int32), sign)]


@pytest.mark.parametrize("nb,nk", [(45, 46), (60, 60), (64, 64), (65, 33), (33, 67), (130, 17), (100, 81)])
@pytest.mark.parametrize("splits", [1, 3])
def test_same_bits_as_the_general_kernel(nb, nk, splits):
    from qodeapplications_gb300 import _lib
    from qodeapplications_gb300._lib import call, ptr, stream_ptr
    rng = np.random.default_rng(1000 * nb + nk)
    counts = np.array([0, 1, 3, 31, 32, 33, 63, 64, 65, 97, 128, 129, 500], dtype=np.int64)
    K = len(counts)
    idx_ptr, n_pos, P, Q, sign = _list(rng, K, 90, 70, counts)
    pad = lambda n: (n + 3) // 4 * 4
    zb, zk = torch.zeros(90, pad(nb), device="cuda"), torch.zeros(70, pad(nk), device="cuda")
    zb[:, :nb], zk[:, :nk] = torch.randn(90, nb, device="cuda"), torch.randn(70, nk, device="cuda")
    ref = torch.zeros(K, nb, nk, dtype=torch.float64, device="cuda")
    out = torch.zeros_like(ref) if splits > 1 else torch.full_like(ref, float("nan"))
    call("xrh_density_accumulate_f32", K, splits, ptr(idx_ptr), ptr(P), ptr(Q), ptr(sign), ptr(zb), nb, ptr(zk), nk,
         ptr(ref), stream_ptr())
    tasks = np.zeros(2, dtype=_lib.DENS_WIDE_TASK_DTYPE)
    other = torch.full_like(ref, float("nan")) if splits == 1 else torch.zeros_like(ref)
    ctas = K * splits * -(-nb // 64) * -(-nk // 64)
    for t, dst, begin in zip(tasks, (out, other), (0, ctas)):
        t["idx_ptr"], t["n_pos"], t["P"], t["Q"] = idx_ptr.data_ptr(), n_pos.data_ptr(), P.data_ptr(), Q.data_ptr()
        t["zb32"], t["zk32"], t["rhoT"] = zb.data_ptr(), zk.data_ptr(), dst.data_ptr()
        t["K"], t["nb"], t["nk"], t["splits"], t["cta_begin"] = K, nb, nk, splits, begin
    tab = torch.from_numpy(tasks.view(np.uint8).copy()).cuda()
    call("xrh_density_accumulate_f32_wide", ptr(tab), 2, 2 * ctas, stream_ptr())
    if splits == 1:
        assert torch.equal(out, ref) and torch.equal(other, ref)
    else:                                              # three FP64 terms in any order: two roundings apart
        for x in (out, other):
            assert bool(((x - ref).abs() <= 4 * 2.0 ** -53 * 500 * 16.0).all())


def test_builder_route(monkeypatch):
    """The FP32 builder sends such blocks there, and only those."""
    from perf import cases
    narrow = cases.prepare(dict(kind="densities", precision="fp32", n_orb=6, n_states=44), 3)["builder"]
    wide = cases.prepare(dict(kind="densities", precision="fp32", n_orb=6, n_states=46), 3)["builder"]
    assert narrow._wide is None and narrow._n_dens_tasks > 0
    assert wide._wide is not None and wide._n_dens_tasks == 0
