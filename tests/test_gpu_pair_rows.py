"""The pair scatter by destination against the scatter by entries: the same copies and signs."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_orb,n_el", [(3, 2), (5, 4), (6, 5)])
@pytest.mark.parametrize("n", [1, 15, 16, 17, 60])
@pytest.mark.parametrize("part", [1.0, 0.05])
def test_same_positions_and_signs(n_orb, n_el, n, part):
    from itertools import combinations
    from qodeapplications_gb300 import _lib
    from qodeapplications_gb300.densities import build_pair_list, pair_offsets
    rng = np.random.default_rng(n_orb * 100 + n)
    masks = np.array([sum(1 << i for i in c) for c in combinations(range(2 * n_orb), n_el)], dtype=np.uint64)
    masks = masks[np.sort(rng.permutation(len(masks))[:max(2, int(part * len(masks)))])]
    pl = build_pair_list(masks, n_orb)
    for k in ("X", "sign", "xptr"):
        pl[k + "_dev"] = torch.from_numpy(pl[k]).cuda()
    off, stride = (torch.from_numpy(x).cuda() for x in pair_offsets(pl, n))
    zT = torch.randn(len(masks), n, dtype=torch.float64, device="cuda")
    dense = 4 * len(pl["X"]) >= pl["L"]
    assert n_orb == 3 or dense == (part == 1.0)        # both sides of the rule
    ref = torch.zeros(n * pl["L"], dtype=torch.float64, device="cuda")
    _lib.call("xrh_pair_scatter", len(pl["X"]), _lib.ptr(pl["X_dev"]), _lib.ptr(off), _lib.ptr(pl["sign_dev"]),
              _lib.ptr(zT), n, _lib.ptr(stride), _lib.ptr(ref), _lib.stream_ptr())
    out = torch.full_like(ref, float("nan")) if dense else torch.zeros_like(ref)
    launch = _lib.PairLaunch([(pl, off, stride, zT, out, n)], False, "cuda")
    assert (launch.rows is not None) == dense
    launch.run()
    assert torch.equal(out, ref)
