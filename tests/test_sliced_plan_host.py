"""Host arithmetic of the digit plans against the library's."""
import pytest

pytest.importorskip("torch")


@pytest.mark.parametrize("block", [32, 64, 128])
def test_slice_ctas(block):
    from qodeapplications_gb300 import _lib, sliced
    L = _lib.lib()
    for rows in (1, 31, 32, 33, 127, 128, 129, 3600):
        for K in (1, 31, 32, 33, 511, 512, 513, 1024, 1025, 21952):
            for batch in (1, 7):
                for trans in (0, 1):
                    want = tuple(L.xrh_slice_ctas(rows, K, batch, trans, block, p) for p in (0, 1))
                    assert sliced.slice_ctas(rows, K, batch, trans, block) == want


def test_a_launch_that_runs_once():
    """Short launches of many tasks that run one time stay on the CUDA cores; long ones do not."""
    from qodeapplications_gb300 import gemm

    def plan(n, M, K, once):
        g = gemm.GroupedGemm(device="cpu")
        g._segs = [(0, 0, K, K, K, 1.0, 0, 0, 0)] * n
        g._tasks = [dict(M=M, N=M, seg_begin=i, seg_count=1, mode=0, splitk=1, C=0, ldc=M, batch=1, sC=0) for i in range(n)]
        return len(g._sliced_tasks(once))
    assert plan(100, 20, 64, False) == 100 and plan(100, 20, 64, True) == 0
    assert plan(3, 3000, 784, True) == 3
    assert plan(1, 64, 1000, True) == 1
