"""Host plan of the sliced FP64 GEMM: panels of a task that exceeds the workspace partition it
exactly (addresses, maps and batches), shown by executing the parts with NumPy."""
import ctypes

import numpy as np
import pytest

pytest.importorskip("torch")


def _read(p, n, dtype):
    return np.frombuffer((ctypes.c_char * (n * np.dtype(dtype).itemsize)).from_address(int(p)), dtype=dtype)


def _write(p, v):
    np.frombuffer((ctypes.c_char * 8).from_address(int(p)), dtype=np.float64)[0] += v


def _execute(t):
    """C += sum of segments, element by element from the task's addresses."""
    for b in range(t["batch"]):
        acc = np.zeros((t["M"], t["N"]))
        for (A, B, lda, ldb, K, alpha, flags, sA, sB) in t["segs"]:
            def op(p, rows, ld, tr):
                n = (K - 1) * ld + rows if tr else (rows - 1) * ld + K
                x = _read(p, n, np.float64)
                st = (8, 8 * ld) if tr else (8 * ld, 8)
                return np.lib.stride_tricks.as_strided(x, (rows, K), st)
            acc += alpha * op(A + 8 * b * sA, t["M"], lda, flags & 1) @ op(B + 8 * b * sB, t["N"], ldb, flags & 2).T
        for m in range(t["M"]):
            for n in range(t["N"]):
                if t["mode"] == 2:
                    r = _read(t["rowA"], t["M"], np.int32)[m] + _read(t["rowB"], t["N"], np.int32)[n]
                    c = _read(t["colA"], t["M"], np.int32)[m] + _read(t["colB"], t["N"], np.int32)[n]
                    off = int(r) * t["ldc"] + int(c)
                else:
                    off = b * t["sC"] + m * t["ldc"] + n
                _write(t["C"] + 8 * off, acc[m, n])


@pytest.mark.parametrize("flags,batch,mode", [(0, 1, 0), (3, 3, 1), (1, 1, 2), (2, 4, 0)])
def test_panels_partition_the_task(flags, batch, mode):
    from qodeapplications_gb300 import sliced
    rng = np.random.default_rng(1)
    M, N, K = 300, 200, 20
    A, B = rng.standard_normal((batch, M, K)), rng.standard_normal((N, K))
    if flags & 1:
        A = np.ascontiguousarray(A.transpose(0, 2, 1))
    if flags & 2:
        B = np.ascontiguousarray(B.T)
    C = np.zeros((batch, M, N))
    t = dict(M=M, N=N, mode=mode, C=C.ctypes.data, ldc=N, batch=batch, sC=M * N,
             segs=[(A.ctypes.data, B.ctypes.data, M if flags & 1 else K, N if flags & 2 else K, K, -2.0, flags, M * K, 0)])
    keep = []
    if mode == 2:
        for name, v in (("rowA", rng.permutation(M)), ("colA", np.zeros(M)), ("rowB", np.zeros(N)), ("colB", np.arange(N))):
            keep.append(v.astype(np.int32))
            t[name] = keep[-1].ctypes.data
        for name, n in (("diagA", M), ("diagB", N)):
            keep.append(np.zeros(n, dtype=np.uint8))
            t[name] = keep[-1].ctypes.data
        t["DA"] = t["DB"] = 0
    waves = sliced.plan_waves([t], limit=120000)
    parts = [p for w in waves for p in w[0]]
    assert len(parts) > 1
    for cur, place, size, zeroed in waves:
        ops = sorted((d, d + sliced._digit_bytes(o)) for o, (d, _e) in place.items())
        ops += sorted((e, e + sliced._exp_bytes(o)) for o, (_d, e) in place.items())
        ops.sort()
        assert all(a[1] <= b[0] for a, b in zip(ops, ops[1:])) and ops[-1][1] <= size
        assert all(e < zeroed for o, (_d, e) in place.items() if o[1])
    for p in parts:
        _execute(p)
    a = A.transpose(0, 2, 1) if flags & 1 else A
    want = -2.0 * a @ (B if flags & 2 else B.T)
    if mode == 2:
        out = np.empty_like(want)
        out[:, keep[0]] = want
        want = out
    np.testing.assert_allclose(C, want, rtol=0, atol=1e-12)
