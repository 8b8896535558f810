"""Host-side plan of the FP64 grouped GEMM on the tensor cores (csrc/gemm_sliced.cu).

The tasks of one GroupedGemm launch become waves: the operands of a wave are written as digit
slices and magnitudes into one workspace (xrh_slice_grouped, every distinct operand once), then one
xrh_gemm_sliced_grouped launch runs its tasks.  Tasks whose digits exceed the workspace limit are
divided into panels.  Every table is built once and uploaded in one copy; run() only launches.
"""
import numpy as np
import torch

from . import _lib
from ._lib import SLICE_TASK_DTYPE, SLICED_SEG_DTYPE, SLICES, TASK_DTYPE, call, ptr, stream_ptr

STAGE_K = 32
BM = 128
SMS = 152
RUN_STAGES = 16384               # stages of a segment collected before a rounding (csrc/gemm_sliced.cu)
ODD_BYTES = 1024                 # marks of a tile and run
WORKSPACE_LIMIT = 1 << 30        # bytes of digits per wave
MIN_STAGES_PER_SPLIT = 8         # 256 K: an accumulating tile is not divided below this


def _bn(N):
    return 32 if N <= 32 else 64


def _tiles(t):
    return -(-t["M"] // BM) * -(-t["N"] // _bn(t["N"])) * t["batch"]


def _stages(K):
    return -(-K // STAGE_K)


def _operands(t):
    """(pointer, transposed, rows, K, ld, batch, batch stride, block) of A and B of every segment."""
    M, N, batch, bn, ops = t["M"], t["N"], t["batch"], _bn(t["N"]), []
    for (A, B, lda, ldb, K, _alpha, flags, sA, sB) in t["segs"]:
        ops.append((A, flags & 1, M, K, lda, batch, sA, BM) if sA and batch > 1 else (A, flags & 1, M, K, lda, 1, 0, BM))
        ops.append((B, flags >> 1 & 1, N, K, ldb, batch, sB, bn) if sB and batch > 1 else
                   (B, flags >> 1 & 1, N, K, ldb, 1, 0, bn))
    return ops


def _digit_bytes(op):
    _p, _tr, rows, K, _ld, batch, _st, block = op
    return 2 * (SLICES + 1) * -(-rows // block) * block * batch * _stages(K) * STAGE_K


def slice_ctas(rows, K, batch, trans, block):
    """xrh_slice_ctas of an operand with rows, K and batch > 0 (tables have hundreds of them): CTAs of the digit
    launch and of the row-maximum launch."""
    rows_p = -(-rows // block) * block
    if trans:
        return batch * (rows_p // 32) * -(-_stages(K) * STAGE_K // 64), batch * -(-rows // 32) * -(-K // 512)
    return (rows_p * batch if K > 1024 else rows_p * batch // 8), 0


def _exp_bytes(op):
    return -(-4 * op[2] * op[5] // 256) * 256


def _part(t, axis, lo, hi):
    """The part [lo, hi) of a task along its batch, M or N axis."""
    r = dict(t, segs=list(t["segs"]))
    n = hi - lo
    r["batch" if axis == "batch" else axis] = n
    for i, (A, B, lda, ldb, K, alpha, flags, sA, sB) in enumerate(r["segs"]):
        if axis == "batch":
            A, B = A + 8 * lo * sA, B + 8 * lo * sB
        elif axis == "M":
            A += 8 * lo * (1 if flags & 1 else lda)
        else:
            B += 8 * lo * (1 if flags & 2 else ldb)
        r["segs"][i] = (A, B, lda, ldb, K, alpha, flags, sA, sB)
    if axis == "batch":
        r["C"] += 8 * lo * t["sC"]
    elif t["mode"] == 2:
        row, col, diag, D = ("rowA", "colA", "diagA", "DA") if axis == "M" else ("rowB", "colB", "diagB", "DB")
        r[row] += 4 * lo
        r[col] += 4 * lo
        r[diag] += lo
        if r[D]:
            r[D] += 8 * lo
    else:
        r["C"] += 8 * lo * (t["ldc"] if axis == "M" else 1)
    return r


def _panels(t, limit):
    """The task as parts whose digits fit the limit."""
    if sum(map(_digit_bytes, set(_operands(t)))) <= limit:
        return [t]
    if t["batch"] > 1:
        axis, n, unit = "batch", t["batch"], 1
    elif t["M"] >= t["N"]:
        axis, n, unit = "M", t["M"], BM
    else:
        axis, n, unit = "N", t["N"], 64
    cut = -(-(n // 2) // unit) * unit
    if not 0 < cut < n:
        return [t]                   # one tile: its own workspace size
    return _panels(_part(t, axis, 0, cut), limit) + _panels(_part(t, axis, cut, n), limit)


def plan_waves(tasks, limit=None):
    """[(tasks, {operand: (digit offset, exponent offset)}, bytes, zeroed bytes)]: row exponents of
    transposed operands first (they are zeroed before each run), then the rest."""
    limit = WORKSPACE_LIMIT if limit is None else limit
    waves, cur, ops, size = [], [], {}, 0            # ops: {operand: (digit bytes, exponent bytes)}
    for t in (p for t in tasks for p in _panels(t, limit)):
        mine = {op: ops.get(op) or (_digit_bytes(op), _exp_bytes(op)) for op in _operands(t)}
        extra = sum(sum(b) for op, b in mine.items() if op not in ops)
        if cur and size + extra > limit:
            waves.append((cur, ops))
            cur, ops, size = [], {}, 0
            extra = sum(map(sum, mine.values()))
        cur.append(t)
        ops.update(mine)
        size += extra
    if cur:
        waves.append((cur, ops))
    out = []
    for cur, ops in waves:
        off, at = 0, {}
        for op in sorted(ops, key=lambda o: not o[1]):
            at[op] = off
            off += ops[op][1]
        zeroed = sum(b for op, (_d, b) in ops.items() if op[1])
        off = -(-off // 1024) * 1024
        place = {}
        for op, (b, _e) in ops.items():
            place[op] = (off, at[op])
            off += b
        out.append((cur, place, off, zeroed))
    return out


def split_factors(tasks):
    """Split-K factor of every task of a wave: accumulating tasks are divided until the launch has
    about four tiles per SM, none below MIN_STAGES_PER_SPLIT stages; stored results are not."""
    stages = [sum(_stages(s[4]) for s in t["segs"]) for t in tasks]
    work = sum(_tiles(t) * n for t, n in zip(tasks, stages))
    per = max(MIN_STAGES_PER_SPLIT, -(-work // (4 * SMS)))
    return [max(1, -(-n // per)) if t["mode"] == 1 else 1 for t, n in zip(tasks, stages)]


# the fields of a task that only the scatter epilogue has
_MAPS = ("rowA", "colA", "rowB", "colB", "DA", "DB", "diagA", "diagB")
_NO_MAPS = (0,) * len(_MAPS)
assert TASK_DTYPE.names == ("M", "N", "seg_begin", "seg_count", "mode", "splitk", "tile_begin", "C", "ldc") + _MAPS + ("batch", "sC")
assert SLICE_TASK_DTYPE.names == ("src", "digits", "exps", "rows", "K", "ld", "Kp", "batch", "sbatch", "trans", "block", "cta_begin",
                                  "max_begin")
assert SLICED_SEG_DTYPE.names == ("digA", "digB", "stages", "rA", "rB", "eA", "eB", "A", "B", "lda", "ldb", "K", "flags", "sA", "sB",
                                  "alpha")


class Workspace:
    """Device memory for the digits of launches that run one after the other (those of a plan and its
    reverse pass, in the order of one stream).  They join when they are planned; allocate(), before the
    first run, gives those that have joined since the last call one buffer as large as the largest needs,
    an earlier one where it is large enough."""

    def __init__(self, device):
        self.device, self.buf, self.waiting = device, None, []

    def join(self, g):
        self.waiting.append(g)

    def allocate(self):
        need = max((g.size for g in self.waiting), default=0)
        if need and (self.buf is None or self.buf.numel() < need):
            self.buf = torch.empty(need, dtype=torch.uint8, device=self.device)
        for g in self.waiting:
            g.bind(self.buf)
        self.waiting = []


class SlicedGemm:
    """tasks: dicts with M, N, mode, C, ldc, batch, sC, mode 2's maps (device addresses) and segs
    [(A, B, lda, ldb, K, alpha, flags, sA, sB)] (addresses).  status: the int32 device word that a
    launch sets when a bounded wait gave up (several plans may share one).  work: a Workspace, whose owner
    allocates it; without one the launch has its own."""

    def __init__(self, tasks, device, status=None, work=None):
        self.device, self.tables = device, None
        waves = plan_waves(tasks)
        splits = [split_factors(w[0]) for w in waves]
        # behind the digits of a wave the marks of its tiles (a range per task) and the list of marked tiles
        tiles_of = [[_tiles(t) * k for t, k in zip(w[0], sk)] for w, sk in zip(waves, splits)]
        runs_of = [[sum(-(-_stages(s[4]) // RUN_STAGES) for s in t["segs"]) for t in w[0]] for w in waves]
        marks = [[n * r for n, r in zip(*x)] for x in zip(tiles_of, runs_of)]
        size_of = lambda w, m, n: -(-w[2] // 1024) * 1024 + sum(m) * ODD_BYTES + 4 * (1 + sum(n))
        self.size = max(map(size_of, waves, marks, tiles_of)) + 1024
        self._plan = list(zip(waves, splits, tiles_of, runs_of, marks))
        self.status = _lib.status_word(device) if status is None else status
        if work is None:
            work = Workspace(device)
            work.join(self)
            work.allocate()
        else:
            work.join(self)

    def bind(self, work):
        """Task tables over the workspace `work` (a byte tensor), uploaded in one copy."""
        self.work = work
        self.base = base = -(-work.data_ptr() // 1024) * 1024
        blob, self.waves = bytearray(), []

        def put(raw):
            at = len(blob)
            blob.extend(raw)
            blob.extend(bytes(-len(blob) % 128))
            return at

        for (cur, place, size, zeroed), splitk, count, runs, mark in self._plan:
            # rows as tuples, then one conversion per table
            st, ctas, max_ctas = [], 0, 0
            # transposed operands last: their tasks own the CTAs of the row-maximum launch
            for op in sorted(place, key=lambda o: o[1]):
                p, tr, rows, K, ld, batch, sb, block = op
                st.append((p, base + place[op][0], base + place[op][1], rows, K, ld, _stages(K) * STAGE_K, batch, sb, tr,
                           block, ctas, max_ctas))
                c, m = slice_ctas(rows, K, batch, tr, block)
                ctas, max_ctas = ctas + c, max_ctas + m
            gt, gs, tiles = [], [], 0
            for t, sk, n in zip(cur, splitk, count):
                gt.append((t["M"], t["N"], len(gs), len(t["segs"]), t["mode"], sk, tiles, t["C"], t["ldc"],
                           *([t[n] for n in _MAPS] if t["mode"] == 2 else _NO_MAPS), t["batch"], t["sC"]))
                tiles += n
                ops = _operands(t)
                for (A, B, lda, ldb, K, alpha, flags, sA, sB), a, b in zip(t["segs"], ops[::2], ops[1::2]):
                    (dA, eA), (dB, eB) = place[a], place[b]
                    gs.append((base + dA, base + dB, _stages(K), a[2] if a[5] > 1 else 0, b[2] if b[5] > 1 else 0, base + eA,
                               base + eB, A, B, lda, ldb, K, flags, sA, sB, alpha))
            st, gt, gs = (np.array(rows, dtype=dtype)
                          for rows, dtype in ((st, SLICE_TASK_DTYPE), (gt, TASK_DTYPE), (gs, SLICED_SEG_DTYPE)))
            odd = np.stack([np.cumsum([0] + mark[:-1]), runs], axis=1).astype(np.int64)
            self.waves.append((put(st.tobytes()), len(st), ctas, max_ctas, zeroed, put(gt.tobytes()), len(gt), tiles,
                               put(gs.tobytes()), put(odd.tobytes()), base + -(-size // 1024) * 1024,
                               base + -(-size // 1024) * 1024 + sum(mark) * ODD_BYTES))
        self.tables = torch.frombuffer(blob, dtype=torch.uint8).to(self.device)
        self._plan = None

    def run(self, stream=None):
        if self.tables is None:
            raise RuntimeError("the workspace of this launch has not been allocated")
        s = stream_ptr(stream)
        t = self.tables.data_ptr()
        for st, n_s, ctas, max_ctas, zeroed, gt, n_t, tiles, gs, odd, bits, marked in self.waves:
            if zeroed:
                call("xrh_zero", self.base, zeroed, s)
            call("xrh_slice_grouped", t + st, n_s, ctas, max_ctas, marked, s)
            call("xrh_gemm_sliced_grouped", t + gt, n_t, tiles, t + gs, t + odd, bits, marked, ptr(self.status), s)

    def check(self):
        """Raise if a bounded device wait gave up (synchronises)."""
        _lib.check_status(self.status, "sliced FP64 GEMM")
