"""A host interpreter of the spread solve's packets (the semantics of spread_solve.cuh), for checking
layouts on the CPU: every right-hand side is one lane. It also checks what the kernel relies on: that a
packet never straddles a page, that a slot is written before it is read, that a row's slots are apart, and
that each partial row is written once."""
import numpy as np

ROWS4, ROWS1, MORE, MOVE, PAGE_END, END = range(6)
SELF, LOAD0, STORE0, CARRY, LOAD1, STORE1 = 1, 2, 4, 8, 16, 32
PAGE = 2048


def sweep(lay, task, back, work, out, partial, top, written):
    n, vb = lay["n"], lay["value_bytes"]
    cplx = lay["dtype"] == np.complex128
    ft = {(False, 8): np.float64, (False, 4): np.float32, (True, 16): np.complex128, (True, 8): np.complex64}[cplx, vb]
    row_bytes = 64 if vb == 16 else 32
    pair_bytes = 48 if vb == 16 else 32 if vb == 8 else 16
    first, count = lay["bwd_page" if back else "fwd_page"][2 * task:2 * task + 2]
    blob = lay["blob"][first * PAGE:(first + count) * PAGE]
    r0, r1 = lay["task_row"][task:task + 2]
    lanes = work.shape[1]
    live = [None] * lay["slots"]
    zero = np.zeros(lanes, work.dtype)
    at, row = 0, (r1 - 1 if back else r0)
    z, carry = zero, zero

    def word(o, k=1):
        return blob[o:o + 4 * k].view(np.uint32).astype(np.int64)

    def value(o):
        return blob[o:o + vb].view(ft)[0]

    def read(s):
        assert live[s] is not None, "a slot read before it is written"
        return live[s]

    def further(o):
        nonlocal z
        w = int(word(o + 2 * vb)[0])
        t0, t1, f = w & 0xff, w >> 8 & 0xff, w >> 16
        second = f & (LOAD1 if back else STORE1)
        assert not second or t0 != t1, "a pair's slots are one"
        if back:
            z = z - value(o) * read(t0)
            if second:
                z = z - value(o + vb) * read(t1)
        else:
            a = -value(o) * z + (read(t0) if f & LOAD0 else 0)
            b = -value(o + vb) * z + (read(t1) if f & LOAD1 else 0) if second else None
            live[t0] = a
            if second:
                live[t1] = b

    while True:
        kind, size, number = (int(v) for v in word(at, 3))
        assert at % 16 == 0 and at // PAGE == (at + size - 1) // PAGE, "a packet across pages"
        if kind == PAGE_END:
            at = (at // PAGE + 1) * PAGE
            continue
        if kind == END:
            break
        if kind in (ROWS4, ROWS1):
            k = 4 if kind == ROWS4 else 1
            assert number == k
            more = at + 16 + k * row_bytes
            for q in range(k):
                o = at + 16 + q * row_bytes
                slots, flags = (int(v) for v in word(o + 3 * vb, 2))
                f, pairs = flags & 0xff, flags >> 8
                s0, t0, t1, dinv = slots & 0xff, slots >> 8 & 0xff, slots >> 16, value(o + 2 * vb)
                assert r0 <= row < r1, "a row of another task"
                if not back:
                    if f & SELF:
                        carry = read(s0)
                        live[s0] = None
                    x0 = read(t0) if f & LOAD0 else zero
                    x1 = read(t1) if f & LOAD1 else zero
                    if f & LOAD0 and not f & STORE0:
                        live[t0] = None  # what waited for the next row goes on in the register
                    z = (work[row] + carry) * dinv
                    out[row] = z
                    carry = x0 - value(o) * z
                    if f & STORE0:
                        live[t0] = carry
                    if f & STORE1:
                        assert not f & STORE0 or t0 != t1
                        live[t1] = x1 - value(o + vb) * z
                    if not f & CARRY:
                        carry = zero
                else:
                    z = work[row] + z if k == 1 else work[row]
                    if f & (LOAD0 | CARRY):
                        z = z - value(o) * (read(t0) if f & LOAD0 else carry)
                    if f & LOAD1:
                        z = z - value(o + vb) * read(t1)
                for _ in range(pairs):
                    further(more)
                    more += pair_bytes
                if back:
                    carry = z * dinv
                    if f & SELF:
                        live[s0] = carry
                    out[row] = carry
                row += -1 if back else 1
            assert more <= at + size
            if back:
                z = zero
        elif kind == MORE:
            for k in range(number):
                further(at + 16 + k * pair_bytes)
        else:
            assert kind == MOVE
            moves = word(at + 16, 2 * number).reshape(-1, 2)
            for index, s in moves:
                if back:
                    live[s] = top[index]
                else:
                    assert not written[index], "a partial row written twice"
                    written[index] = True
                    partial[index] = read(s)
                    live[s] = None
        at += size
    assert row == (r0 - 1 if back else r1), "rows left over"


def triangle(t, spec, lower):
    ptr, col, val, dinv = spec
    m = np.diag(1.0 / dinv) if t else np.zeros((0, 0))
    for i in range(t):
        m[i, col[ptr[i]:ptr[i + 1]]] = val[ptr[i]:ptr[i + 1]]
    return m


def run(lay, rhs):
    """Solves the rows of `rhs` (count x n, natural order) through the packets; the top by substitution."""
    n, t = lay["n"], lay["top"]
    rhs = np.atleast_2d(np.asarray(rhs, lay["dtype"]))
    assert sorted(lay["in_pos"]) == list(range(n)) and lay["task_row"][-1] == n - t
    work = np.zeros((n, rhs.shape[0]), lay["dtype"])
    work[lay["in_pos"]] = rhs.T
    partial = np.zeros((lay["partials"], rhs.shape[0]), lay["dtype"])
    written = np.zeros(lay["partials"], bool)
    for task in range(lay["tasks"]):
        sweep(lay, task, False, work, work, partial, None, written)
    assert written.all(), "a partial row not written"
    x = work[n - t:].copy()
    for k in range(t):
        x[k] += partial[lay["part_ptr"][k]:lay["part_ptr"][k + 1]].sum(axis=0)
    ptr, col, val, dinv = lay["lower"]
    for k in range(t):
        some = slice(ptr[k], ptr[k + 1])
        x[k] = (x[k] - val[some] @ x[col[some]]) * dinv[k]
    ptr, col, val, dinv = lay["upper"]
    for k in range(t - 1, -1, -1):
        some = slice(ptr[k], ptr[k + 1])
        x[k] = (x[k] - val[some] @ x[col[some]]) * dinv[k]
    work[n - t:] = x
    for task in range(lay["tasks"]):
        sweep(lay, task, True, work, work, partial, x, written)
    return work[lay["out_pos"]].T.copy()
