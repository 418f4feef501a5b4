"""The halo exchange and the sums of the cluster kernels (csrc/pf_mg_coarse.cuh)
under every order in which warps and messages can run.

The steps of a half-sweep, of the prolongation and of the CG's product are read
from the source and run by a model of two neighbouring CTAs.  In each, one warp
owns the boundary plane (it reads the halo and sends), another one holds the
thread that announces the bytes an exchange brings, and a message lands at any
time after it was sent.  An mbarrier's phase completes when its one arrival and
all announced bytes have come, whichever exchange they belong to.  Checked: no
order ends in a wait that never completes, and a read of a halo plane finds the
neighbour's last exchange of that colour."""

import os
import re

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                   "implementation-of-adaptive-phase-field-flip_b200", "csrc", "pf_mg_coarse.cuh")


def body(signature):
    """The braced block that follows the first text matching `signature`."""
    text = re.sub(r"//[^\n]*", "", open(SRC).read())
    i = text.index("{", re.search(signature, text).end())
    depth, j = 0, i
    while True:
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        j += 1
        if depth == 0:
            return text[i:j]


def steps(code, colour=None, halo=True):
    """[("read", colour) | ("send", colour) | ("settle", exchanges)] in the order
    of the code.  A residual of colour c reads the halo of colour 1 - c."""
    out = []
    pat = (r"(?:(residual)<(\w)>\(\w+\)|(put)<(\w)>\(\w+, (true|false|halo)\)|settle\((\d|halo \? 1 : 0)\))")
    for res, rc, put, pc, flag, n in re.findall(pat, code):
        if res:
            out.append(("read", 1 - (colour if rc == "C" else int(rc))))
        elif put:
            if flag == "true" or (flag == "halo" and halo):
                out.append(("send", colour if pc == "C" else int(pc)))
        else:
            k = int(halo) if n.startswith("halo") else int(n)
            if k:
                out.append(("settle", k))
            else:
                out.append(("sync", 0))
    return out


def half_sweep(c, halo=True):
    return steps(body(r"void half_sweep\(bool halo\)"), c, halo)


def post_sweeps():
    return half_sweep(1) + half_sweep(0) + half_sweep(1) + half_sweep(0, halo=False)


def pre_sweeps():
    return half_sweep(0) + half_sweep(1) + half_sweep(0) + half_sweep(1)


def product():
    code = body(r"\bk_solve\(const")
    code = code[code.index("put<0>(q0"):]
    return steps(code[:code.index("reduce(")])


def test_source_steps_found():
    assert half_sweep(0) == [("read", 1), ("send", 0), ("settle", 1)]
    prolong = steps(body(r"void prolong\(int l\)"))
    assert prolong[0][0] == "send" and prolong[-1][0] == "settle"
    assert [s for s in product() if s[0] == "read"] == [("read", 1), ("read", 0)]


PROGRAMS = {
    "pre": lambda: pre_sweeps() + [("cluster", 0)] + pre_sweeps(),
    "prolong": lambda: steps(body(r"void prolong\(int l\)")) + post_sweeps(),
    "product": lambda: product() + [("cluster", 0)] + pre_sweeps() + [("cluster", 0)] + product(),
}


@pytest.mark.parametrize("name", sorted(PROGRAMS))
def test_halo_exchange_in_every_order(name):
    prog = PROGRAMS[name]()
    # exchange number of every send, and what each read must find
    turn, newest, number, expect = 0, [0, 0], {}, {}
    for k, (op, v) in enumerate(prog):
        if op == "send":
            turn += 1
            newest[v] = turn
            number[k] = turn
        elif op == "read":
            expect[k] = newest[v]

    # state per CTA: pc of the boundary warp, pc of the announcing warp, two
    # barriers (pending arrivals, bytes to come, phases completed), phases waited
    # for, halo contents, messages in flight towards this CTA
    one = (0, 0, ((1, 0, 0), (1, 0, 0)), (0, 0), (0, 0), frozenset())

    def bar(bars, q, arrivals, tx):
        p, t, ph = bars[q]
        p, t = p - arrivals, t + tx
        if p == 0 and t == 0:
            p, t, ph = 1, 0, ph + 1
        return tuple((p, t, ph) if k == q else bars[k] for k in range(2))

    def turns_before(k):
        return sum(1 for j in number if j < k)

    def moves(state):
        for c in range(2):
            edge, lead, bars, waited, halo, fly = state[c]
            other = state[1 - c]

            def put(mine, theirs=other):
                return (mine, theirs) if c == 0 else (theirs, mine)

            for m in fly:
                q, colour, num = m
                h = tuple(num if k == colour else halo[k] for k in range(2))
                yield put((edge, lead, bar(bars, q, 0, -1), waited, h, fly - {m}))
            if edge < len(prog):
                op, v = prog[edge]
                if op == "read":
                    assert halo[v] == expect[edge], f"stale halo of colour {v} at step {edge} of {prog}"
                    yield put((edge + 1, lead, bars, waited, halo, fly))
                elif op == "send":
                    n = number[edge]
                    o = other[:5] + (other[5] | {((n - 1) & 1, v, n)},)
                    yield put((edge + 1, lead, bars, waited, halo, fly), o)
            if lead < len(prog):
                op, v = prog[lead]
                if op == "read":
                    yield put((edge, lead + 1, bars, waited, halo, fly))
                elif op == "send":
                    yield put((edge, lead + 1, bar(bars, (number[lead] - 1) & 1, 1, 1), waited, halo, fly))
            if edge == lead < len(prog):
                op, v = prog[edge]
                if op == "sync":
                    yield put((edge + 1, lead + 1, bars, waited, halo, fly))
                elif op == "settle":
                    t = turns_before(edge)
                    qs = [(t - k) & 1 for k in range(v, 0, -1)]
                    if all(bars[q][2] > waited[q] for q in qs):
                        w = tuple(waited[k] + qs.count(k) for k in range(2))
                        yield put((edge + 1, lead + 1, bars, w, halo, fly))
                elif op == "cluster" and c == 0 and other[0] == other[1] == edge:
                    yield ((edge + 1, lead + 1) + state[0][2:], (edge + 1, lead + 1) + other[2:])

    seen, todo = {(one, one)}, [(one, one)]
    while todo:
        s = todo.pop()
        nxt = list(moves(s))
        assert nxt or all(c[0] == c[1] == len(prog) for c in s), f"a wait that never ends at {s} of {prog}"
        for n in nxt:
            if n not in seen:
                seen.add(n)
                todo.append(n)


def test_sums_in_a_row_in_every_order():
    """The mean of a swept coarsest level and the mean of the result follow each
    other with no cluster barrier between when that level is the only one.  A sum
    writes the CTA's part into every CTA's buffer, passes the cluster barrier and
    reads the buffer; a CTA whose reads are late must not find the next sum's
    parts there."""
    coarsest = re.findall(r"level_sum\(l, t, sred, (\w+)\)", body(r"void coarsest_solve\("))
    kernel = body(r"\bk_coarse\(const")
    (cycle,) = re.findall(r"cy\.cycle\(sred, (\w+)\)", kernel)
    (last,) = re.findall(r"level_sum\(0, ls, sred, (\w+)\)", kernel)
    assert coarsest and all(b == "s_part" for b in coarsest)  # the cycle's argument
    bufs = [cycle, last]
    prog = []
    for k, b in enumerate(bufs):
        prog += [("sync", k), ("write", k), ("cluster", k), ("read", k)]
    # per CTA: pc of the warp that writes, pc of a warp that only reads; who wrote each (buffer, part) last
    start = (((0, 0), (0, 0)), frozenset())
    seen, todo = {start}, [start]
    while todo:
        pcs, mem = todo.pop()
        found = dict(mem)
        nxt = []
        for c in range(2):
            for w in range(2):
                if pcs[c][w] == len(prog):
                    continue
                op, k = prog[pcs[c][w]]
                one = tuple(tuple(pcs[a][b] + (a == c and b == w) for b in range(2)) for a in range(2))
                if op == "write":
                    new = dict(found)
                    if w == 0:
                        new[bufs[k], 0, c] = new[bufs[k], 1, c] = k  # part c in the buffers of both CTAs
                    nxt.append((one, frozenset(new.items())))
                elif op == "read":
                    for part in range(2):
                        assert found[bufs[k], c, part] == k, f"sum {k} read a part of sum {found[bufs[k], c, part]}"
                    nxt.append((one, mem))
                elif op == "sync" and w == 0 and pcs[c][0] == pcs[c][1]:
                    both = tuple(tuple(pcs[a][b] + (a == c) for b in range(2)) for a in range(2))
                    nxt.append((both, mem))
                elif op == "cluster" and c == w == 0 and len({p for q in pcs for p in q}) == 1:
                    nxt.append((tuple(tuple(p + 1 for p in q) for q in pcs), mem))
        assert nxt or all(p == len(prog) for q in pcs for p in q)
        for n in nxt:
            if n not in seen:
                seen.add(n)
                todo.append(n)


def test_an_expired_wait_reaches_the_status_of_a_solve():
    """The flag of a thread whose wait ran out goes to the CTA that stores the
    status, before the cluster barrier after which that CTA stores it, and no
    other thread stores a status.  It also ends the iteration: the value that all
    CTAs compare with the tolerance becomes infinite."""
    code = body(r"\bk_solve\(const")
    stores = [m.start() for m in re.finditer(r"a\.st->status\s*=", code)]
    assert len(stores) == 1
    tail = code[:stores[0]]
    flag, barrier = tail.rindex("smem_u32(&s_fail), L.c0)"), tail.rindex("cc_sync();")
    assert flag < barrier and "s_fail ? ST_TMA_TIMEOUT : status" in code[stores[0]:]
    loop = code[code.index("while (agree(go))"):barrier]
    assert re.search(r"red\[0\] = cy\.fail \? \(double\)INFINITY[^;]*;\s*reduce\(k1, mx, red\)", loop)
