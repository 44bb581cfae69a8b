"""Static 32-lane schedules of the warp-cooperative Rosenbrock attempt.

The warp-cooperative attempt runs one cell on a whole warp, so that the few
cells that need thousands of attempts in one host step finish sooner than on
a single lane.  Each tableau stage of the attempt (the Jacobian partials, W,
the fill-in zeros, the LU factorisation, F, the right-hand side and the
triangular solve) is one *program*: the per-thread kernel's scalar floating
point operations, in its order, each written as one uniform operation on
the per-cell store S in shared memory:

    FMA  S[out] = fma(+-S[a], S[b], S[c])
    RCP  S[out] = 1 / S[out]          (a pivot; zero flags the matrix singular)

Constant slots holding 1, +0, -0, the mechanism's literal coefficients and
the attempt's 1/(gamma h) and c_ij/h make every other form exact:

    x * y           fma(x, y, -0)          round(x * y); x*y + (-0) keeps the sign of zero
    x (copy)        fma(x, 1, -0)
    -x              fma(-x, 1, -0)
    0.0             fma(+0, +0, +0)
    acc + t         fma(t, 1, acc)         round(t + acc)
    acc - t         fma(-t, 1, acc)
    fma(c, t, acc)  fma(c, t, acc)

So every slot receives exactly the roundings of the per-thread kernel (which
is built with --fmad=false, so only its explicit fma() calls fuse), and a
cell gives the same bits on either kernel.

Dependencies are the read-after-write, write-after-read and write-after-write
hazards on slots, in program order.  ``pipeline`` packs the operations into
steps of at most 32 for the device loop of csrc/warp_engine.cuh, which stores a
step's results during the next step and loads operands one step ahead: a value
is readable from its slot two steps after the operation that makes it, and one
step after it by the same lane alone, from the register that holds the lane's
previous result ("forwarded").  SAPRC99's attempt takes 2296 steps, of which
1722 are the dependence chain of its three solves, whose row sums keep a fixed
order.

``schedule`` is plain list scheduling for a machine whose step sees all
earlier steps; the tests use it as the reference for the dependencies.

Encoding, one 64-bit word per lane and step, four fields of a 14-bit slot and
two flags below it, so that a field is a byte offset after one shift:
  bits 0-15   a: slot * 4 + (negate the product)
  bits 16-31  b: slot * 4 + (the lane's previous result instead)
  bits 32-47  c: slot * 4 + (the lane's previous result instead)
  bits 48-63  out: slot * 4 + 2 * (reciprocal of b) + (store nothing)
Storing nothing is an idle lane, or a result that only the lane's next
operation reads.  A program that addresses a slot beyond 14 bits (``is_wide``;
none of the shipped ones) has words of four 32-bit fields, laid out alike.
"""

from __future__ import annotations

import heapq

FMA, RCP = 1, 2
LANES = 32
AHEAD = 8             # steps per unrolled group of the device loop
NARROW, WIDE = 16, 32  # bits of a word's field
PREV = -1             # operand: the lane's previous result


def is_wide(*programs) -> bool:
    """Whether the programs' slots need the wide words."""
    return any(x >= 1 << (NARROW - 2) for ops in programs for op in ops for x in op[1:5])


class Program:
    """Sequential uniform operations, built in per-thread program order.

    `zn`, `zp`, `one` are the slots of -0.0, +0.0 and 1.0; `lit(value)`
    returns the slot of a literal constant."""

    def __init__(self, zn: int, zp: int, one: int, lit):
        self.ops: list[tuple[int, int, int, int, int, int]] = []
        self.zn, self.zp, self.one, self.lit = zn, zp, one, lit

    def fma(self, out, a, b, c, neg=False):
        self.ops.append((FMA, out, a, b, c, int(bool(neg))))

    def rcp(self, out):
        self.ops.append((RCP, out, 0, 0, 0, 0))

    def mul(self, out, a, b):
        """S[out] = S[a] * S[b]."""
        self.fma(out, a, b, self.zn)

    def copy(self, out, a):
        self.fma(out, a, self.one, self.zn)

    def zero(self, out):
        self.fma(out, self.zp, self.zp, self.zp)

    def acc_term(self, out, first: bool, coef: float, t: int, acc: int | None = None):
        """One term of a sum accumulated left to right into S[out]: the first
        term is t, -t or c*t; later ones acc + t, acc - t or fma(c, t, acc).
        `acc` (default out) is where the running sum is read from."""
        acc = out if acc is None else acc
        if first:
            if coef == 1.0:
                self.copy(out, t)
            elif coef == -1.0:
                self.fma(out, t, self.one, self.zn, neg=True)
            else:
                self.fma(out, t, self.lit(coef), self.zn)
        else:
            if coef == 1.0:
                self.fma(out, t, self.one, acc)
            elif coef == -1.0:
                self.fma(out, t, self.one, acc, neg=True)
            else:
                self.fma(out, self.lit(coef), t, acc)

    def lu(self, plan):
        """Row-wise Doolittle factorisation in place on the LU slots (fill-in
        slots zeroed beforehand): products in plan order, then the pivot
        reciprocal or the multiply of an L entry by it."""
        diag = set(plan.diag)
        for out, w, b, e, dg in plan.ops:
            for q in range(b, e):
                pa, pb = plan.products[q]
                self.fma(out, pa, pb, out, neg=True)
            if out in diag:
                self.rcp(out)
            elif dg >= 0:
                self.mul(out, out, dg)

    def solve(self, plan, base: int):
        """(LU) x = b in place on S[base .. base + NV): unit-L forward rows
        ascending, U backward rows descending, then the reciprocal pivot."""
        nv = plan.n_var
        for i in range(nv):
            for col, slot in plan.lower[i]:
                self.fma(base + i, slot, base + col, base + i, neg=True)
        for i in range(nv - 1, -1, -1):
            for col, slot in plan.upper[i]:
                self.fma(base + i, slot, base + col, base + i, neg=True)
            self.mul(base + i, base + i, plan.diag[i])


def lu_zero_slots(plan) -> list[int]:
    """Operation outputs that start from 0 rather than from a W slot."""
    return [out for out, w, b, e, dg in plan.ops if w < 0]


def _locations(op):
    kind, out, a, b, c, _ = op
    if kind == FMA:
        return (a, b, c), (out,)
    return (out,), (out,)


def dependencies(ops) -> list[list[int]]:
    """Hazard edges of each operation on earlier operations."""
    last_write: dict = {}
    readers: dict = {}
    deps = []
    for n, op in enumerate(ops):
        reads, writes = _locations(op)
        d = set()
        for loc in reads:
            if loc in last_write:
                d.add(last_write[loc])
        for loc in writes:
            if loc in last_write:
                d.add(last_write[loc])
            d.update(r for r in readers.get(loc, ()) if r != n)
        deps.append(sorted(d))
        for loc in reads:
            readers.setdefault(loc, []).append(n)
        for loc in writes:
            last_write[loc] = n
            readers[loc] = []
    return deps


def schedule(ops, lanes: int = LANES) -> list[list[int]]:
    """Steps of at most `lanes` operations; every operation after all of its
    dependencies.  Priority: longest remaining dependency path, then program
    order."""
    n = len(ops)
    deps = dependencies(ops)
    succ = [[] for _ in range(n)]
    indeg = [len(d) for d in deps]
    for i, d in enumerate(deps):
        for j in d:
            succ[j].append(i)
    tail = [1] * n
    for i in range(n - 1, -1, -1):
        for s in succ[i]:
            tail[i] = max(tail[i], 1 + tail[s])
    ready = [(-tail[i], i) for i in range(n) if indeg[i] == 0]
    heapq.heapify(ready)
    steps = []
    done = 0
    while done < n:
        batch = [heapq.heappop(ready)[1] for _ in range(min(lanes, len(ready)))]
        if not batch:
            raise RuntimeError("dependency cycle in warp schedule")
        batch.sort()
        steps.append(batch)
        done += len(batch)
        for i in batch:
            for s in succ[i]:
                indeg[s] -= 1
                if indeg[s] == 0:
                    heapq.heappush(ready, (-tail[s], s))
    return steps


LOAD = 2              # steps from an operation to a reader through its slot


def pivot_every(ops) -> int:
    """Steps from one that may hold reciprocals to the next.  Each of them
    costs the device loop a vote, and one with a reciprocal several steps, so a
    long program gathers them (SAPRC99: 37 steps instead of 56, TS1 104 instead
    of 163, at the same length); a short one would wait for them."""
    return AHEAD if len(ops) >= 5000 else 1


def pipeline(ops, lanes: int = LANES) -> list[list[int | None]]:
    """Steps of `lanes` entries (an operation or None) for the device loop.
    Priority: longest remaining path, a sum's next term one step after, any
    other reader LOAD steps."""
    every = pivot_every(ops)
    n = len(ops)
    raw: list[list[int]] = []
    raw_succ: list[list[int]] = [[] for _ in range(n)]
    other_succ: list[list[tuple[int, int]]] = [[] for _ in range(n)]
    left = [0] * n
    last: dict = {}
    readers: dict = {}
    for i, op in enumerate(ops):
        reads, (out,) = _locations(op)
        r = sorted({last[x] for x in reads if x in last})
        raw.append(r)
        # A slot's next writer may share the step of its readers (they have
        # loaded it before), and follows an earlier writer.
        after = {q: 0 for q in readers.get(out, ()) if q not in r}
        if out in last and last[out] not in r:
            after[last[out]] = 1
        for j in r:
            raw_succ[j].append(i)
        for j, lag in after.items():
            other_succ[j].append((i, lag))
        left[i] = len(r) + len(after)
        for x in reads:
            readers.setdefault(x, []).append(i)
        last[out], readers[out] = i, []
    tail = [1] * n
    for i in range(n - 1, -1, -1):
        for t in raw_succ[i]:
            lag = (every + 1) // 2 if ops[t][0] == RCP else 1 if ops[t][4] == ops[i][1] else LOAD
            tail[i] = max(tail[i], lag + tail[t])
        for t, lag in other_succ[i]:
            tail[i] = max(tail[i], lag + tail[t])
    step, lane, earliest = [-1] * n, [-1] * n, [0] * n
    from_slots = {0: [i for i in range(n) if left[i] == 0]}   # step -> operations ready then
    forwarded: dict[int, list[tuple[int, int]]] = {}          # step -> (operation, the one it follows)
    ready: list[tuple[int, int]] = []
    s = done = 0

    def release(i):
        at = max([earliest[i]] + [step[j] + LOAD for j in raw[i]])
        if raw[i]:
            j = max(raw[i], key=lambda q: step[q])
            f = step[j] + 1
            square = ops[i][0] == FMA and ops[i][2] == ops[i][3] == ops[j][1]   # one factor can be forwarded
            if (s < f < at and f >= earliest[i] and not square
                    and all(step[q] + LOAD <= f for q in raw[i] if q != j)):
                forwarded.setdefault(f, []).append((i, j))
        if at <= s:
            heapq.heappush(ready, (-tail[i], i))
        else:
            from_slots.setdefault(at, []).append(i)

    def place(i):
        step[i] = s
        for t in raw_succ[i]:
            left[t] -= 1
            if left[t] == 0:
                release(t)
        for t, lag in other_succ[i]:
            earliest[t] = max(earliest[t], s + lag)
            left[t] -= 1
            if left[t] == 0:
                release(t)

    pivots: list[tuple[int, int]] = []

    while done < n:
        for i in from_slots.pop(s, ()):
            if step[i] < 0:
                heapq.heappush(ready, (-tail[i], i))
        follow = sorted((-tail[i], i, j) for i, j in forwarded.pop(s, ()))
        # Reciprocals wait for a step that has the code for them.
        pivot_step = s % every == every - 1
        if pivot_step:
            while pivots:
                heapq.heappush(ready, heapq.heappop(pivots))
        else:
            follow = [x for x in follow if ops[x[1]][0] != RCP]
        used: set[int] = set()
        anywhere = []
        f = count = 0
        while count < lanes and (ready or f < len(follow)):
            if f < len(follow) and (not ready or follow[f][:2] <= ready[0]):
                _, i, j = follow[f]
                f += 1
                if lane[j] in used:
                    continue
                lane[i] = lane[j]
                used.add(lane[i])
            else:
                top = heapq.heappop(ready)
                i = top[1]
                if step[i] >= 0:
                    continue
                if ops[i][0] == RCP and not pivot_step:
                    pivots.append(top)
                    continue
                anywhere.append(i)
            place(i)
            count += 1
        rest = (q for q in range(lanes) if q not in used)
        for i in anywhere:
            lane[i] = next(rest)
        done += count
        s += 1
    rows: list[list[int | None]] = [[None] * lanes for _ in range(s)]
    for i in range(n):
        rows[step[i]][lane[i]] = i
    return rows


def sequential(ops) -> list[list[int]]:
    """One operation per step, for a single thread; an idle step before the
    square of the result just made (one factor can be forwarded)."""
    steps: list[list[int]] = []
    for i, op in enumerate(ops):
        if i and op[0] == FMA and op[2] == op[3] == ops[i - 1][1]:
            steps.append([])
        steps.append([i])
    return steps


def encode(ops, steps, lanes: int = LANES, bits: int = NARROW) -> list[int]:
    """steps x lanes words with fields of `bits` (a step lists the operations of its lanes, None or
    missing for an idle lane).  An operand whose writer is the lane's
    previous operation, one step before, is taken from the lane's register,
    and a result that nothing else reads is not stored.  With several lanes
    and narrow words an odd number of steps is filled up with an idle one, and
    two steps' words of a lane are side by side."""
    idle = 1 << 3 * bits
    where = {}
    for s, row in enumerate(steps):
        for q, i in enumerate(row):
            if i is not None:
                where[i] = (s, q)
    fields: list = [None] * len(ops)
    stored = [False] * len(ops)
    last: dict = {}
    for i, (kind, out, a, b, c, neg) in enumerate(ops):
        if kind == RCP:
            a, b, c = 0, b or out, 0
        reads = [b] if kind == RCP else [a, b, c]
        prev = {x for x in reads if x in last and where[last[x]] == (where[i][0] - 1, where[i][1])}
        assert len(prev) <= 1
        if kind == FMA and a in prev and a != b:
            a, b = b, a
        x_b = b in prev and not (kind == FMA and a == b)
        x_c = kind == FMA and c in prev
        from_slot = ([a] if kind == FMA else []) + ([] if x_b else [b]) + ([c] if kind == FMA and not x_c else [])
        for x in from_slot:
            if x in last:
                assert where[last[x]][0] <= where[i][0] - LOAD
                stored[last[x]] = True
        fields[i] = (a, PREV if x_b else b, PREV if x_c else c)
        last[out] = i
    for i in last.values():
        stored[i] = True
    rows = []
    pairs = lanes > 1 and bits == NARROW
    for row in list(steps) + [[]] * (len(steps) % 2 if pairs else 0):
        line = [idle] * lanes
        for q, i in enumerate(row):
            if i is None:
                continue
            kind, out, _, _, _, neg = ops[i]
            a, b, c = fields[i]
            assert all(PREV <= x < 1 << (bits - 2) for x in (out, a, b, c)) and a >= 0, "a slot exceeds its field"
            lo = (a << 2 | bool(neg)) | (max(b, 0) << 2 | (b == PREV)) << bits
            hi = (max(c, 0) << 2 | (c == PREV)) | (out << 2 | (kind == RCP) << 1 | (not stored[i])) << bits
            line[q] = lo | hi << 2 * bits
        rows.append(line)
    if not pairs:
        return [word for line in rows for word in line]
    return [line[q] for s in range(0, len(rows), 2) for q in range(lanes) for line in rows[s:s + 2]]


def decode(word: int, bits: int = NARROW) -> tuple[int, int, int, int, int, int]:
    """(kind, out, a, b, c, neg) of one word; kind 0 for a lane that stores
    nothing, operand -1 for the lane's previous result."""
    a, b, c, out = ((word >> bits * f) & ((1 << bits) - 1) for f in range(4))
    if out & 1:
        return 0, out >> 2, 0, 0, 0, 0
    b_, c_ = (PREV if x & 1 else x >> 2 for x in (b, c))
    return RCP if out & 2 else FMA, out >> 2, a >> 2, b_, c_, a & 1
