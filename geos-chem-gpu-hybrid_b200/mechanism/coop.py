"""Tables for the cooperative kernel (one thread block per cell).

The one-thread-per-cell kernels run straight-line statement lists.  In the
cooperative kernel the threads of a block share one cell, so every thread
runs the same instructions on different entries: Fun, Jac, the
factorisation and the solves become loops over tables.  This module turns
the mechanism IR into those tables; ``coop_inc`` emits them as C arrays.

Expressions.  Every rate A(j), production P_VAR(i), destruction D_VAR(i),
Jacobian partial B(m) and entry JVS(k) of the IR is a left-associated
signed sum ``((t0 op t1) op t2) ...`` (the first term possibly negated) of
left-associated products ``((f0*f1)*f2)*f3`` whose factors are variable
species V, fixed species F, rate constants RCT, rates A / partials B (one
scratch array) or literals.  A term is stored as four 16-bit factor codes
(kind << 13 | index, 0xFFFF for none) and an operation code (0 first term,
1 first term negated, 2 add, 3 subtract).  Evaluated in table order, each
value gets exactly the operations of the generated Fun_SPLIT / Jac_SP
statements (gckpp_Function.F90:2170-5060, gckpp_Jacobian.F90:47-20887), so
the --fmad=false build rounds like them.  A mechanism with any other
expression shape gets no tables (``compile_tables`` returns None) and no
cooperative kernel.

Factorisation (KppDecomp, gckpp_LinearAlgebra.F90:46-84), right-looking.
The reference eliminates row by row: row k receives, in increasing pivot
order j, ``W(c) = W(c) + a*U(j,c)`` with ``a = -(W(j)/U(j,j))``, and stores
``-a`` as L(k,j).  Step j of the right-looking form first forms the
multipliers of column j (every row i > j with L(i,j) in the pattern) and
then applies pivot row j to all those rows at once.  Each entry still
receives its updates in increasing pivot order and the same operations, so
the result is the same bit for bit; the parallelism is the rows and columns
of one step instead of one row's columns.

Solves (KppSolve, gckpp_LinearAlgebra.F90:645-2311).  The forward sweep
``X(i) = X(i) - L(i,j)*X(j)`` over increasing j is run column by column:
at step j, X(j) is final and every row i with L(i,j) subtracts its term --
the same per-row order.  The backward sweep subtracts U(i,c)*X(c) in
increasing c and then divides; its rows are grouped into levels (a row's
level is one more than the highest level among its columns), rows of one
level run in parallel, each row's terms in the reference order.  That
order makes the sweep a chain of every row's terms (2,452 dependent
subtractions for the synthetic mechanism), so the FMA build, which need
not round like the reference, runs the backward sweep by columns too
(``bwc``: at step i, X(i) = acc(i)/U(i,i) and every row r < i with U(r,i)
subtracts its term), in the reverse of the reference's per-row order.
"""
from __future__ import annotations

from . import codegen

KIND_V, KIND_F, KIND_K, KIND_S, KIND_N = 0, 1, 2, 3, 4
NONE = 0xFFFF
OP_FIRST, OP_NEG, OP_ADD, OP_SUB = 0, 1, 2, 3
MAX_FACTORS = 4
MAX_INDEX = 1 << 13


class Unsupported(ValueError):
    pass


def _factors(node, consts):
    """Factor codes of a left-associated product chain."""
    out = []
    while isinstance(node, list) and node[0] == "*":
        out.append(node[2])
        node = node[1]
    out.append(node)
    out.reverse()
    codes = []
    for f in out:
        tag = f[0]
        if tag == "v":
            kind, idx = KIND_V, f[1]
        elif tag == "f":
            kind, idx = KIND_F, f[1]
        elif tag == "k":
            kind, idx = KIND_K, f[1]
        elif tag in ("a", "b"):
            kind, idx = KIND_S, f[1]
        elif tag == "n":
            val = float(codegen.literal(f[1]))
            if val not in consts:
                consts[val] = len(consts)
            kind, idx = KIND_N, consts[val]
        else:
            raise Unsupported(f"factor {f}")
        if not 0 <= idx < MAX_INDEX:
            raise Unsupported(f"index {idx}")
        codes.append((kind << 13) | idx)
    if len(codes) > MAX_FACTORS:
        raise Unsupported("product of more than four factors")
    return codes + [NONE] * (MAX_FACTORS - len(codes))


def _sum_terms(node, consts):
    """(op, factor codes) of a left-associated signed sum of products."""
    terms = []
    for i, (op, t) in enumerate(codegen._chain(node)):
        if i == 0:
            code = OP_FIRST
            if t[0] == "neg":
                code, t = OP_NEG, t[1]
        else:
            code = OP_ADD if op == "+" else OP_SUB
        terms.append((code, _factors(t, consts)))
    return terms


def compile_tables(mech: dict):
    """All tables of the cooperative kernel, or None when some expression
    falls outside the supported shapes."""
    n, nnz = mech["nvar"], mech["nnz"]
    nreact, nb = mech["nreact"], mech["nb"]
    crow, diag, icol = mech["lu_crow"], mech["lu_diag"], mech["lu_icol"]
    where = mech["lu_where"]
    if nnz >= 1 << 16 or n >= 1 << 16:
        return None
    consts: dict = {}
    sums = []
    try:
        for e in mech["rates"]:                       # A(j): ids 0 .. NREACT-1
            sums.append(_sum_terms(e, consts))
        for e in mech["prod"]:                        # P_VAR(i)
            sums.append(_sum_terms(e, consts))
        for e in mech["dest"]:                        # D_VAR(i)
            sums.append(_sum_terms(e, consts))
        bexpr = [["n", "0"]] * nb                     # indices no entry reads
        for m, e in mech["jac_b"]:
            bexpr[m] = e
        for e in bexpr:                               # B(m)
            sums.append(_sum_terms(e, consts))
        for e in mech["jvs"]:                         # JVS(k)
            sums.append(_sum_terms(e, consts))
    except Unsupported:
        return None
    off, ops, fac = [0], [], []
    for s in sums:
        for op, codes in s:
            ops.append(op)
            fac.extend(codes)
        off.append(len(ops))

    # right-looking factorisation: per pivot j, the L(i,j) positions and the
    # updates (target (i,c), multiplier (i,j), source (j,c))
    mul = [[] for _ in range(n)]
    upd = [[] for _ in range(n)]
    for i in range(n):
        for kk in range(crow[i], diag[i]):
            j = icol[kk]
            mul[j].append(kk)
            for jj in range(diag[j] + 1, crow[j + 1]):
                upd[j].append((where[(i, icol[jj])], kk, jj))
    mul_off, mul_pos, upd_off, upd_ent = [0], [], [0], []
    for j in range(n):
        mul_pos += mul[j]
        mul_off.append(len(mul_pos))
        upd_ent += upd[j]
        upd_off.append(len(upd_ent))

    # forward sweep by columns: per j, the (row, L position) pairs
    fwd = [[] for _ in range(n)]
    for i in range(n):
        for kk in range(crow[i], diag[i]):
            fwd[icol[kk]].append((i, kk))
    fwd_off, fwd_ent = [0], []
    for j in range(n):
        fwd_ent += fwd[j]
        fwd_off.append(len(fwd_ent))

    # backward sweep by levels
    lev = [0] * n
    for i in range(n - 1, -1, -1):
        lev[i] = max([lev[icol[jj]] + 1 for jj in range(diag[i] + 1, crow[i + 1])] + [0])
    nlev = max(lev) + 1 if n else 0
    bwd_rows, bwd_off = [], [0]
    for level in range(nlev):
        bwd_rows += [i for i in range(n) if lev[i] == level]
        bwd_off.append(len(bwd_rows))

    # backward sweep by columns (FMA build): per column i, from the last, the
    # (row r < i, U(r,i) position) pairs
    bwc = [[] for _ in range(n)]
    for r in range(n):
        for jj in range(diag[r] + 1, crow[r + 1]):
            bwc[icol[jj]].append((r, jj))
    bwc_off, bwc_ent = [0], []
    for i in range(n - 1, -1, -1):
        bwc_ent += bwc[i]
        bwc_off.append(len(bwc_ent))

    kdiag = [-1] * nnz
    for i in range(n):
        kdiag[diag[i]] = i

    cvals = [0.0] * len(consts)
    for v, k in consts.items():
        cvals[k] = v
    return {
        "nsum": len(sums), "sum_off": off, "term_op": ops, "term_fac": fac,
        "consts": cvals or [0.0],
        "mul_off": mul_off, "mul_pos": mul_pos or [0],
        "upd_off": upd_off, "upd": upd_ent,
        "fwd_off": fwd_off, "fwd": fwd_ent,
        "bwd_off": bwd_off, "bwd_rows": bwd_rows, "nlev": nlev,
        "bwc_off": bwc_off, "bwc": bwc_ent,
        "kdiag": kdiag,
        "sid_rate": 0, "sid_prod": nreact, "sid_dest": nreact + n,
        "sid_b": nreact + 2 * n, "sid_jvs": nreact + 2 * n + nb,
    }


# ---------------------------------------------------------------------------
# Level programs as warp streams.
#
# The elimination order of a sparse mechanism is a chain of rows, but its
# dependencies are shallow: in fullchem (353 species) the forward sweep has 37
# levels, the backward sweep 33 and the factorisation, taken entry by entry,
# 62.  Every phase of the solver is therefore a program of levels; the entries
# of a level are independent.  An entry is computed by a group of 1, 2, 4 .. 32
# consecutive lanes that share its products:
#
#     acc (lane 0 of the group: the entry's start value) -= A(word.lo)*B(word.hi)
#
# after which the group is summed by butterfly exchanges and lane 0 finishes
# the entry.  The build that must round like the reference takes groups of one
# lane (each entry's terms stay one left-to-right sum, in the reference's
# order); the production build splits long sums (up to 327 terms in fullchem).
#
# The generator places the groups on the block's warps and writes one stream
# per warp: a list of operations of WORDS words per lane, in the order in which
# the warp executes them.  The addresses of a stream are known in advance, so
# the kernel fetches operations several ahead of their use.
#
# Operands are given as byte offsets in their array (the kernel keeps the cell
# in shared memory), so that a word needs no arithmetic; a missing operand
# points at a constant 0 (or 1) behind the array, so that it needs no test.
#
#   rate operations   four products (f0 | f1<<16, f2 | f3<<16).  Product k of
#                     operation i of warp w and lane l is number
#                     ((i*4 + k)*NW + w)*32 + l.
#   dest operations   header, control, three products (f0 | f1<<16, f2)
#   sum operations    two halves of a header and three words (prod, jvs)
#   level operations  header, control, six words (lu, sweep)
#
# Control word, per lane: L_* flags, log2 of the lane's group, exchanges that
# the warp does (the largest of its groups), products in use, a chain's first
# step, block barriers after the operation.  A sum's header is its entry's
# offset | control << 16; a level's is the entry's offset | the offset of its
# scale in R << 16.

WORDS = 8
DEPTH = 4              # operations fetched ahead; a segment is a multiple of it
L_LEAD, L_FIRST, L_END, L_CHAIN, L_DIAG, L_SCALED = 1, 2, 4, 8, 16, 32
L_DIAGS = 1 << 15      # factorisation: some lane of the warp has L_DIAG
L_GROUP, L_FOLD, L_USED, L_STEP, L_SYNC = 6, 9, 12, 15, 20
CHAIN_MAX = 32         # rows of a warp chain (one lane per row)
# cycles of an operation: fixed part, per product, per exchange, end of an
# entry (measured latencies on a B200: shared memory 29, FP64 FMA 9, barrier of
# 128 threads 19; a lone warp issues every ~3 cycles); they only steer how far
# sums are split
OP_COST, TERM_COST, FOLD_COST, END_COST = 70, 18, 40, 40


def _lanes(items, k, split):
    """Warp rounds of one level: [(header, words)] -> lists of at most 32
    (header, log2 group, words of the lane), groups aligned to their size."""
    sized = []
    for head, words in items:
        g = 1
        while split and g < 32 and -(-len(words) // g) > k:
            g *= 2
        sized.append((g, -(-len(words) // g), head, words))
    sized.sort(key=lambda x: (-x[0], -x[1]))
    rounds, lanes = [], []
    for g, _, head, words in sized:
        if len(lanes) + g > 32:
            rounds.append(lanes)
            lanes = []
        lanes += [(head, g.bit_length() - 1, words[q::g]) for q in range(g)]
    if lanes:
        rounds.append(lanes)
    return rounds


def _cost(lanes, per_op):
    k = max(len(w) for _, _, w in lanes)
    s = max(lg for _, lg, _ in lanes)
    return OP_COST * max(1, -(-k // per_op)) + TERM_COST * k + FOLD_COST * s + END_COST


def _place(items, nw, split, per_op):
    """A level's rounds on nw warps: (warp lists, cost of the longest)."""
    best, cost = None, None
    longest = max([len(w) for _, w in items] + [1])
    for k in (range(1, min(longest, 40) + 1) if split else (longest,)):
        warps, load = [[] for _ in range(nw)], [0] * nw
        for lanes in sorted(_lanes(items, k, split), key=lambda r: -_cost(r, per_op)):
            w = load.index(min(load))
            warps[w].append(lanes)
            load[w] += _cost(lanes, per_op)
        if cost is None or max(load) < cost:
            best, cost = warps, max(load)
    return best, cost


class Segment:
    """One phase: per warp a list of operations (32 lanes x WORDS words).
    `none`: the word of a missing product (for rates and dest two words)."""

    def __init__(self, nw, none, head=0):
        self.nw, self.none, self.head = nw, none, head
        self.ops = [[] for _ in range(nw)]
        self.cost = 0

    def idle(self):
        if isinstance(self.none, tuple):
            return list(self.none) * 4 if self.head is None else [self.head, 0] + list(self.none) * 3
        return [self.head, 0] + [self.none] * 6

    def pad(self, idle=None):
        for ops in self.ops:
            while not ops or len(ops) % DEPTH:
                ops.append([list(idle or self.idle()) for _ in range(32)])
        return self

    def rates(self, products):
        for n, words in enumerate(products):
            v, w = n // 32 % self.nw, n // (32 * self.nw)
            if w % 4 == 0 and len(self.ops[v]) == w // 4:
                self.ops[v].append([self.idle() for _ in range(32)])
            self.ops[v][w // 4][n % 32][w % 4 * 2:w % 4 * 2 + 2] = words
        return self.pad()

    def _split(self, lanes, per_op):
        """A warp round as operations: (lane words, header, control) lists."""
        k = max(len(w) for _, _, w in lanes)
        s = max(lg for _, lg, _ in lanes)
        n = max(1, -(-k // per_op))
        for t in range(n):
            ctl = (L_FIRST if t == 0 else 0) | (L_END if t == n - 1 else 0) | s << L_FOLD | \
                min(per_op, k - per_op * t) << L_USED
            out = []
            for x in range(32):
                if x < len(lanes):
                    (head, flags), lg, words = lanes[x]
                    w = words[per_op * t:per_op * (t + 1)]
                    lead = 0 if x % (1 << lg) else L_LEAD
                    out.append((head, ctl | lead | flags | lg << L_GROUP, w + [self.none] * (per_op - len(w))))
                else:
                    out.append((self.head, ctl, [self.none] * per_op))
            yield out

    def dest(self, items, split):
        warps, self.cost = _place(items, self.nw, split, 3)
        for v, rounds in enumerate(warps):
            for lanes in rounds:
                for op in self._split(lanes, 3):
                    self.ops[v].append([[h, c] + [x for w in ws for x in w] for h, c, ws in op])
        return self.pad()

    def sums(self, items, split):
        warps, self.cost = _place(items, self.nw, split, 3)
        idle = [(self.head, 0, [self.none] * 3)] * 32
        for v, rounds in enumerate(warps):
            halves = [op for lanes in rounds for op in self._split(lanes, 3)]
            if len(halves) % 2:
                halves.append(idle)
            for a, b in zip(halves[::2], halves[1::2]):
                self.ops[v].append([[h | (c & 0xFFF) << 16] + w + [g | (d & 0xFFF) << 16] + u
                                    for (h, c, w), (g, d, u) in zip(a, b)])
        return self.pad([self.head] + [self.none] * 3 + [self.head] + [self.none] * 3)

    def level(self, items, split):
        warps, cost = _place(items, self.nw, split, 6)
        self.cost += cost + 30
        for v, rounds in enumerate(warps):
            for lanes in rounds:
                diags = L_DIAGS if any(flags & L_DIAG for (_, flags), _, _ in lanes) else 0
                for op in self._split(lanes, 6):
                    self.ops[v].append([[h, c | diags] + w for h, c, w in op])
        self._sync()

    def chain(self, rows, pos):
        """A warp chain over `rows` [(header, flags)]: lane r owns row r; step
        j broadcasts row j's value and every lane with an entry (r, j)
        subtracts its term."""
        m = len(rows)
        for j0 in range(0, m, 6):
            used = min(6, m - j0)
            ctl = (L_FIRST if j0 == 0 else 0) | (L_END if j0 + used == m else 0) | \
                used << L_USED | L_CHAIN | j0 << L_STEP
            op = []
            for r in range(32):
                head, flags, lead = rows[r] + (L_LEAD,) if r < m else (self.head, rows[0][1], 0)
                op.append([head, ctl | lead | flags] +
                          [pos.get((r, j), self.none & 0xFFFF) if j < m else self.none & 0xFFFF
                           for j in range(j0, j0 + 6)])
            self.ops[0].append(op)
        self.cost += 45 * m + 100
        self._sync()

    def _sync(self):
        """A block barrier after everything so far."""
        for ops in self.ops:
            if not ops:
                ops.append([self.idle() for _ in range(32)])
            for lane in ops[-1]:
                lane[1] += 1 << L_SYNC


def _sweep(seg, n, deps, split, forward):
    """Levels of a triangular sweep.  deps[i]: [(column, factor position)] in
    the reference's order.  Runs of levels with very few rows become warp
    chains (at most CHAIN_MAX rows): first one level subtracts every term whose
    column lies outside the chain, then one warp walks the chain."""
    one = 8 * n << 16                    # offset of the constant 1 behind R

    def head(i):
        return (8 * i | one, 0) if forward else (8 * i | 8 * i << 16, L_SCALED)

    lev = [0] * n
    order = list(range(n)) if forward else list(range(n - 1, -1, -1))
    for i in order:
        lev[i] = max([lev[c] + 1 for c, _ in deps[i]] + [0])
    nlev = max(lev) + 1 if n else 0
    by = [[i for i in order if lev[i] == k] for k in range(nlev)]

    def items(rows, skip=(), bulk=False):
        return [((8 * i | one, 0) if bulk else head(i), [8 * p | 8 * c << 16 for c, p in deps[i] if c not in skip])
                for i in rows]

    k = 1 if forward else 0              # the forward sweep leaves level 0 as it is
    while k < nlev:
        e = k
        if split:
            rows = 0
            while e < nlev and len(by[e]) <= (4 if e == 0 else 2) and rows + len(by[e]) <= CHAIN_MAX:
                rows += len(by[e])
                e += 1
        if e - k >= 4:
            rows = [i for q in range(k, e) for i in by[q]]
            inside = {i: r for r, i in enumerate(rows)}
            bulk = [it for it in items(rows, inside, True) if it[1]]
            if bulk:
                seg.level(bulk, split)
            seg.chain([head(i) for i in rows],
                      {(inside[i], inside[c]): 8 * p for i in rows for c, p in deps[i] if c in inside})
            k = e
        else:
            seg.level(items(by[k]), split)
            k += 1


def level_programs(mech: dict, split: bool, nw: int):
    """The cooperative kernel's programs, or None for unsupported expression
    shapes.  split: sums may be divided over lanes (production build); nw:
    warps of the block."""
    if compile_tables(mech) is None:
        return None
    n, nfix, nnz, nreact = mech["nvar"], mech["nfix"], mech["nnz"], mech["nreact"]
    crow, diag, icol, where = mech["lu_crow"], mech["lu_diag"], mech["lu_icol"], mech["lu_where"]
    if nnz >= (1 << 13) - 1:           # byte offsets of 16 bits
        return None
    extra = {}                 # first factors behind the rate constants: (reaction or
                               # -1, literal), the literal itself or RCT(j)*literal
    ext = {1.0: 0}             # constants behind the species (other factors)
    coef = {1.0: 0}            # coefficients of the sums

    def slot(table, value):
        return table.setdefault(value, len(table))

    def product(node):
        """[first, f1, f2, f3]: first indexes [RCT | extra], the others
        [V | FIX | ext]; missing factors are the constant 1, whose product
        is exact.  A leading RCT(j)*literal is formed once per cell."""
        fs = []
        while isinstance(node, list) and node[0] == "*":
            fs.append(node[2])
            node = node[1]
        fs.append(node)
        fs.reverse()

        def num(f):
            return float(codegen.literal(f[1]))

        def other(f):
            if f[0] == "v":
                return f[1]
            if f[0] == "f":
                return n + f[1]
            if f[0] == "n":
                return n + nfix + slot(ext, num(f))
            raise Unsupported(str(f))

        f0 = fs[0]
        if f0[0] == "k" and len(fs) > 1 and fs[1][0] == "n":
            first, fs = nreact + slot(extra, (f0[1], num(fs[1]))), fs[1:]
        elif f0[0] == "k":
            first = f0[1]
        elif f0[0] == "n":
            first = nreact + slot(extra, (-1, num(f0)))
        else:                  # 1*v is exact
            first, fs = nreact + slot(extra, (-1, 1.0)), [None] + fs
        rest = [other(f) for f in fs[1:]]
        if len(rest) > 3:
            raise Unsupported("product of more than four factors")
        return [first] + rest + [n + nfix] * (3 - len(rest))

    def signed(node):
        out = []
        for i, (op, t) in enumerate(codegen._chain(node)):
            sign = -1.0 if op == "-" else 1.0
            if t[0] == "neg":
                if i:
                    raise Unsupported("negated inner term")
                sign, t = -sign, t[1]
            out.append((sign, t))
        return out

    def scaled(node, tag, index, flip=1.0):
        """Words coef | value << 16 of a sum of +-[literal *] tag(index)."""
        words = []
        for sign, t in signed(node):
            c = sign * flip
            if t[0] == "n" and float(codegen.literal(t[1])) == 0.0 and not words:
                continue
            if t[0] == "*" and t[1][0] == "n":
                c, t = c * float(codegen.literal(t[1][1])), t[2]
            if t[0] != tag:
                raise Unsupported(str(t))
            words.append(slot(coef, c) | index(t[1]) << 16)
        return words

    try:
        rate = [product(e) for e in mech["rates"]]
        # partials B: each feeds one column of the Jacobian only, so they are
        # formed for a part of the columns at a time, as many as the rates'
        # scratch array holds
        col_of = {}
        for p, e in enumerate(mech["jvs"]):
            for b in codegen._refs(e, "b"):
                if col_of.setdefault(b, icol[p]) != icol[p]:
                    raise Unsupported("partial of two columns")
        bexpr = dict(mech["jac_b"])
        parts, part_of = [[]], {}
        for c in range(n):
            mine = sorted(b for b, k in col_of.items() if k == c)
            if len(parts[-1]) + len(mine) > nreact:
                parts.append([])
            part_of[c] = len(parts) - 1
            parts[-1] += mine
        bmap = {b: k for part in parts for k, b in enumerate(part)}
        if max(len(part) for part in parts) > nreact:
            raise Unsupported("column with too many partials")
        bpart = [[product(bexpr[b]) for b in part] for part in parts]
        dest = []
        for i, e in enumerate(mech["dest"]):
            words = []
            for sign, t in signed(e):
                if t[0] == "n" and float(codegen.literal(t[1])) == 0.0 and not words:
                    continue
                f = product(t)
                if sign < 0 or f[3] != n + nfix:
                    raise Unsupported("destruction term")
                words.append(f)
            dest.append((i, words))
        prod = [(i, scaled(e, "a", lambda j: j)) for i, e in enumerate(mech["prod"])]
        jvs = [scaled(e, "b", lambda j: bmap[j], -1.0) for e in mech["jvs"]]
    except (Unsupported, KeyError):
        return None
    nx = n + nfix + len(ext)
    zero = 8 * (nreact + len(extra))     # the constant 0 behind [RCT | extra]
    one = 8 * (n + nfix)
    if max(8 * nx, zero, 8 * len(coef)) >= 1 << 16:
        return None

    def words4(f):
        return [8 * f[0] | 8 * f[1] << 16, 8 * f[2] | 8 * f[3] << 16]

    def dword(f):          # (f0*f1)*f2, with the constant 1 in the middle of k*v
        p, q = (f[2], f[1]) if f[2] == n + nfix else (f[1], f[2])
        return (8 * f[0] | 8 * p << 16, 8 * q)

    def scaled_words(words):
        return [8 * (w & 0xFFFF) | 8 * (w >> 16) << 16 for w in words]

    no_rate, no_dest, no_sum = (zero | one << 16, one | one << 16), (zero | one << 16, one), 8 * nreact << 16
    segs = {"rate": Segment(nw, no_rate, None).rates([words4(f) for f in rate]),
            "dest": Segment(nw, no_dest).dest([((8 * i, 0), [dword(f) for f in w]) for i, w in dest], split),
            "prod": Segment(nw, no_sum).sums([((8 * i, 0), scaled_words(w)) for i, w in prod], split)}
    # KppDecomp entry by entry: G(i,c) = G(i,c) - sum L(i,j) U(j,c), and for
    # c < i the product with 1/U(c,c); an entry's level is one above those of
    # the factors (and of the pivot) that it reads
    row_of = mech["lu_irow"]
    upd = [[] for _ in range(nnz)]
    for i in range(n):
        for kk in range(crow[i], diag[i]):
            j = icol[kk]
            for jj in range(diag[j] + 1, crow[j + 1]):
                upd[where[(i, icol[jj])]].append((kk, jj))
    # -Jac0 (the coefficients carry the sign); the kernel adds ghinv to the
    # diagonal and forms the reciprocals of the diagonals without updates
    for q, part in enumerate(bpart):
        segs[f"bpart{q}"] = Segment(nw, no_rate, None).rates([words4(f) for f in part])
        segs[f"jvs{q}"] = Segment(nw, no_sum).sums(
            [((8 * p, 0), scaled_words(jvs[p])) for p in range(nnz) if part_of[icol[p]] == q], split)
    elev = [0] * nnz
    for i in range(n):
        for p in range(crow[i], crow[i + 1]):
            c = icol[p]
            lv = max([max(elev[a], elev[b]) + 1 for a, b in upd[p]] + [0])
            if c < i:
                lv = max(lv, elev[diag[c]] + 1)
            elev[p] = lv
    none = 8 * nnz | 8 * nnz << 16       # the constant 0 behind G, times itself
    lu = segs["lu"] = Segment(nw, none, 8 * nnz | 8 * n << 16)
    for k in range(1, max(elev) + 1):
        items = []
        for p in range(nnz):
            if elev[p] == k:
                i, c = row_of[p], icol[p]
                head = (8 * p | 8 * (c if c <= i else n) << 16, L_SCALED if c < i else L_DIAG if c == i else 0)
                items.append((head, [8 * a | 8 * b << 16 for a, b in upd[p]]))
        lu.level(items, split)
    sweep = segs["sweep"] = Segment(nw, 8 * nnz | 8 * n << 16, 8 * n | 8 * n << 16)
    _sweep(sweep, n, [[(icol[p], p) for p in range(crow[i], diag[i])] for i in range(n)], split, True)
    _sweep(sweep, n, [[(icol[p], p) for p in range(diag[i] + 1, crow[i + 1])] for i in range(n)], split, False)
    lu.pad(), sweep.pad()
    return {"segs": segs, "parts": len(parts), "extra": extra, "ext": ext, "coef": coef, "nx": nx,
            "nbp": [len(part) for part in parts],
            "diag": [(8 * diag[i], not upd[diag[i]]) for i in range(n)]}


def coop_inc(mech: dict) -> str:
    """coop.inc: MECH_COOP and, when the programs exist, their C arrays for
    both builds (COOP_SPLIT) and both block sizes, included by one translation
    unit."""
    t = compile_tables(mech)
    if t is None or level_programs(mech, True, 4) is None:
        return "/* no cooperative-kernel tables: unsupported expression shape */\n" \
               "#define MECH_COOP 0\n"

    def arr(ctype, name, vals, space="__device__ const"):
        body = ",".join(str(v) for v in vals) if vals else "0"
        return f"static {space} {ctype} {name}[{max(len(vals), 1)}] = {{{body}}};"

    def doubles(name, vals):
        return arr("double", name, [repr(float(v)) for v in vals] or [0.0])

    lines = ["/* generated cooperative-kernel tables; do not edit */", "#pragma once",
             "#define MECH_COOP 1", f"#define COOP_NUPD {len(t['upd'])}", f"#define COOP_DEPTH {DEPTH}"]
    for split in (False, True):
        lines.append("#if COOP_SPLIT" if split else "#if !COOP_SPLIT")
        for nw in (4, 8):
            p = level_programs(mech, split, nw)
            if nw == 4:
                lines += [f"#define COOP_NX {p['nx']}", f"#define COOP_NEXT {len(p['ext'])}",
                          f"#define COOP_NEXTRA {len(p['extra'])}", f"#define COOP_PARTS {p['parts']}",
                          "#define COOP_NSEG %d" % len(p["segs"]),
                          doubles("coop_ext", p["ext"]),
                          arr("int", "coop_extra_src", [j for j, _ in p["extra"]]),
                          doubles("coop_extra_val", [v for _, v in p["extra"]]),
                          f"#define COOP_NCOEF {len(p['coef'])}", doubles("coop_coef", p["coef"]),
                          "#define COOP_NBP(q) (%s)" % " : ".join(
                              [f"(q) == {k} ? {v}" for k, v in enumerate(p["nbp"])] + ["0"]),
                          arr("int", "coop_diag", [o | (e and 1) for o, e in p["diag"]])]
                lines += [f"#define COOP_SEG_{name.upper()} {k}" for k, name in enumerate(p["segs"])]
            words, where = [], []
            for seg in p["segs"].values():
                for ops in seg.ops:
                    where.append("{%d,%d}" % (len(words) // 4, len(ops)))
                    for op in ops:                   # first four words of the lanes, then the others
                        words += [x for lane in op for x in lane[:4]] + [x for lane in op for x in lane[4:]]
            lines.append(f"static __constant__ int2 coop_seg{nw}[{len(where)}] = {{{','.join(where)}}};")
            lines.append(arr("unsigned int", f"coop_words{nw}", [f"{w}u" for w in words],
                             "__device__ const __align__(16)"))
        lines.append("#endif")
    return "\n".join(lines) + "\n"
