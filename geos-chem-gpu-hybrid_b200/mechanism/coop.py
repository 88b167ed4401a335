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
# Level programs.
#
# The elimination order of a sparse mechanism is a chain of rows, but its
# dependencies are shallow: in fullchem (353 species) the forward sweep has 37
# levels, the backward sweep 33 and the factorisation, taken entry by entry,
# 62.  Every phase of the solver is therefore stored as a program of rounds.
# A round is at most LANES_PER_ROUND lanes; a lane belongs to a group of
# 1, 2, 4 .. 32 consecutive lanes that shares one result, and adds up at most
# K products of it:
#
#     acc (lane 0 of the group: the entry's start value) -= A(word.lo)*B(word.hi)
#
# after which the group is summed by S butterfly exchanges and lane 0 finishes
# the entry.  Rounds of one level need no barrier between them.  The build that
# must round like the reference takes groups of one lane only (each entry's
# terms stay one left-to-right sum, in the reference's order); the production
# build splits long sums (up to 327 terms in fullchem).

LANES_PER_ROUND = 256
NO_WORD = 0xFFFFFFFF
# cost of a round in cycles (round overhead, per product, per exchange): picks
# how far a level's sums are split
ROUND_COST, TERM_COST, FOLD_COST = 60, 12, 45
MAX_TERMS = 16         # most products of one lane where sums are split
CHAIN_MAX = 32         # rows of a warp chain (one lane per row)
BARRIER = 1            # round flag: the block synchronises after the round
CHAIN = 2              # pseudo round: a warp chain


def _group(count, k):
    g = 1
    while g < 32 and -(-count // g) > k:
        g *= 2
    return g


def _pack(items, k, split):
    """Rounds of one level: items [(header, words)] -> [(K, S, lanes)], lanes
    a list of (header, log2 group, words)."""
    sized = []
    for head, words in items:
        g = _group(len(words), k) if split else 1
        sized.append((g, -(-len(words) // g), head, words))
    # aligned groups: wider groups first; alike lanes share a round
    sized.sort(key=lambda x: (-x[0], -x[1]))
    rounds, lanes, kmax, gmax = [], [], 0, 1
    for g, per, head, words in sized:
        if len(lanes) + g > LANES_PER_ROUND:
            rounds.append((kmax, gmax.bit_length() - 1, lanes))
            lanes, kmax, gmax = [], 0, 1
        for q in range(g):
            lanes.append((head, g.bit_length() - 1, words[q::g]))
        kmax, gmax = max(kmax, per), max(gmax, g)
    if lanes:
        rounds.append((kmax, gmax.bit_length() - 1, lanes))
    return rounds


def _level_rounds(items, split):
    best, cost = None, None
    for k in (range(1, MAX_TERMS + 1) if split else (1 << 20,)):
        r = _pack(items, k, split)
        c = sum(ROUND_COST + TERM_COST * kk + FOLD_COST * ss for kk, ss, _ in r)
        if cost is None or c < cost:
            best, cost = r, c
    return best


class Program:
    """Rounds and their table words.  A round's words are its headers (one
    per lane), then K words per lane, lane-contiguous."""

    def __init__(self):
        self.rounds, self.words = [], []

    def level(self, items, split, barrier=True):
        rs = _level_rounds(items, split)
        for n, (k, s, lanes) in enumerate(rs):
            nl = -(-len(lanes) // 32) * 32
            off = len(self.words)
            heads = [NO_WORD] * nl
            cols = [[NO_WORD] * nl for _ in range(k)]
            for v, (head, lg, words) in enumerate(lanes):
                heads[v] = head | lg << 13
                for t, w in enumerate(words):
                    cols[t][v] = w
            self.words += heads + [w for c in cols for w in c]
            self.rounds.append((off, nl, k, s, BARRIER if barrier and n == len(rs) - 1 else 0))

    def chain(self, rows, pos):
        """A warp chain over `rows`: lane r owns row r; step j broadcasts row
        j's value and every lane with an entry (r, j) subtracts its term.
        Words: the rows, the lanes' step masks, then for every two steps the
        lanes' factor positions (low and high half)."""
        m = len(rows)
        off = len(self.words)
        mask = [sum(1 << j for j in range(m) if (r, j) in pos) for r in range(m)]
        pad = [0] * (32 - m)
        self.words += list(rows) + pad + mask + pad
        for j in range(0, m, 2):
            self.words += [pos.get((r, j), 0) | pos.get((r, j + 1), 0) << 16 for r in range(m)] + pad
        self.rounds.append((off, 32, m, 0, CHAIN | BARRIER))


def _sweep(n, deps, split, keep_first):
    """Program of a triangular sweep.  deps[i]: [(column, factor position)] in
    the reference's order.  Runs of levels with at most two rows become warp
    chains (at most CHAIN_MAX rows): first one round level subtracts every
    term whose column lies outside the chain, then one warp walks the chain."""
    lev = [0] * n
    order = list(range(n)) if keep_first else list(range(n - 1, -1, -1))
    for i in order:
        lev[i] = max([lev[c] + 1 for c, _ in deps[i]] + [0])
    nlev = max(lev) + 1 if n else 0
    by = [[i for i in order if lev[i] == l] for l in range(nlev)]
    prog = Program()

    def items(rows, skip=()):
        return [(i, [p | c << 16 for c, p in deps[i] if c not in skip]) for i in rows]

    l = 0
    while l < nlev:
        e = l
        if split and (l > 0 or not keep_first):
            rows = 0
            while e < nlev and len(by[e]) <= (4 if e == 0 else 2) and rows + len(by[e]) <= CHAIN_MAX:
                rows += len(by[e])
                e += 1
        if e - l >= 4:
            rows = [i for k in range(l, e) for i in by[k]]
            inside = {i: r for r, i in enumerate(rows)}
            bulk = [it for it in items(rows, inside) if it[1]]
            if bulk:
                prog.level([(h | 1 << 28, w) for h, w in bulk], split)
            prog.chain(rows, {(inside[i], inside[c]): p for i in rows for c, p in deps[i] if c in inside})
            l = e
            continue
        it = items(by[l])
        if l == 0 and keep_first:
            it = []                  # the forward sweep leaves level 0 as it is
        if it:
            prog.level(it, split)
        l += 1
    return prog


def level_programs(mech: dict, split: bool):
    """The cooperative kernel's programs, or None for unsupported expression
    shapes.  split: sums may be divided over lanes (production build)."""
    if compile_tables(mech) is None:
        return None
    n, nfix, nnz, nreact = mech["nvar"], mech["nfix"], mech["nnz"], mech["nreact"]
    crow, diag, icol, where = mech["lu_crow"], mech["lu_diag"], mech["lu_icol"], mech["lu_where"]
    if nnz >= 1 << 13 or n >= 1 << 12:
        return None
    extra = {}                 # first factors behind the rate constants: (reaction or
                               # -1, literal), the literal itself or RCT(j)*literal
    ext = {1.0: 0}             # constants behind the species (other factors)
    coef = {1.0: 0}            # coefficients of the sums

    def slot(table, value):
        return table.setdefault(value, len(table))

    def product(node):
        """(first, f1, f2, f3): first indexes [RCT | extra], the others
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
        bmap = {m: k for k, (m, _) in enumerate(mech["jac_b"])}
        bpart = [product(e) for _, e in mech["jac_b"]]
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
    nrx = nreact + len(extra)
    if nx >= 1 << 10 or nrx >= 1 << 11 or len(bpart) >= 1 << 16:
        return None
    pd = Program()
    pd.level([(i, [f[0] | f[1] << 11 | f[2] << 21 for f in w]) for i, w in dest], split, False)
    pp = Program()
    pp.level(prod, split)
    # -Jac0 (the coefficients carry the sign), ghinv on the diagonal; bit 28:
    # a diagonal without updates, whose reciprocal is formed here
    upd = [[] for _ in range(nnz)]
    for i in range(n):
        for kk in range(crow[i], diag[i]):
            j = icol[kk]
            for jj in range(diag[j] + 1, crow[j + 1]):
                upd[where[(i, icol[jj])]].append((kk, jj))
    row_of = mech["lu_irow"]
    pj = Program()
    items = []
    for p in range(nnz):
        h = p
        if p == diag[row_of[p]]:
            h |= (row_of[p] + 1) << 16 | (0 if upd[p] else 1 << 28)
        items.append((h, jvs[p]))
    pj.level(items, split)
    # KppDecomp entry by entry: G(i,c) = G(i,c) - sum L(i,j) U(j,c), and for
    # c < i the product with 1/U(c,c); an entry's level is one above those of
    # the factors (and of the pivot) that it reads
    elev = [0] * nnz
    for i in range(n):
        for p in range(crow[i], crow[i + 1]):
            c = icol[p]
            lv = max([max(elev[a], elev[b]) + 1 for a, b in upd[p]] + [0])
            if c < i:
                lv = max(lv, elev[diag[c]] + 1)
            elev[p] = lv
    pl = Program()
    for l in range(1, max(elev) + 1):
        items = []
        for p in range(nnz):
            if elev[p] == l:
                i, c = row_of[p], icol[p]
                h = p | c << 16 | (1 << 28 if c < i else (1 << 29 if c == i else 0))
                items.append((h, [a | b << 16 for a, b in upd[p]]))
        pl.level(items, split)
    lower = [[(icol[p], p) for p in range(crow[i], diag[i])] for i in range(n)]
    upper = [[(icol[p], p) for p in range(diag[i] + 1, crow[i + 1])] for i in range(n)]
    return {"rate": rate, "bpart": bpart, "extra": extra, "ext": ext, "coef": coef, "nx": nx,
            "dest": pd, "prod": pp, "jvs": pj, "lu": pl,
            "fwd": _sweep(n, lower, split, True), "bwd": _sweep(n, upper, split, False)}


PROGRAMS = ("dest", "prod", "jvs", "lu", "fwd", "bwd")


def coop_inc(mech: dict) -> str:
    """coop.inc: MECH_COOP and, when the programs exist, their C arrays for
    both builds (COOP_SPLIT), included by one translation unit."""
    t = compile_tables(mech)
    progs = None if t is None else {sp: level_programs(mech, sp) for sp in (False, True)}
    if t is None or progs[True] is None:
        return "/* no cooperative-kernel tables: unsupported expression shape */\n" \
               "#define MECH_COOP 0\n"

    def arr(ctype, name, vals, align="", space="__device__ const"):
        body = ",".join(str(v) for v in vals) if vals else "0"
        return f"static {space} {align}{ctype} {name}[{max(len(vals), 1)}] = {{{body}}};"

    def doubles(name, table):
        return arr("double", name, [repr(float(v)) for v in table])

    lines = ["/* generated cooperative-kernel tables; do not edit */", "#pragma once",
             "#define MECH_COOP 1", f"#define COOP_NUPD {len(t['upd'])}"]
    for sp in (False, True):
        p = progs[sp]
        lines.append("#if COOP_SPLIT" if sp else "#if !COOP_SPLIT")
        lines += [f"#define COOP_NX {p['nx']}", f"#define COOP_NEXT {len(p['ext'])}",
                  f"#define COOP_NEXTRA {len(p['extra'])}", f"#define COOP_NCOEF {len(p['coef'])}",
                  f"#define COOP_NBP {len(p['bpart'])}",
                  doubles("coop_ext", p["ext"]),
                  arr("int", "coop_extra_src", [j for j, _ in p["extra"]]),
                  doubles("coop_extra_val", [v for _, v in p["extra"]] or [0.0]),
                  doubles("coop_coef", p["coef"]),
                  arr("unsigned short", "coop_rate", [x for f in p["rate"] for x in f], "__align__(8) "),
                  arr("unsigned short", "coop_bpart", [x for f in p["bpart"] for x in f], "__align__(8) ")]
        rounds = []
        for name in PROGRAMS:
            pr = p[name]
            lines.append(f"#define COOP_R0_{name.upper()} {len(rounds)}")
            rounds += pr.rounds
            lines.append(f"#define COOP_R1_{name.upper()} {len(rounds)}")
            lines.append(arr("unsigned int", f"coop_w_{name}", [f"{w}u" for w in pr.words]))
        body = ",".join("{%d,%d}" % (off, nl | k << 10 | s << 20 | f << 24) for off, nl, k, s, f in rounds)
        lines.append(f"static __constant__ int2 coop_round[{len(rounds)}] = {{{body}}};")
        lines.append("#endif")
    return "\n".join(lines) + "\n"
