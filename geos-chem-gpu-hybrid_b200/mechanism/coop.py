"""Programs for the cooperative kernel (one thread block per cell).

The one-thread-per-cell kernels run straight-line statement lists.  In the
cooperative kernel the warps of a block share one cell, and each executes its
own list of operations on the cell's arrays.  ``level_programs`` turns the
mechanism IR into those lists, ``coop_inc`` emits them as C arrays.  The two
forms (split or not), the levels, the inverses of the sweeps and the format of
the words are described where they are built.

``compile_tables`` holds the expressions themselves as flat tables, with the
factorisation and the solves as lists of updates in the reference's order.  The
kernel does not read them: they refuse expressions of an unknown shape, and the
CPU tests evaluate them as the plain form of what the programs compute.

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

Factorisation and solves.  Each entry of KppDecomp
(gckpp_LinearAlgebra.F90:46-84) receives its updates in increasing pivot order,
each row of KppSolve (:645-2311) its terms in the reference's order, with the
same operations: the results of the unsplit programs are the reference's bit
for bit, whatever the order in which independent entries are formed.
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


def _pack(lo, hi):
    """Two 16-bit fields of a word; a field that does not fit must not spill
    into the other."""
    if not (0 <= lo < 1 << 16 and 0 <= hi < 1 << 16):
        raise Unsupported("offset of more than 16 bits")
    return lo | hi << 16


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
    """The mechanism's plain tables (see the module's docstring), or None when
    some expression falls outside the supported shapes."""
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
# 61.  Every phase of the solver is therefore a program of levels; the entries
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
# in shared memory), so that a word needs no arithmetic, or, in a mechanism whose
# arrays are beyond 64 KB, as indices that the kernel multiplies (COOP_UNIT); a
# missing operand points at a constant 0 (or 1) behind the array, so that it needs no test.
#
#   rate operations   four products (f0 | f1<<16, f2 | f3<<16).  Product k of
#                     operation i of warp w and lane l is number
#                     ((i*4 + k)*NW + w)*32 + l.
#   sum operations    two halves of a header and three words (jvs)
#   single operations four pairs (entry | coefficient<<16, partial)
#   level operations  header, control, six words (dest, prod, lu, sweep)
#
# Control word, per lane: L_* flags, log2 of the lane's group, exchanges that
# the warp does (the largest of its groups), products in use, block barriers
# after the operation.  A sum's header is its entry's offset | control << 16; a
# level's is the entry's offset | the offset of its scale << 16.
#
# The sweeps of the production build use partitioned inverses (Alvarado and
# Schreiber, Optimal parallel solution of sparse triangular systems, 1993):
# consecutive levels form a part whose rows get the entries of the inverse of
# their diagonal block, so that a part is solved by one level (its rows'
# products with the inverse) after one level that subtracts the terms outside
# the part.  fullchem: two parts of each sweep and the tail block, 9 levels
# instead of 69.  The inverses are rows
# of the same recurrence as the factors and are formed by the factorisation's
# program, next to the entries that become final at the same level:
#
#   forward, unit diagonal   V(i,j) = L(i,j) - sum_c L(i,c) V(c,j),
#                            x_i = b_i - sum_j V(i,j) b_j
#   backward                 T(i,j) = (U(i,j) R_j - sum_c U(i,c) T(c,j)) R_i,
#                            x_i = R_i b_i - sum_j T(i,j) b_j,   R = 1/U(i,i)
#
# with c over the row's columns inside the part.
#
# The last rows are nearly dense and their pivots follow one another, two
# levels each (fullchem: 49 of the 61 levels belong to the last 32 rows).  They
# are left out of the levels: the program only forms their Schur complement,
# which one block-wide Gauss-Jordan elimination turns into its negative inverse,
# rows over warps and columns over lanes; the sweeps then need one level for
# these rows.
#
# The factor array of a cell is [G | tail block | V and T | -R | -1 | 0]; the
# vector array is [X | 0 | Z], where a row's solution goes to the other half
# when its part's rows are still read.
#
# The order of the terms of Fun's sums is the reference's in every build: the
# difference of production and destruction is where their rounding is amplified
# most (a step size of a sensitive cell moves by 1e-7 relative when these sums
# are split over lanes, by 1e-8 when all the others are).  Long ones are formed
# in two passes: all threads write their products one after the other into a
# buffer, then one lane per sum adds them up, two instructions per term.

WORDS = 8
DEPTH = 4              # operations fetched ahead; a segment is a multiple of it
L_LEAD, L_FIRST, L_END, L_START, L_DIAG, L_SCALED = 1, 2, 4, 8, 16, 32
L_DIAGS = 1 << 15      # some lane of the warp has L_DIAG
L_GROUP, L_FOLD, L_USED, L_SYNC = 6, 9, 12, 20
# cycles of an operation: fixed part, per product, per exchange, end of an
# entry (an operation of six products and three exchanges measures ~650 on a
# B200); they steer how far sums are split and which parts get inverses
OP_COST, TERM_COST, FOLD_COST, END_COST = 250, 25, 45, 60


BLOCK = 8              # terms that a chain adds between two tests of its length
NO_ENTRY = 0xFFFF      # single operations: an idle pair
# The discrete adjoint adds four segments: the transposed sweeps (U^T, then L^T;
# the parts in reverse, each [terms outside the part, product with the
# transposed inverse]), t_j = S_j . u per reaction (tj), the partials
# dA(j)/dV(i) of every rate (apart), and per species the sums of t_j times a
# partial and of t_j times its derivative along a stage vector (vthl).
ADJOINT = ("sweept", "tj", "apart", "vthl")

LONG = 60              # terms of Fun's sums above which a sum goes through the buffer


def _lanes(items, k, split, dense=False):
    """Warp rounds of one level: [(header, words)] -> lists of at most 32
    (header, log2 group, words of the lane), groups aligned to their size.
    dense: the items are rows of the tail block, a multiple of 16 doubles apart;
    each starts with another column, or all rows' entries of a column, which are
    in one bank of shared memory, would be read together (synthetic mechanism:
    13,400 passes of a half warp's loads per attempt in the sweeps, 6,200 so)."""
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
        if dense:
            turn = len(lanes) % len(words)
            words = words[turn:] + words[:turn]
        lanes += [(head, g.bit_length() - 1, words[q::g]) for q in range(g)]
    if lanes:
        rounds.append(lanes)
    return rounds


def _cost(lanes, per_op):
    k = max(len(w) for _, _, w in lanes)
    s = max(lg for _, lg, _ in lanes)
    return OP_COST * max(1, -(-k // per_op)) + TERM_COST * k + FOLD_COST * s + END_COST


def _place(items, nw, split, per_op, dense=False):
    """A level's rounds on nw warps: (warp lists, cost of the longest)."""
    best, cost = None, None
    longest = max([len(w) for _, w in items] + [1])
    for k in (range(1, min(longest, 40) + 1) if split else (longest,)):
        warps, load = [[] for _ in range(nw)], [0] * nw
        for lanes in sorted(_lanes(items, k, split, dense), key=lambda r: -_cost(r, per_op)):
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
                    lead = flags & ~L_START if x % (1 << lg) else flags | L_LEAD
                    out.append((head, ctl | lead | lg << L_GROUP, w + [self.none] * (per_op - len(w))))
                else:
                    out.append((self.head, ctl, [self.none] * per_op))
            yield out

    def lines(self, items):
        """Sums of one lane each, six products an operation; no barrier."""
        warps, self.cost = _place(items, self.nw, False, 6)
        for v, rounds in enumerate(warps):
            for lanes in rounds:
                for op in self._split(lanes, 6):
                    self.ops[v].append([[h, c] + w for h, c, w in op])
        return self.pad()

    def sums(self, items, split):
        warps, self.cost = _place(items, self.nw, split, 3)
        idle = [(self.head, 0, [self.none] * 3)] * 32
        for v, rounds in enumerate(warps):
            halves = [op for lanes in rounds for op in self._split(lanes, 3)]
            if len(halves) % 2:
                halves.append(idle)
            for a, b in zip(halves[::2], halves[1::2]):
                self.ops[v].append([[_pack(h, c & 0xFFF)] + w + [_pack(g, d & 0xFFF)] + u
                                    for (h, c, w), (g, d, u) in zip(a, b)])
        return self.pad([self.head] + [self.none] * 3 + [self.head] + [self.none] * 3)

    def singles(self, items):
        """Entries of one product: four (entry | coefficient<<16, partial)
        pairs per lane."""
        for n, (head, word) in enumerate(items):
            v, w = n // 32 % self.nw, n // (32 * self.nw)
            if w % 4 == 0 and len(self.ops[v]) == w // 4:
                self.ops[v].append([self.idle() for _ in range(32)])
            self.ops[v][w // 4][n % 32][w % 4 * 2:w % 4 * 2 + 2] = [_pack(head, word & 0xFFFF), word >> 16]
        return self.pad()

    def level(self, items, split, dense=False):
        warps, cost = _place(items, self.nw, split, 6, dense)
        self.cost += cost + 30
        for v, rounds in enumerate(warps):
            for lanes in rounds:
                diags = L_DIAGS if any(flags & L_DIAG for (_, flags), _, _ in lanes) else 0
                for op in self._split(lanes, 6):
                    self.ops[v].append([[h, c | diags] + w for h, c, w in op])
        self._sync()

    def in_units(self, unit):
        """Element indices (both halves of headers and words) as offsets."""
        def offsets(w):
            return _pack(unit * (w & 0xFFFF), unit * (w >> 16))

        for ops in self.ops:
            for op in ops:
                for lane in op:
                    lane[0] = offsets(lane[0])
                    lane[2:] = [offsets(w) for w in lane[2:]]
        self.none = offsets(self.none)
        return self.pad()

    def _sync(self):
        """A block barrier after everything so far."""
        for ops in self.ops:
            if not ops:
                ops.append([self.idle() for _ in range(32)])
            for lane in ops[-1]:
                lane[1] += 1 << L_SYNC


def _sweep_levels(n, deps, order):
    lev = [0] * n
    for i in order:
        lev[i] = max([lev[c] + 1 for c, _ in deps[i] if c < n] + [0])
    return lev


def _parts(n, deps, order, limit):
    """Parts of a triangular sweep: runs of levels whose diagonal block's
    inverse has at most `limit` entries more than the block.  Returns [(rows in
    order, {row: columns of its inverse inside the part})]."""
    lev = _sweep_levels(n, deps, order)
    nlev = max(lev) + 1 if n else 0

    def part(k, e):
        rows = sorted((i for i in order if k <= lev[i] < e), key=lambda i: lev[i])
        inside, reach, fill = set(rows), {}, 0
        for i in rows:
            cols = [c for c, _ in deps[i] if c in inside]
            reach[i] = set(cols).union(*[reach[c] for c in cols])
            fill += len(reach[i]) - len(cols)
        return rows, reach, fill

    out, k = [], 0
    while k < nlev:
        e = k + 1
        while e < nlev and part(k, e + 1)[2] <= limit:
            e += 1
        out.append(part(k, e)[:2])
        k = e
    return out


SHARED = 227 * 1024 // 8    # doubles of shared memory that a block may have


def cell_doubles(ng, nx, n, nreact, nextra, buffer):
    """Shared memory of a cell (CoopAt in csrc/coop.cu)."""
    products = (ng + 1 + nx + 2 * n + 2 + nreact + 1 + nreact + nextra + 2) // 2 * 2
    return (products + buffer + 10) // 2 * 2


def level_programs(mech: dict, split: bool, nw: int):
    """The cooperative kernel's programs, or None for expression shapes or
    sizes that they do not hold.  split: sums may be divided over lanes
    (production build); nw: warps of the block."""
    try:
        return _fitting_programs(mech, split, nw)
    except Unsupported:
        return None


def _fitting_programs(mech, split, nw):
    """Offsets are in bytes where 16 bits hold them, else in doubles ("unit").
    A cell that does not fit in shared memory goes without the buffer of the
    long sums, then without the tail block; the inverses of the sweeps' parts
    are chosen within what is left.  What is taken does not depend on nw."""
    why = None
    for long, with_tail in ((LONG, True), (1 << 30, True), (1 << 30, False)):
        for unit in (8, 1):
            try:
                return _programs(mech, split, nw, unit, long, with_tail)
            except Unsupported as e:
                why = why or e
    raise why


def _programs(mech, split, nw, unit, long, with_tail):
    if compile_tables(mech) is None:
        raise Unsupported("expression shape")
    n, nfix, nnz, nreact = mech["nvar"], mech["nfix"], mech["nnz"], mech["nreact"]
    crow, diag, icol, where = mech["lu_crow"], mech["lu_diag"], mech["lu_icol"], mech["lu_where"]
    extra = {}                 # first factors behind the rate constants: (reaction or
                               # -1, literal), the literal itself or RCT(j)*literal
    ext = {1.0: 0}             # constants behind the species (other factors)
    coef = {1.0: 0}            # coefficients of the sums

    def slot(table, value):
        return table.setdefault(value, len(table))

    def product(node, sign=1.0):
        """[first, f1, f2, f3]: first indexes [RCT | extra], the others
        [V | FIX | ext]; missing factors are the constant 1, whose product
        is exact.  A leading RCT(j)*literal is formed once per cell.  A
        negative sign goes into the first factor, which rounds alike."""
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
            first, fs = nreact + slot(extra, (f0[1], sign * num(fs[1]))), fs[1:]
        elif f0[0] == "k":
            first = f0[1] if sign > 0 else nreact + slot(extra, (f0[1], sign))
        elif f0[0] == "n":
            first = nreact + slot(extra, (-1, sign * num(f0)))
        else:                  # 1*v is exact
            first, fs = nreact + slot(extra, (-1, sign)), [None] + fs
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
            words.append(_pack(slot(coef, c), index(t[1])))
        return words

    try:
        rate = [product(e) for e in mech["rates"]]
        # partials B are formed for a part of the columns at a time, as many as
        # the rates' scratch array holds; each feeds one column of the Jacobian
        # as KPP writes them, one read by several is formed for each
        column = [set() for _ in range(n)]
        for p, e in enumerate(mech["jvs"]):
            column[icol[p]].update(codegen._refs(e, "b"))
        bexpr = dict.fromkeys(range(mech["nb"]), ["n", "0"])
        bexpr.update(mech["jac_b"])
        parts, part_of, bmap = [[]], {}, {}
        for c in range(n):
            if len(parts[-1]) + len(column[c]) > nreact:
                parts.append([])
            part_of[c] = len(parts) - 1
            for b in sorted(column[c]):
                bmap[(b, c)] = len(parts[-1])
                parts[-1].append(b)
        if max(len(part) for part in parts) > nreact:
            raise Unsupported("column with too many partials")
        bpart = [[product(bexpr[b]) for b in part] for part in parts]
        dest = []
        for i, e in enumerate(mech["dest"]):
            words = []
            for sign, t in signed(e):
                if t[0] == "n" and float(codegen.literal(t[1])) == 0.0 and not words:
                    continue
                words.append(product(t, sign))
            dest.append((i, words))
        prod = [(i, scaled(e, "a", lambda j: j)) for i, e in enumerate(mech["prod"])]
        jvs = [scaled(e, "b", lambda j, c=c: bmap[(j, c)], -1.0) for e, c in zip(mech["jvs"], icol)]
    except KeyError as e:
        raise Unsupported(f"missing partial {e}") from None
    nx = n + nfix + len(ext)
    zero = unit * (nreact + len(extra))  # the constant 0 behind [RCT | extra]
    one = unit * (n + nfix)

    def words4(f):
        return [_pack(unit * f[0], unit * f[1]), _pack(unit * f[2], unit * f[3])]

    def scaled_words(words):
        return [_pack(unit * (w & 0xFFFF), unit * (w >> 16)) for w in words]

    no_rate, no_sum = (_pack(zero, one), _pack(one, one)), _pack(0, unit * nreact)
    segs = {"rate": Segment(nw, no_rate, None).rates([words4(f) for f in rate]),
            "dest": None, "bufd": None, "prod": None, "bufp": None}
    # a destruction term of three factors or more has no place in a line's words
    long_d = [i for i, w in dest if len(w) > long and split or
              any(sum(x != n + nfix for x in f[1:]) > 1 for f in w)]
    long_p = [i for i, w in prod if len(w) > long and split or i in long_d]
    # the buffer: the long sums' products, each sum padded to whole blocks
    first = {}

    def buffer(key, sums, none, at):
        out = []
        for c, (i, words) in enumerate(sums):
            # the lanes' pairs of products start in different banks
            out += [none] * ((2 * c - at - len(out)) % 16)
            first[(key, i)] = (at + len(out), -(-len(words) // BLOCK))
            out += words + [none] * (-len(words) % BLOCK)
        return out

    rates_d = buffer("d", [(i, [words4(f) for f in w]) for i, w in dest if i in long_d], list(no_rate), 0)
    ones_p = buffer("p", [(i, scaled_words(w)) for i, w in prod if i in long_p], no_sum, len(rates_d))
    if not long_p:
        del segs["bufd"], segs["bufp"]
    segs["dest"] = Segment(nw, _pack(zero, one)).lines(
        [((unit * i, 0), [_pack(unit * f[0], unit * next((x for x in f[1:] if x != n + nfix), n + nfix)) for f in w])
         for i, w in dest if i not in long_d])
    if long_p:
        segs["bufd"] = Segment(nw, no_rate, None).rates(rates_d)
    segs["prod"] = Segment(nw, no_sum).lines([((unit * i, 0), scaled_words(w)) for i, w in prod if i not in long_p])
    if long_p:
        segs["bufp"] = Segment(nw, (NO_ENTRY, unit * nreact), None).singles(
            [(unit * (len(rates_d) + k), w) for k, w in enumerate(ones_p)])
    # chain l of lane l % 32: species, first product, blocks
    chains = [[(i,) + first[(key, i)] for i in rows] for key, rows in (("d", long_d), ("p", long_p))]
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
    # the tail block: its entries live in a dense array behind G
    tail = _tail_rows(n, row_of, icol, nreact) if split and with_tail else 0
    t0 = n - tail
    in_tail = [row_of[p] >= t0 and icol[p] >= t0 for p in range(nnz)]
    block = nnz - sum(in_tail)
    place = [0] * nnz                    # where an entry of the LU pattern lives
    for k, p in enumerate(p for p in range(nnz) if not in_tail[p]):
        place[p] = k
    for p in range(nnz):
        if in_tail[p]:
            place[p] = block + (row_of[p] - t0) * tail + icol[p] - t0
    if unit * (block + tail * tail) > NO_ENTRY:
        raise Unsupported("tail block")
    # -Jac0 (the coefficients carry the sign); the kernel adds ghinv to the
    # diagonal and forms the reciprocals of the diagonals without updates
    fill = set(range(block, block + tail * tail)) - {place[p] for p in range(nnz)}
    for q, part in enumerate(bpart):
        mine = [(unit * place[p], scaled_words(jvs[p])) for p in range(nnz) if part_of[icol[p]] == q]
        mine += [(unit * p, []) for p in sorted(fill)] if q == 0 else []
        segs[f"bpart{q}"] = Segment(nw, no_rate, None).rates([words4(f) for f in part])
        segs[f"jvs{q}"] = Segment(nw, no_sum).sums([((h, 0), w) for h, w in mine if len(w) > 1], split)
        segs[f"one{q}"] = [(h, w[0] if w else no_sum) for h, w in mine if len(w) <= 1]
    lower = [[(icol[p], place[p]) for p in range(crow[i], diag[i])] for i in range(n)]
    upper = [[(icol[p], place[p]) for p in range(diag[i] + 1, crow[i + 1])] for i in range(n)]
    # entries (row, column, place, updates by the pivots before the tail)
    entries = [(row_of[p], icol[p], place[p], [(place[a], place[b]) for a, b in upd[p] if icol[a] < t0])
               for p in range(nnz)]
    at_diag = [place[p] for p in diag]
    buffered = len(rates_d) + len(ones_p)
    coefs = len(coef) + len(coef) % 2

    def fits(ng):
        return unit * ng < 1 << 16 and coefs + cell_doubles(ng, nx, n, nreact, len(extra), buffered) <= SHARED

    limits = None
    if split:
        tried = [(f, u) for f in INVERSE_LIMITS for u in INVERSE_LIMITS]
        tried = [lim for lim in tried if fits(_factor_and_sweeps(
            n, tail, block, entries, at_diag, lower, upper, split, nw, lim, True)["ng"])]
        if not tried:
            raise Unsupported("cell beyond 16-bit offsets or the shared memory of a block")
        limits = min(tried, key=lambda lim: _factor_and_sweeps(
            n, tail, block, entries, at_diag, lower, upper, split, nw, lim, True)["cost"])
    best = _factor_and_sweeps(n, tail, block, entries, at_diag, lower, upper, split, nw, limits)
    if not fits(best["ng"]):
        raise Unsupported("cell beyond 16-bit offsets or the shared memory of a block")
    for f in ("lu", "sweep", "sweept"):
        if f in best:
            best[f].pad().in_units(unit)
    for q in range(len(bpart)):
        segs[f"one{q}"] = Segment(nw, (NO_ENTRY, unit * nreact), None).singles(segs[f"one{q}"])
    segs["lu"], segs["sweep"] = best["lu"], best["sweep"]
    extra_of = [j for j, _ in extra]
    scoef, apart, by_species = {1.0: 0}, [], [[] for _ in range(n)]
    if split:
        one_x = n + nfix
        for j, f in enumerate(rate):
            for k in (1, 2, 3):
                if f[k] < n:
                    rest = [x for q, x in enumerate(f) if q not in (0, k)]
                    by_species[f[k]].append(_pack(unit * j, unit * len(apart)))
                    apart.append([f[0]] + rest + [one_x])
        react = [[] for _ in range(nreact)]
        for i, j, v in mech["stoich"]:
            react[j].append(_pack(unit * slot(scoef, float(codegen.literal(v))), unit * i))
        segs["sweept"] = best["sweept"]
        segs["tj"] = Segment(nw, _pack(0, unit * n)).sums([((unit * j, 0), w) for j, w in enumerate(react)], True)
        segs["apart"] = Segment(nw, no_rate, None).rates([words4(f) for f in apart])
        segs["vthl"] = Segment(nw, _pack(unit * nreact, unit * len(apart))).sums(
            [((unit * i, 0), w) for i, w in enumerate(by_species)], True)
    return {"segs": segs, "unit": unit, "parts": len(parts), "cell": cell_doubles(best["ng"], nx, n, nreact, len(extra), buffered), "extra": extra, "ext": ext, "coef": coef, "nx": nx,
            "nbp": [len(part) for part in parts], "ng": best["ng"], "place": best["place"], "tail": tail,
            "chains": chains, "buffer": buffered, "nbufd": len(rates_d), "factor": place, "block": block, "diag": [(at_diag[i], i < t0 and not upd[diag[i]]) for i in range(n)],
            "cost": best["cost"], "scoef": scoef, "napart": len(apart), "place_t": best["place_t"],
            "has_k": [int(f[0] < nreact or extra_of[f[0] - nreact] >= 0) for f in rate]}


# most entries that a part's inverse may add; every pair is tried
INVERSE_LIMITS = (0, 50, 100, 200, 400)


def _tail_rows(n, row_of, icol, nreact):
    """Rows of the tail block: 64 where they are dense, else 32; the rates'
    scratch array hands over two of them at a time."""
    for m, least in ((64, 0.9), (32, 0.0)):
        if n >= 2 * m - 8 and nreact >= 2 * m and sum(r >= n - m and c >= n - m for r, c in zip(row_of, icol)) >= least * m * m:
            return m
    return 0


def _factor_and_sweeps(n, tail, block, entries, diag, lower, upper, split, nw, limits, estimate=False):
    """The factorisation's program (with the inverses of the sweeps' parts) and
    the sweeps' one, for one choice of parts; estimate: only their cost, the
    factorisation's from the products per level."""
    t0 = n - tail
    if 2 * n + 2 >= 1 << 16:
        raise Unsupported("vector of the sweeps beyond 16-bit indices")
    fwd, bwd = ([], []) if limits is None else \
        (_parts(t0, lower, range(t0), limits[0]), _parts(t0, upper, range(t0 - 1, -1, -1), limits[1]))
    at = {}                                # (row, column) -> index of V or T
    for parts in (fwd, bwd):
        for rows, reach in parts:
            for i in rows:
                for j in sorted(reach[i]):
                    at[(i, j)] = block + tail * tail + len(at)
    rbase = block + tail * tail + len(at)    # -R, then -1, then 0
    minus, zero = rbase + n, rbase + n + 1
    if zero >= 1 << 16 and not estimate:
        raise Unsupported("factors beyond 16-bit indices")
    # nodes: index, start value read, scale, flags, products
    level, nodes = {minus: 0}, []

    def node(index, start, scale, flags, terms):
        lv = max([max(level[a], level[b]) + 1 for a, b in terms] + [0])
        if scale != minus and not flags & L_DIAG:
            lv = max(lv, level[scale] + 1)
        level[index] = lv
        if flags & L_DIAG:
            level[scale] = lv
        if lv:
            nodes.append((lv, index, start, scale, flags, terms))

    for i, c, p, terms in entries:
        if c < i and c < t0:
            node(p, True, rbase + c if split else diag[c], L_SCALED, terms)
        elif c == i and i < t0:
            node(p, True, rbase + c, L_DIAG, terms)
        else:
            node(p, True, minus, 0, terms)
    for rows, reach in fwd:
        for i in rows:
            for j in sorted(reach[i]):
                terms = [(p, minus) for c, p in lower[i] if c == j]
                terms += [(p, at[(c, j)]) for c, p in lower[i] if c > j and (i, c) in at and (c, j) in at]
                node(at[(i, j)], False, minus, 0, terms)
    for rows, reach in bwd:
        for i in rows:
            for j in sorted(reach[i]):
                terms = [(p, rbase + j) for c, p in upper[i] if c == j]
                terms += [(p, at[(c, j)]) for c, p in upper[i] if c < j and (i, c) in at and (c, j) in at]
                node(at[(i, j)], False, rbase + i, L_SCALED, terms)
    lu = Segment(nw, zero | zero << 16, zero | minus << 16)
    last = max(level.values())
    if estimate:
        work = [0] * (last + 1)
        for lv, _, _, _, _, terms in nodes:
            work[lv] += len(terms)
        lu.cost = sum(400 + 70 * w // (32 * nw) for w in work)
        nodes, last = [], 0
    by = [[] for _ in range(last + 1)]
    work = [0] * (last + 1)
    late = []
    for lv, index, start, scale, flags, terms in nodes:
        early = [t for t in terms if max(level[t[0]], level[t[1]]) + 1 <= lv - EARLY] if split else []
        if len(early) < 3:
            early = []
        rest = [t for t in terms if t not in early] if early else terms
        by[lv].append((index, start or bool(early), scale, flags, rest))
        work[lv] += len(rest)
        if early:
            late.append((max(max(level[a], level[b]) + 1 for a, b in early), lv, index, start, early))
    # the bulk of a long sum runs at the emptiest level between its operands
    # and its end, so that the end is short
    for lo, hi, index, start, early in sorted(late, key=lambda x: -len(x[4])):
        k = min(range(lo, hi), key=lambda q: (work[q], q))
        by[k].append((index, start, minus, 0, early))
        work[k] += len(early)
    for k in range(1, last + 1):
        lu.level([((index | scale << 16, flags | (L_START if start else 0)), [a | b << 16 for a, b in terms])
                  for index, start, scale, flags, terms in by[k]], split)
    sweep = Segment(nw, zero | n << 16, n | minus << 16)
    x = list(range(n))                     # where a row's current value is
    if limits is None:
        for deps, order, scaled in ((lower, range(n), False), (upper, range(n - 1, -1, -1), True)):
            lev = _sweep_levels(n, deps, order)
            for k in range(0 if scaled else 1, max(lev) + 1):
                sweep.level([((i | (diag[i] if scaled else minus) << 16, L_START | (L_SCALED if scaled else 0)),
                              [p | c << 16 for c, p in deps[i]]) for i in order if lev[i] == k], split)
    for parts, deps, scaled in ((fwd, lower, False), (bwd, upper, True)):
        for rows, reach in parts:
            inside = set(rows)
            out = [(i, [p | x[c] << 16 for c, p in deps[i] if c not in inside]) for i in rows]
            out = [((x[i] | minus << 16, L_START), w) for i, w in out if w]
            if out:
                sweep.level(out, split)
            new, items = list(x), []
            for i in rows:
                if scaled or reach[i]:
                    new[i] = (x[i] + n + 1) % (2 * n + 2)
                    items.append(((new[i] | minus << 16, 0), [(rbase + i if scaled else minus) | x[i] << 16] +
                                  [at[(i, j)] | x[j] << 16 for j in sorted(reach[i])]))
            if items:
                sweep.level(items, split)
            x = new
        if tail and not scaled:            # the tail block, once both sweeps reach it
            out = [(i, [p | x[c] << 16 for c, p in lower[i] if c < t0]) for i in range(t0, n)]
            sweep.level([((x[i] | minus << 16, L_START), w) for i, w in out if w], split)
            new = [i if i < t0 else i + n + 1 for i in range(n)]
            sweep.level([((new[i] | minus << 16, 0),
                          [block + (i - t0) * tail + j - t0 | x[j] << 16 for j in range(t0, n)])
                         for i in range(t0, n)], split, True)
            x = x[:t0] + new[t0:]
    out = {"lu": lu, "sweep": sweep, "ng": zero, "place": x, "cost": lu.cost + 4 * sweep.cost}
    if limits is not None and not estimate:
        out["sweept"], out["place_t"] = _transposed(n, tail, block, fwd, bwd, lower, upper, at, rbase, split, nw)
    else:
        out["place_t"] = x
    return out


def _transposed(n, tail, block, fwd, bwd, lower, upper, at, rbase, split, nw):
    """The sweeps with the transposed matrix on the same factors and inverses."""
    t0, minus, zero = n - tail, rbase + n, rbase + n + 1
    seg = Segment(nw, zero | n << 16, n | minus << 16)
    x = list(range(n))

    def columns(deps):
        cols = [[] for _ in range(n)]
        for i in range(n):
            for c, p in deps[i]:
                cols[c].append((i, p))
        return cols

    def outside(rows, cols, done):
        out = [((x[c] | minus << 16, L_START), [p | x[i] << 16 for i, p in cols[c] if done(i)]) for c in rows]
        out = [it for it in out if it[1]]
        if out:
            seg.level(out, split)

    def product(items):
        """items {row: words}: the rows' values go to their other place."""
        nonlocal x
        new = list(x)
        for j in items:
            new[j] = (x[j] + n + 1) % (2 * n + 2)
        if items:
            seg.level([((new[j] | minus << 16, 0), w) for j, w in items.items()], split)
        x = new

    for parts, deps, scaled in ((bwd, upper, True), (fwd, lower, False)):
        cols = columns(deps)
        for rows, reach in reversed(parts):
            inside = set(rows)
            outside(rows, cols, lambda i: i not in inside)
            of = {j: [] for j in rows}
            for i in rows:
                for j in reach[i]:
                    of[j].append(at[(i, j)] | x[i] << 16)
            product({j: [(rbase + j if scaled else minus) | x[j] << 16] + of[j]
                     for j in rows if scaled or of[j]})
        if tail and scaled:
            outside(range(t0, n), cols, lambda i: i < t0)
            product({j: [block + (i - t0) * tail + j - t0 | x[i] << 16 for i in range(t0, n)]
                     for j in range(t0, n)})
    return seg, x


EARLY = 2              # levels between an early product's readiness and its sum's end


def coop_inc(mech: dict) -> str:
    """coop.inc: MECH_COOP and, when the programs exist, their C arrays for
    both builds (COOP_SPLIT) and both block sizes, included by one translation
    unit."""
    forms = {}
    try:
        for split in (False, True):
            for nw in (4, 8):
                forms[split, nw] = _fitting_programs(mech, split, nw)
            for k in ("unit", "tail", "block", "buffer", "chains", "coef", "parts"):
                assert forms[split, 4][k] == forms[split, 8][k], k
    except Unsupported as e:
        return f"/* no cooperative kernel for this mechanism: {e} */\n#define MECH_COOP 0\n"

    def arr(ctype, name, vals, space="__device__ const"):
        body = ",".join(str(v) for v in vals) if vals else "0"
        return f"static {space} {ctype} {name}[{max(len(vals), 1)}] = {{{body}}};"

    def doubles(name, vals):
        return arr("double", name, [repr(float(v)) for v in vals] or [0.0])

    lines = ["/* generated cooperative-kernel tables; do not edit */", "#pragma once",
             "#define MECH_COOP 1", f"#define COOP_NUPD {len(compile_tables(mech)['upd'])}",
             f"#define COOP_DEPTH {DEPTH}"]
    for split in (False, True):
        lines.append("#if COOP_SPLIT" if split else "#if !COOP_SPLIT")
        for nw in (4, 8):
            p = forms[split, nw]
            rounds = max([1] + [-(-len(c) // 32) for c in p["chains"]])
            if nw == 4:
                lines += [f"#define COOP_NX {p['nx']}",
                          f"#define COOP_NEXTRA {len(p['extra'])}", f"#define COOP_PARTS {p['parts']}",
                          doubles("coop_ext", p["ext"]),
                          arr("int", "coop_extra_src", [j for j, _ in p["extra"]]),
                          doubles("coop_extra_val", [v for _, v in p["extra"]]),
                          f"#define COOP_NCOEF {len(p['coef']) + len(p['coef']) % 2}",
                          doubles("coop_coef", list(p["coef"]) + [0.0] * (len(p["coef"]) % 2)),
                          f"#define COOP_NAPART {p['napart']}", f"#define COOP_NSCOEF {len(p['scoef'])}",
                          doubles("coop_scoef", p["scoef"]), arr("unsigned char", "coop_has_k", p["has_k"]),
                          f"#define COOP_BUFFER {p['buffer']}", f"#define COOP_NBUFD {p['nbufd']}",
                          f"#define COOP_UNIT {p['unit']}", f"#define COOP_CHAINS {rounds}",
                          arr("int", "coop_chain_of", [x for c in p["chains"] for k in range(32 * rounds)
                                                    for x in (c[k] if k < len(c) else (-1, 0, 0))]),
                          f"#define COOP_TAIL {p['tail']}", f"#define COOP_BLOCK {p['block']}", "#define COOP_NBP(q) (%s)" % " : ".join(
                              [f"(q) == {k} ? {v}" for k, v in enumerate(p["nbp"])] + ["0"]),
                          arr("int", "coop_diag", [o << 1 | (e and 1) for o, e in p["diag"]])]
                lines += [f"#define COOP_SEG_{name.upper()} {k}" for k, name in enumerate(p["segs"])]
                lines.append(arr("int", f"coop_place_t{nw}", p["place_t"]))
            lines += [f"#define COOP_NG{nw} {p['ng']}",
                      f"#define COOP_CELL{nw} {p['cell']}", arr("int", f"coop_place{nw}", p["place"])]
            words, where = [], []
            for name, seg in p["segs"].items():
                if nw == 8 and name in ADJOINT:      # the adjoint has 4 warps
                    continue
                for ops in seg.ops:
                    where.append("{%d,%d}" % (len(words) // 4, len(ops)))
                    for op in ops:                   # first four words of the lanes, then the others
                        words += [x for lane in op for x in lane[:4]] + [x for lane in op for x in lane[4:]]
            lines.append(f"static __constant__ int2 coop_seg{nw}[{len(where)}] = {{{','.join(where)}}};")
            lines.append(arr("unsigned int", f"coop_words{nw}", [f"{w}u" for w in words],
                             "__device__ const __align__(16)"))
        lines.append("#endif")
    return "\n".join(lines) + "\n"
