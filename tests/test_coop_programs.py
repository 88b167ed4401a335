"""The cooperative kernel's warp streams, walked on the CPU.

Every segment (rates, destruction and production sums, Jacobian partials and
entries, factorisation, sweeps) is executed operation by operation with
Python floats, as the kernel's warps do: between two block barriers a warp
sees only what was there at the first of them, lanes add their products in
table order, groups are summed by the butterfly, chains broadcast their rows
in turn.  The streams without split sums must give the oracle's results bit
for bit; those with split sums (the production build) agree to the rounding
of differently ordered sums.
"""
import numpy as np
import pytest
from scipy.linalg import solve_triangular

from mechanism import codegen, coop


@pytest.fixture(scope="module", params=("synth120", "fullchem"))
def case(request):
    import oracle
    m = codegen.load(request.param)
    oracle.load(request.param)
    rng = np.random.default_rng(11)
    V = 10.0 ** rng.uniform(0, 6, m["nvar"])
    F = 10.0 ** rng.uniform(15, 19, m["nfix"])
    K = 10.0 ** rng.uniform(-18, 2, m["nreact"])
    return request.param, m, V, F, K


class Array:
    """Elements addressed by byte offset; the one behind the last may not be
    written."""

    def __init__(self, values, last):
        self.v = list(values) + [last]

    def __getitem__(self, off):
        assert off % 8 == 0
        return self.v[off // 8]

    def __setitem__(self, off, x):
        assert off % 8 == 0 and off // 8 < len(self.v) - 1
        self.v[off // 8] = x


def _rates(seg, product, n):
    out = [None] * n
    for v, ops in enumerate(seg.ops):
        for i, op in enumerate(ops):
            for lane in range(32):
                for k in range(4):
                    j = ((i * 4 + k) * seg.nw + v) * 32 + lane
                    lo, hi = op[lane][2 * k:2 * k + 2]
                    x = product(lo & 0xFFFF, lo >> 16, hi & 0xFFFF, hi >> 16)
                    if j < n:
                        out[j] = x
                    else:
                        assert x == 0.0
    return out


def _fold(acc, ctl):
    s = (ctl[0] >> coop.L_FOLD) & 7
    assert all((c >> coop.L_FOLD) & 7 == s and (c >> coop.L_GROUP) & 7 <= s for c in ctl)
    for e in range(s):
        acc = [a + acc[v ^ (1 << e)] if e < ((ctl[v] >> coop.L_GROUP) & 7) else a for v, a in enumerate(acc)]
    return acc


def _sum_steps(seg, kind):
    """(header, control, words) of the 32 lanes, step by step, per warp."""
    for ops in seg.ops:
        yield None
        for op in ops:
            if kind == "line":
                yield [(x[0], x[1], x[2:]) for x in op]
            else:
                for h in (0, 4):
                    yield [(x[h] & 0xFFFF, x[h] >> 16, x[h + 1:h + 4]) for x in op]


def _sums(seg, kind, product, finish):
    acc = None
    for step in _sum_steps(seg, kind):
        if step is None:
            acc = [0.0] * 32
            continue
        ctl = [c for _, c, _ in step]
        assert len({c & (coop.L_FIRST | coop.L_END) for c in ctl}) == 1
        if ctl[0] & coop.L_FIRST:
            acc = [0.0] * 32
        for x, (_, c, words) in enumerate(step):
            for w in words:
                acc[x] = product(acc[x], w)
        if ctl[0] & coop.L_END:
            acc = _fold(acc, ctl)
            for x, (h, c, _) in enumerate(step):
                if c & coop.L_LEAD:
                    finish(h, acc[x])


def _levels(seg, G, X, finish):
    """All warps from barrier to barrier; finished entries become visible at
    the next one.  Every warp must pass the same number of barriers."""
    place, wait = [(0, [0.0] * 32)] * seg.nw, [0] * seg.nw
    while any(i < len(ops) for (i, _), ops in zip(place, seg.ops)):
        done = []
        for v, ops in enumerate(seg.ops):
            if wait[v]:
                wait[v] -= 1
                continue
            i, acc = place[v]
            sync = 0
            while i < len(ops) and not sync:
                op = ops[i]
                i += 1
                ctl = [x[1] for x in op]
                uniform = coop.L_FIRST | coop.L_END | -1 << coop.L_FOLD
                assert len({c & uniform for c in ctl}) == 1
                if ctl[0] & coop.L_FIRST:
                    acc = [X[x[0] & 0xFFFF] if x[1] & coop.L_START else 0.0 for x in op]
                used = (ctl[0] >> coop.L_USED) & 7
                assert all(w == seg.none for x in op for w in x[2 + used:])
                for x in range(32):
                    for w in op[x][2:]:
                        acc[x] = acc[x] - G[w & 0xFFFF] * X[w >> 16]
                if ctl[0] & coop.L_END:
                    acc = _fold(acc, ctl)
                    done += [(x[0], x[1], acc[k]) for k, x in enumerate(op) if x[1] & coop.L_LEAD]
                    assert bool(ctl[0] & coop.L_DIAGS) == any(x[1] & coop.L_DIAG for x in op)
                sync = ctl[0] >> coop.L_SYNC
            wait[v] = max(sync - 1, 0)
            place[v] = (i, acc)
        assert len({h & 0xFFFF for h, _, _ in done}) == len(done)
        for h, c, a in done:
            finish(h & 0xFFFF, h >> 16, c, a)
    assert not any(wait)


def _run(m, V, F, K, split, nw, ghinv, rhs):
    p = coop.level_programs(m, split, nw)
    segs = p["segs"]
    n, nnz, nreact = m["nvar"], m["nnz"], m["nreact"]
    xv = Array(list(V) + list(F) + list(p["ext"]), None)
    rx = Array(list(K) + [(K[j] * v if j >= 0 else v) for j, v in p["extra"]], 0.0)
    coef = Array(list(p["coef"]), None)

    def prod4(a, b, c, d):
        return ((rx[a] * xv[b]) * xv[c]) * xv[d]

    A = Array(_rates(segs["rate"], prod4, nreact), 0.0)
    X = Array([None] * n, 0.0)

    def add(area):
        return lambda a, w: a + coef[w & 0xFFFF] * area[w >> 16]

    def set_x(h, acc):
        assert X[h] is None
        X[h] = acc

    _sums(segs["dest"], "line", lambda a, w: a + rx[w & 0xFFFF] * xv[w >> 16], set_x)

    buf = Array([None] * p["buffer"], None)
    if p["buffer"]:
        for k, x in enumerate(_rates(segs["bufd"], prod4, p["nbufd"])):
            buf[8 * k] = x

    def singles(seg, area, put):
        for op in (op for ops in segs[seg].ops for op in ops):
            for x in op:
                for k in range(0, 8, 2):
                    if x[k] & 0xFFFF != coop.NO_ENTRY:
                        put(x[k] & 0xFFFF, coef[x[k] >> 16] * area[x[k + 1]])

    def put_buf(d, x):
        assert buf[d] is None
        buf[d] = x

    def chain(first, blocks):
        s = 0.0
        for k in range(first, first + blocks * coop.BLOCK):
            s = s + buf[8 * k]
        return s

    for i, first, blocks in p["chains"][0]:
        set_x(8 * i, chain(first, blocks))

    def fin_prod(h, acc):
        X[h] = acc - X[h] * xv[h]

    _sums(segs["prod"], "line", add(A), fin_prod)
    if p["buffer"]:
        singles("bufp", A, put_buf)
        assert None not in buf.v[:-1]
    for i, first, blocks in p["chains"][1]:
        fin_prod(8 * i, chain(first, blocks))
    fun = np.array(X.v[:n])
    ng = p["ng"]
    recip = ng - 1 - n
    G = Array([None] * ng, 0.0)
    G[8 * ng - 8] = -1.0

    def set_g(h, acc):
        assert G[h] is None
        G[h] = acc

    for q in range(p["parts"]):
        B = Array(_rates(segs[f"bpart{q}"], prod4, p["nbp"][q]) + [None] * (nreact - p["nbp"][q]), 0.0)
        _sums(segs[f"jvs{q}"], "sum", add(B), set_g)
        singles(f"one{q}", B, set_g)
    for i, (o, final) in enumerate(p["diag"]):
        G[8 * o] = G[8 * o] + ghinv
        if final and split:
            G[8 * (recip + i)] = -1.0 / G[8 * o] if G[8 * o] else float("-inf")
    tail, t0 = p["tail"], n - p["tail"]
    block = [[8 * (p["block"] + i * tail + c) for c in range(tail)] for i in range(tail)]
    G0 = np.array([G[8 * k] for k in p["factor"]])

    def set_lu(d, e, c, acc):
        if c & coop.L_DIAG:
            if split:
                G[e] = -1.0 / acc if acc else float("-inf")
        elif split:
            acc = -(acc * G[e])
        elif c & coop.L_SCALED:
            acc = acc / G[e]
        G[d] = acc

    _levels(segs["lu"], G, G, set_lu)
    schur = np.array([[G[k] for k in row] for row in block]).reshape(tail, tail)
    inv = schur.copy()
    for k in range(tail):                     # Gauss-Jordan in place, no pivoting
        row = inv[k] / inv[k, k]
        row[k] = 1.0 / inv[k, k]
        f = inv[:, k].copy()
        inv[:, k] = 0.0
        inv -= np.outer(f, row)
        inv[k] = row
    for i in range(tail):
        for c in range(tail):
            G[block[i][c]] = -inv[i, c]
    X = Array(list(rhs) + [0.0] + [None] * (n + 1), None)

    def set_sweep(d, e, c, acc):
        assert d != 8 * n
        X[d] = acc / G[e] if c & coop.L_SCALED else acc

    _levels(segs["sweep"], G, X, set_sweep)
    # the factors, the tail's from its Schur complement
    lu = np.array([G[8 * k] for k in p["factor"]])
    for k in range(tail):
        for i in range(k + 1, tail):
            schur[i, k] /= schur[k, k]
            schur[i, k + 1:] -= schur[i, k] * schur[k, k + 1:]
    for q in range(nnz):
        i, c = m["lu_irow"][q] - t0, m["lu_icol"][q] - t0
        if tail and min(i, c) >= 0:
            lu[q] = schur[i, c]
    return fun, G0, lu, np.array([X[8 * k] for k in p["place"]])


def _oracle(name, m, V, F, K, ghinv, rhs):
    import oracle
    Fp = F if m["nfix"] else K
    fun = oracle.fun(V, Fp, K, mech=name)
    G0 = -oracle.jac(V, Fp, K, mech=name)
    G0[np.array(m["lu_diag"])] += ghinv
    G, ier = oracle.decomp(G0, mech=name)
    assert ier == 0
    return fun, G0, G, oracle.solve(G, rhs, mech=name)


@pytest.mark.parametrize("nw", [4, 8])
def test_unsplit_streams_match_oracle_bits(case, nw):
    name, m, V, F, K = case
    rhs = np.random.default_rng(5).standard_normal(m["nvar"]) * 1e5
    ghinv = 1.0 / (30.0 * 0.5)
    got = _run(m, V, F, K, False, nw, ghinv, rhs)
    ref = _oracle(name, m, V, F, K, ghinv, rhs)
    for g, r, what in zip(got, ref, ("fun", "prep", "lu", "solve")):
        # equal bits but for the sign of zeros (0 + x instead of x)
        assert np.array_equal(g + 0.0, r + 0.0), what


@pytest.mark.parametrize("nw", [4, 8])
def test_split_streams_within_rounding(case, nw):
    """Componentwise rounding-error bounds (Higham, Accuracy and Stability of
    Numerical Algorithms, ch. 3, 8, 9 and 14), gamma_k = k u / (1 - k u):
    a sum of k products is off by at most gamma_k of the sum of magnitudes and
    the factorisation by gamma_n |L||U|.  A part's inverse formed by rows, and
    the product with it, are off by gamma_n |M^-1||M||M^-1| for its block M, so
    the solution by gamma |U^-1||L^-1||L||U||x| with the inverses of the
    magnitudes' comparison matrices for |U^-1| and |L^-1|.  Reciprocal pivots
    add a rounding to a multiplier and a quotient."""
    name, m, V, F, K = case
    n, crow, icol, irow = (m[k] for k in ("nvar", "lu_crow", "lu_icol", "lu_irow"))
    rhs = np.random.default_rng(5).standard_normal(n) * 1e5
    ghinv = 1.0 / (30.0 * 0.5)
    fun, G0, G, x = _run(m, V, F, K, True, nw, ghinv, rhs)
    rfun, rG0, _, _ = _oracle(name, m, V, F, K, ghinv, rhs)
    u = 2.0 ** -53

    def gamma(k):
        return k * u / (1.0 - k * u)

    # sums of magnitudes: every coefficient and rate is taken positive
    def plus(e):
        if e[0] in ("+", "-"):
            return ["+", plus(e[1]), plus(e[2])]
        return e[1] if e[0] == "neg" else e

    absm = dict(m, jvs=[plus(e) for e in m["jvs"]])
    aG0 = _run(absm, V, F, K, False, nw, 0.0, rhs)[1]
    most = 4 + max(len(codegen._chain(e)) for e in m["jvs"])
    assert (np.abs(G0 - rG0) <= 2 * gamma(most + 6) * (np.abs(aG0) + ghinv)).all()
    P = _run(dict(m, dest=[["n", "0"]] * n), V, F, K, False, nw, ghinv, rhs)[0]
    most = 6 + max(len(codegen._chain(e)) for e in m["prod"] + m["dest"])
    assert (np.abs(fun - rfun) <= 2 * gamma(most + 6) * (2 * np.abs(P) + np.abs(rfun))).all()
    A, L, U = np.zeros((n, n)), np.eye(n), np.zeros((n, n))
    A[irow, icol] = G0
    for i in range(n):
        for p in range(crow[i], crow[i + 1]):
            (L if icol[p] < i else U)[i, icol[p]] = G[p]
    bound = np.abs(L) @ np.abs(U)
    # the product L U is itself formed in doubles here
    assert (np.abs(L @ U - A) <= gamma(2 * n + 8) * bound).all()
    ref = solve_triangular(U, solve_triangular(L, rhs, lower=True, unit_diagonal=True))
    cL, cU = 2 * np.eye(n) - np.abs(L), 2 * np.diag(np.abs(np.diag(U))) - np.abs(U)

    def inverse_magnitudes(v):
        return solve_triangular(cU, solve_triangular(cL, v, lower=True))

    reach = inverse_magnitudes(bound @ np.abs(ref) + np.abs(rhs))
    assert (reach >= 0).all()
    assert (np.abs(x - ref) <= gamma(8 * n) * reach).all()


@pytest.mark.parametrize("split", [False, True])
def test_segments_fill_the_fetch_depth(case, split):
    """The kernel fetches a segment's operations in blocks of DEPTH."""
    name, m, *_ = case
    for nw in (4, 8):
        p = coop.level_programs(m, split, nw)
        assert max(p["nbp"]) <= m["nreact"]
        for seg in p["segs"].values():
            assert len(seg.ops) == nw
            for ops in seg.ops:
                assert ops and len(ops) % coop.DEPTH == 0
                assert all(len(op) == 32 and all(len(x) == coop.WORDS for x in op) for op in ops)
