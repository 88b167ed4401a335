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
    """Elements addressed by byte offset; the one behind the last is a constant."""

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
            if kind == "dest":
                yield [(x[0], x[1], [(x[2 + 2 * t], x[3 + 2 * t]) for t in range(3)]) for x in op]
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
        for x, (_, c, words) in enumerate(step):
            a = 0.0 if c & coop.L_FIRST else acc[x]
            for w in words:
                a = product(a, w)
            acc[x] = a
        if ctl[0] & coop.L_END:
            acc = _fold(acc, ctl)
            for x, (h, c, _) in enumerate(step):
                if c & coop.L_LEAD:
                    finish(h, acc[x])


def _levels(seg, start, product, scale, finish):
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
                uniform = coop.L_FIRST | coop.L_END | coop.L_CHAIN | -1 << coop.L_FOLD
                assert len({c & uniform for c in ctl}) == 1
                if ctl[0] & coop.L_FIRST:
                    acc = [start(x[0] & 0xFFFF) if x[1] & coop.L_LEAD else 0.0 for x in op]
                used = (ctl[0] >> coop.L_USED) & 7
                if ctl[0] & coop.L_CHAIN:
                    for t in range(used):
                        j = ((ctl[0] >> coop.L_STEP) & 31) + t
                        xj = scale(op[j][0] >> 16, op[j][1], acc[j])
                        for x in range(32):
                            if op[x][2 + t] != seg.none & 0xFFFF:
                                assert x > j
                                acc[x] = acc[x] - product.factor(op[x][2 + t]) * xj
                else:
                    assert all(w == seg.none for x in op for w in x[2 + used:])
                    for x in range(32):
                        for w in op[x][2:]:
                            acc[x] = product(acc[x], w)
                if ctl[0] & coop.L_END:
                    acc = _fold(acc, ctl)
                    done += [(x[0], x[1], acc[k]) for k, x in enumerate(op) if x[1] & coop.L_LEAD]
                sync = ctl[0] >> coop.L_SYNC
            wait[v] = max(sync - 1, 0)
            place[v] = (i, acc)
        for h, c, a in done:
            finish(h & 0xFFFF, h >> 16, c, scale(h >> 16, c, a))
    assert not any(wait)


class _Term:
    def __init__(self, G, X):
        self.G, self.X = G, X

    def factor(self, p):
        return self.G[p]

    def __call__(self, acc, w):
        return acc - self.G[w & 0xFFFF] * self.X[w >> 16]


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

    _sums(segs["dest"], "dest",
          lambda a, w: a + (rx[w[0] & 0xFFFF] * xv[w[0] >> 16]) * xv[w[1]], set_x)

    def fin_prod(h, acc):
        X[h] = acc - X[h] * xv[h]

    _sums(segs["prod"], "sum", add(A), fin_prod)
    fun = np.array(X.v[:n])
    G, R = Array([None] * nnz, 0.0), Array([None] * n, 1.0)

    def set_g(h, acc):
        assert G[h] is None
        G[h] = acc

    for q in range(p["parts"]):
        B = Array(_rates(segs[f"bpart{q}"], prod4, p["nbp"][q]) + [None] * (nreact - p["nbp"][q]), 0.0)
        _sums(segs[f"jvs{q}"], "sum", add(B), set_g)
    for i, (o, final) in enumerate(p["diag"]):
        G[o] = G[o] + ghinv
        if final:
            R[8 * i] = 1.0 / G[o] if G[o] else float("inf")
    G0 = np.array(G.v[:nnz])

    def scale(r, c, acc):
        if split:
            return acc if c & coop.L_DIAG else acc * R[r]
        return acc / G[p["diag"][r // 8][0]] if c & coop.L_SCALED else acc

    def set_lu(d, r, c, acc):
        G[d] = acc
        if c & coop.L_DIAG:
            R[r] = 1.0 / acc if acc else float("inf")

    _levels(segs["lu"], lambda d: G[d], _Term(G, G), scale, set_lu)
    X = Array(rhs, 0.0)

    def set_sweep(d, r, c, acc):
        X[d] = acc

    _levels(segs["sweep"], lambda d: X[d], _Term(G, X), scale, set_sweep)
    return fun, G0, np.array(G.v[:nnz]), np.array(X.v[:n])


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
    Numerical Algorithms, ch. 3, 8 and 9), gamma_k = k u / (1 - k u):
    a sum of k products is off by at most gamma_k of the sum of magnitudes,
    the factorisation by gamma_n |L||U|, the solves by gamma_3n |L||U||x|.
    Reciprocal pivots add one rounding to a multiplier and to a quotient."""
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
    # the products L U and L U x are themselves formed in doubles here
    assert (np.abs(L @ U - A) <= gamma(2 * n + 8) * bound).all()
    assert (np.abs(L @ (U @ x) - rhs) <= gamma(5 * n + 8) * (bound @ np.abs(x))).all()


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
