"""The cooperative kernel's level programs, walked on the CPU.

Each program (destruction sums, production sums, Jacobian entries,
factorisation, forward and backward sweep) is executed round by round with
Python floats, as the kernel does: a round reads only what earlier levels
finished, lanes add their products in table order, groups are summed by the
butterfly, chains walk their rows in turn.  The programs without split sums
must give the oracle's results bit for bit; those with split sums (the
production build) agree to the rounding of differently ordered sums.
"""
import numpy as np
import pytest

from mechanism import codegen, coop

NO = coop.NO_WORD


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


def _rounds(prog, start, product, finish, chain=None):
    """start(h) -> an entry's first value, product(acc, word), finish(h, acc)."""
    pending = []
    for off, nl, k, s, flags in prog.rounds:
        if flags & coop.CHAIN:
            for args in pending:
                finish(*args)
            pending = []
            chain(k, prog.words[off:off + 64 + 32 * ((k + 1) // 2)])
            continue
        heads = prog.words[off:off + nl]
        acc = []
        for v, h in enumerate(heads):
            lg = (h >> 13) & 7
            lead = h != NO and v % (1 << lg) == 0
            a = start(h) if lead else 0.0
            for t in range(k):
                w = prog.words[off + nl * (1 + t) + v]
                if w != NO:
                    assert h != NO
                    a = product(a, w)
            acc.append(a)
        for e in range(s):
            acc = [a + acc[v ^ (1 << e)] if e < ((heads[v] >> 13) & 7) else a
                   for v, a in enumerate(acc)]
        for v, h in enumerate(heads):
            if h != NO and v % (1 << ((h >> 13) & 7)) == 0:
                assert (h >> 13) & 7 <= s
                pending.append((h, acc[v]))      # visible after the level only
        if flags & coop.BARRIER:
            for args in pending:
                finish(*args)
            pending = []
    for args in pending:
        finish(*args)


def _programs(m, V, F, K, split, ghinv, rhs):
    p = coop.level_programs(m, split)
    n, nnz = m["nvar"], m["nnz"]
    diag = m["lu_diag"]
    xv = list(V) + list(F) + list(p["ext"])
    rx = list(K) + [(K[j] * v if j >= 0 else v) for j, v in p["extra"]]
    coef = list(p["coef"])

    def prod4(f):
        return ((rx[f[0]] * xv[f[1]]) * xv[f[2]]) * xv[f[3]]

    A = [prod4(f) for f in p["rate"]]
    B = [prod4(f) for f in p["bpart"]]
    out = [None] * n

    def dest_word(acc, w):
        return acc + (rx[w & 0x7FF] * xv[(w >> 11) & 0x3FF]) * xv[w >> 21]

    def set_out(h, acc):
        out[h & 0x1FFF] = acc

    _rounds(p["dest"], lambda h: 0.0, dest_word, set_out)

    def fin_prod(h, acc):
        i = h & 0x1FFF
        out[i] = acc - out[i] * V[i]

    _rounds(p["prod"], lambda h: 0.0, lambda a, w: a + coef[w & 0xFFFF] * A[w >> 16], fin_prod)
    G, R = [None] * nnz, [None] * n

    def recip(i):
        R[i] = 1.0 / G[diag[i]] if G[diag[i]] else float("inf")

    def fin_jvs(h, acc):
        row = ((h >> 16) & 0xFFF) - 1
        G[h & 0x1FFF] = acc + ghinv if row >= 0 else acc
        if h >> 28 & 1:
            recip(row)

    _rounds(p["jvs"], lambda h: 0.0, lambda a, w: a + coef[w & 0xFFFF] * B[w >> 16], fin_jvs)
    G0 = list(G)

    def fin_lu(h, acc):
        c = (h >> 16) & 0xFFF
        if h & 1 << 28:
            acc = acc * R[c] if split else acc / G[diag[c]]
        G[h & 0x1FFF] = acc
        if h & 1 << 29:
            recip(c)

    _rounds(p["lu"], lambda h: G[h & 0x1FFF], lambda a, w: a - G[w & 0xFFFF] * G[w >> 16], fin_lu)
    X = list(rhs)

    def term(a, w):
        return a - G[w & 0xFFFF] * X[w >> 16]

    def fin_fwd(h, acc):
        X[h & 0x1FFF] = acc

    def fin_bwd(h, acc):
        i = h & 0x1FFF
        X[i] = acc if h >> 28 & 1 else (acc * R[i] if split else acc / G[diag[i]])

    def chain_of(scale):
        def chain(k, words):
            rows, mask = words[:k], words[32:32 + k]
            acc = [X[r] for r in rows]
            for j in range(k):
                xj = acc[j] * R[rows[j]] if scale else acc[j]
                for r in range(k):
                    if mask[r] >> j & 1:
                        assert r > j
                        acc[r] -= G[(words[64 + 32 * (j // 2) + r] >> 16 * (j & 1)) & 0xFFFF] * xj
            for r in range(k):
                X[rows[r]] = acc[r] * R[rows[r]] if scale else acc[r]
        return chain

    _rounds(p["fwd"], lambda h: X[h & 0x1FFF], term, fin_fwd, chain_of(False))
    _rounds(p["bwd"], lambda h: X[h & 0x1FFF], term, fin_bwd, chain_of(True))
    return np.array(out), np.array(G0), np.array(G), np.array(X)


def _oracle(name, m, V, F, K, ghinv, rhs):
    import oracle
    Fp = F if m["nfix"] else K
    fun = oracle.fun(V, Fp, K, mech=name)
    G0 = -oracle.jac(V, Fp, K, mech=name)
    G0[np.array(m["lu_diag"])] += ghinv
    G, ier = oracle.decomp(G0, mech=name)
    assert ier == 0
    return fun, G0, G, oracle.solve(G, rhs, mech=name)


def test_unsplit_programs_match_oracle_bits(case):
    name, m, V, F, K = case
    rhs = np.random.default_rng(5).standard_normal(m["nvar"]) * 1e5
    ghinv = 1.0 / (30.0 * 0.5)
    got = _programs(m, V, F, K, False, ghinv, rhs)
    ref = _oracle(name, m, V, F, K, ghinv, rhs)
    for g, r, what in zip(got, ref, ("fun", "prep", "lu", "solve")):
        # equal bits but for the sign of zeros (0 + x instead of x)
        assert np.array_equal(g + 0.0, r + 0.0), what


def test_split_programs_within_rounding(case):
    """Componentwise rounding-error bounds (Higham, Accuracy and Stability of
    Numerical Algorithms, ch. 3, 8 and 9), gamma_k = k u / (1 - k u):
    a sum of k products is off by at most gamma_k of the sum of magnitudes,
    the factorisation by gamma_n |L||U|, the solves by gamma_3n |L||U||x|.
    Reciprocal pivots add one rounding to a multiplier and to a quotient."""
    name, m, V, F, K = case
    n, crow, diag, icol, irow = (m[k] for k in ("nvar", "lu_crow", "lu_diag", "lu_icol", "lu_irow"))
    rhs = np.random.default_rng(5).standard_normal(n) * 1e5
    ghinv = 1.0 / (30.0 * 0.5)
    fun, G0, G, x = _programs(m, V, F, K, True, ghinv, rhs)
    rfun, rG0, _, _ = _oracle(name, m, V, F, K, ghinv, rhs)
    u = 2.0 ** -53

    def gamma(k):
        return k * u / (1.0 - k * u)

    # sums of magnitudes: every coefficient and rate is taken positive
    absm = dict(m)

    def plus(e):
        if e[0] in ("+", "-"):
            return ["+", plus(e[1]), plus(e[2])]
        return e[1] if e[0] == "neg" else e

    absm["jvs"] = [plus(e) for e in m["jvs"]]
    aG0 = _programs(absm, V, F, K, False, 0.0, rhs)[1]
    most = 4 + max(len(codegen._chain(e)) for e in m["jvs"])
    assert (np.abs(G0 - rG0) <= 2 * gamma(most + 6) * (np.abs(aG0) + ghinv)).all()
    absm = dict(m)
    absm["dest"] = [["n", "0"]] * n
    P = _programs(absm, V, F, K, False, ghinv, rhs)[0]
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


def test_every_entry_once_and_in_bounds(case):
    name, m, *_ = case
    n, nnz, crow, diag = m["nvar"], m["nnz"], m["lu_crow"], m["lu_diag"]
    for split in (False, True):
        p = coop.level_programs(m, split)
        assert p["nx"] < 1 << 10 and m["nreact"] + len(p["extra"]) < 1 << 11
        for prog, entries in (("dest", n), ("prod", n), ("jvs", nnz)):
            seen = []
            _rounds(p[prog], lambda h: 0.0, lambda a, w: a, lambda h, a: seen.append(h & 0x1FFF))
            assert sorted(seen) == list(range(entries))
        terms = []
        _rounds(p["lu"], lambda h: 0.0, lambda a, w: terms.append((w & 0xFFFF, w >> 16)) or a,
                lambda h, a: None)
        want = sum(crow[m["lu_icol"][q] + 1] - diag[m["lu_icol"][q]] - 1
                   for i in range(n) for q in range(crow[i], diag[i]))
        assert len(terms) == want and max(max(t) for t in terms) < nnz
        for off, nl, k, s, flags in (r for q in coop.PROGRAMS for r in p[q].rounds):
            assert nl % 32 == 0 and nl <= coop.LANES_PER_ROUND and k < 1 << 10 and s <= 5
