"""One cell of any mechanism through the cooperative kernel's streams, on the
CPU, with Python floats.

``Walk`` executes the forward segments (Fun, the prepared Jacobian, the
factorisation, a solve) as test_coop_programs.py does for the shipped
mechanisms, keeps what the adjoint needs, and then executes the adjoint's
segments (transposed solve, t_j, partials, their derivatives along a stage
vector, the species' sums, the rates' gradient).  Offsets are in the
programs' own unit.  ``reference`` is the plain evaluation of the same
mechanism, in the reference's order, by the tables of test_coop_tables.py."""
import numpy as np
from scipy.linalg import solve_triangular

import test_coop_programs as streams
import test_coop_tables as tables
from mechanism import codegen, coop

U = 2.0 ** -53


def gamma(k):
    return k * U / (1.0 - k * U)


class Array(streams.Array):
    """Elements addressed by offset, `unit` apart."""

    def __init__(self, values, last, unit):
        super().__init__(values, last)
        self.unit = unit

    def __getitem__(self, off):
        assert off % self.unit == 0
        return self.v[off // self.unit]

    def __setitem__(self, off, x):
        assert off % self.unit == 0 and off // self.unit < len(self.v) - 1
        self.v[off // self.unit] = x


class Walk:
    def __init__(self, m, split, nw, V, F, K, ghinv, rhs):
        self.m, self.p = m, coop.level_programs(m, split, nw)
        self.n, self.nreact = m["nvar"], m["nreact"]
        self.V, self.F, self.K, self.split = V, F, K, split
        p = self.p
        if p is None:
            return
        self.unit = p.get("unit", 8)
        self.rx = self.array(list(K) + [(K[j] * v if j >= 0 else v) for j, v in p["extra"]], 0.0)
        self.coef = self.array(list(p["coef"]), None)
        self._fun()
        self._prepare(ghinv)
        self._factor()
        self.x = self._solve("sweep", "place", rhs)

    def array(self, values, last):
        return Array(values, last, self.unit)

    def state(self, V):
        return self.array(list(V) + list(self.F) + list(self.p["ext"]), None)

    def product(self, xv):
        rx = self.rx
        return lambda a, b, c, d: ((rx[a] * xv[b]) * xv[c]) * xv[d]

    def _add(self, area):
        coef = self.coef
        return lambda a, w: a + coef[w & 0xFFFF] * area[w >> 16]

    def _singles(self, seg, area, put):
        for x in (x for ops in self.p["segs"][seg].ops for op in ops for x in op):
            for k in range(0, 8, 2):
                if x[k] & 0xFFFF != coop.NO_ENTRY:
                    put(x[k] & 0xFFFF, self.coef[x[k] >> 16] * area[x[k + 1]])

    def _fun(self):
        p, segs, n, u = self.p, self.p["segs"], self.n, self.unit
        xv, rx = self.state(self.V), self.rx
        A = self.array(streams._rates(segs["rate"], self.product(xv), self.nreact), 0.0)
        X = self.array([None] * n, 0.0)

        def set_x(h, acc):
            assert X[h] is None
            X[h] = acc

        streams._sums(segs["dest"], "line", lambda a, w: a + rx[w & 0xFFFF] * xv[w >> 16], set_x)
        buf = self.array([None] * p["buffer"], None)
        if p["buffer"]:
            for k, x in enumerate(streams._rates(segs["bufd"], self.product(xv), p["nbufd"])):
                buf[u * k] = x

        def put_buf(d, x):
            assert buf[d] is None
            buf[d] = x

        def chain(first, blocks):
            s = 0.0
            for k in range(first, first + blocks * coop.BLOCK):
                s = s + buf[u * k]
            return s

        for i, first, blocks in p["chains"][0]:
            set_x(u * i, chain(first, blocks))

        def fin(h, acc):
            X[h] = acc - X[h] * xv[h]

        streams._sums(segs["prod"], "line", self._add(A), fin)
        if p["buffer"]:
            self._singles("bufp", A, put_buf)
            assert None not in buf.v[:-1]
        for i, first, blocks in p["chains"][1]:
            fin(u * i, chain(first, blocks))
        self.fun = np.array(X.v[:n])

    def _prepare(self, ghinv):
        p, n, u = self.p, self.n, self.unit
        ng = p["ng"]
        self.recip = ng - 1 - n
        G = self.G = self.array([None] * ng, 0.0)
        G[u * (ng - 1)] = -1.0
        xv = self.state(self.V)

        def set_g(h, acc):
            assert G[h] is None
            G[h] = acc

        for q in range(p["parts"]):
            B = self.array(streams._rates(p["segs"][f"bpart{q}"], self.product(xv), p["nbp"][q]) +
                           [None] * (self.nreact - p["nbp"][q]), 0.0)
            streams._sums(p["segs"][f"jvs{q}"], "sum", self._add(B), set_g)
            self._singles(f"one{q}", B, set_g)
        for i, (o, final) in enumerate(p["diag"]):
            G[u * o] = G[u * o] + ghinv
            if final and self.split:
                G[u * (self.recip + i)] = -1.0 / G[u * o]
        self.G0 = np.array([G[u * k] for k in p["factor"]])

    def _factor(self):
        m, p, n, u, G, split = self.m, self.p, self.n, self.unit, self.G, self.split
        tail, t0 = p["tail"], n - p["tail"]
        block = [[u * (p["block"] + i * tail + c) for c in range(tail)] for i in range(tail)]

        def put(d, e, c, acc):
            if c & coop.L_DIAG:
                if split:
                    G[e] = -1.0 / acc
            elif split:
                acc = -(acc * G[e])
            elif c & coop.L_SCALED:
                acc = acc / G[e]
            G[d] = acc

        streams._levels(p["segs"]["lu"], G, G, put)
        schur = np.array([[G[k] for k in row] for row in block]).reshape(tail, tail)
        inv = schur.copy()
        for k in range(tail):                 # Gauss-Jordan in place, no pivoting
            row = inv[k] / inv[k, k]
            row[k] = 1.0 / inv[k, k]
            f = inv[:, k].copy()
            inv[:, k] = 0.0
            inv -= np.outer(f, row)
            inv[k] = row
        for i in range(tail):
            for c in range(tail):
                G[block[i][c]] = -inv[i, c]
        self.lu = np.array([G[u * k] for k in p["factor"]])
        for k in range(tail):
            for i in range(k + 1, tail):
                schur[i, k] /= schur[k, k]
                schur[i, k + 1:] -= schur[i, k] * schur[k, k + 1:]
        for q in range(m["nnz"]):
            i, c = m["lu_irow"][q] - t0, m["lu_icol"][q] - t0
            if tail and min(i, c) >= 0:
                self.lu[q] = schur[i, c]

    def _solve(self, seg, place, rhs):
        n, u, G = self.n, self.unit, self.G
        X = self.array(list(rhs) + [0.0] + [None] * (n + 1), None)

        def put(d, e, c, acc):
            assert d != u * n
            X[d] = acc / G[e] if c & coop.L_SCALED else acc

        streams._levels(self.p["segs"][seg], G, X, put)
        return np.array([X[u * k] for k in self.p[place]])

    def adjoint_stage(self, Vs, k, rhs):
        """One stage of the backward sweep on this cell's factors: u, t, the
        species' sums (J(Vs)^T u and the Hessian term of the stage vector k at
        the state V) and the increments of the rates' gradient."""
        p, n, segs = self.p, self.n, self.p["segs"]
        u = self._solve("sweept", "place_t", rhs)
        UX, sc = self.array(list(u), 0.0), self.array(list(p["scoef"]), None)
        T = self.array([None] * self.nreact, 0.0)

        def put_t(h, acc):
            assert T[h] is None
            T[h] = acc

        streams._sums(segs["tj"], "sum", lambda a, w: a + sc[w & 0xFFFF] * UX[w >> 16], put_t)
        vs, yb, rx = self.state(Vs), self.state(self.V), self.rx
        kx = self.array(list(k) + [0.0] * (p["nx"] - n), None)
        na = p["napart"]
        BM = self.array(streams._rates(segs["apart"], self.product(vs), na), 0.0)

        def dual(a, b, c, d):
            assert d == self.unit * (n + self.m["nfix"]) and yb[d] == 1.0
            return rx[a] * (kx[b] * yb[c] + yb[b] * kx[c])

        DM = self.array(streams._rates(segs["apart"], dual, na), 0.0)
        sums = []
        for area in (BM, DM):
            out = self.array([None] * n, None)

            def put(h, acc, out=out):
                assert out[h] is None
                out[h] = acc

            streams._sums(segs["vthl"], "sum", lambda a, w, area=area: a + T[w & 0xFFFF] * area[w >> 16], put)
            sums.append(np.array(out.v[:n]))

        def mu(a, b, c, d):
            z, y, e = (vs[b], vs[c], vs[d]), (yb[b], yb[c], yb[d]), (kx[b], kx[c], kx[d])
            return ((rx[a] * z[0]) * z[1]) * z[2] + \
                rx[a] * (e[0] * y[1] * y[2] + e[1] * y[0] * y[2] + e[2] * y[0] * y[1])

        g = streams._rates(segs["rate"], mu, self.nreact)
        g = [T[self.unit * j] * x if p["has_k"][j] else 0.0 for j, x in enumerate(g)]
        return u, np.array(T.v[:-1]), sums[0], sums[1], np.array(g)


def reference(m, V, F, K, ghinv, rhs):
    """Fun, the prepared Jacobian, its factors and a solve, bit for bit the
    reference's statements."""
    t = coop.compile_tables(m)
    fun = tables._fun(m, t, list(V), list(F), list(K))
    J = tables._jac(m, t, list(V), list(F), list(K))
    G0 = -J
    G0[np.array(m["lu_diag"])] += ghinv
    G = tables._prep_decomp(m, t, list(J), ghinv)
    return fun, G0, G, tables._solve(m, t, list(G), list(rhs))


def _plus(e):
    """The expression with every coefficient taken positive."""
    if e[0] in ("+", "-"):
        return ["+", _plus(e[1]), _plus(e[2])]
    return e[1] if e[0] == "neg" else e


def dense(m, w):
    """L, U and the prepared matrix of a walk."""
    n = m["nvar"]
    A, L, U_ = np.zeros((n, n)), np.eye(n), np.zeros((n, n))
    A[m["lu_irow"], m["lu_icol"]] = w.G0
    for q, (i, c) in enumerate(zip(m["lu_irow"], m["lu_icol"])):
        (L if c < i else U_)[i, c] = w.lu[q]
    return A, L, U_


def comparison(L, U_):
    """Comparison matrices: their inverses bound |L^-1| and |U^-1|."""
    n = len(L)
    return 2 * np.eye(n) - np.abs(L), 2 * np.diag(np.abs(np.diag(U_))) - np.abs(U_)


def check_split(m, w, V, F, K, ghinv, rhs):
    """The bounds of test_coop_programs.test_split_streams_within_rounding,
    for any mechanism."""
    n = m["nvar"]
    fun, G0, _, _ = reference(m, V, F, K, ghinv, rhs)
    t = coop.compile_tables(dict(m, prod=[_plus(e) for e in m["prod"]], dest=[_plus(e) for e in m["dest"]],
                                 jvs=[_plus(e) for e in m["jvs"]]))
    S = [tables._eval(t, t["sid_rate"] + j, list(V), list(F), list(K), None) for j in range(m["nreact"])]
    P = np.array([tables._eval(t, t["sid_prod"] + i, V, F, K, S) for i in range(n)])
    D = np.array([tables._eval(t, t["sid_dest"] + i, V, F, K, S) for i in range(n)])
    aJ = tables._jac(m, t, list(V), list(F), list(K))
    most = max(len(codegen._chain(e)) for e in m["prod"] + m["dest"] + m["jvs"]) + 12
    assert (np.abs(w.fun - fun) <= 2 * gamma(most) * (P + D * V)).all()
    assert (np.abs(w.G0 - G0) <= 2 * gamma(most) * (aJ + ghinv)).all()
    A, L, U_ = dense(m, w)
    bound = np.abs(L) @ np.abs(U_)
    assert (np.abs(L @ U_ - A) <= gamma(2 * n + 8) * bound).all()
    ref = solve_triangular(U_, solve_triangular(L, rhs, lower=True, unit_diagonal=True))
    cL, cU = comparison(L, U_)
    reach = solve_triangular(cU, solve_triangular(cL, bound @ np.abs(ref) + np.abs(rhs), lower=True))
    assert (np.abs(w.x - ref) <= gamma(8 * n) * reach).all()
