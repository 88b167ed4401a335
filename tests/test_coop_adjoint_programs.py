"""The streams that only the adjoint uses, walked on the CPU: the transposed
sweeps, t_j = S_j . u, the partials of the rates and their derivatives along a
stage vector, the species' sums and the rates' gradient.

Each is compared, component by component, with what the mechanism's own rates
and stoichiometry give.  A sum of k products of at most m factors is off by at
most gamma_{k+m} of the sum of the magnitudes (Higham, Accuracy and Stability of
Numerical Algorithms, ch. 3); the transposed solve by the bound that
test_coop_programs.test_split_streams_within_rounding gives for the other, with
L and U exchanged and transposed."""
import numpy as np
import pytest
from scipy.linalg import solve_triangular

import coop_walk
from coop_walk import gamma
from mechanism import codegen, synthetic


def rates(m):
    """Per reaction: rate constant or None, literal, variable species, fixed."""
    out = []
    for e in m["rates"]:
        fs = []
        while e[0] == "*":
            fs.append(e[2])
            e = e[1]
        fs.append(e)
        lit = 1.0
        for f in fs:
            if f[0] == "n":
                lit *= float(codegen.literal(f[1]))
        ks = [f[1] for f in fs if f[0] == "k"]
        assert len(ks) <= 1
        out.append((ks[0] if ks else None, lit, [f[1] for f in fs if f[0] == "v"],
                    [f[1] for f in fs if f[0] == "f"]))
    return out


@pytest.mark.parametrize("name", ["synth120", "fullchem", "random"])
def test_adjoint_streams(name):
    m = codegen.finalize(synthetic.generate(7, 60, 200)) if name == "random" else codegen.load(name)
    n, nr = m["nvar"], m["nreact"]
    rng = np.random.default_rng(23)
    V, Vs = (10.0 ** rng.uniform(0, 6, n) for _ in range(2))
    F = 10.0 ** rng.uniform(15, 19, m["nfix"])
    K = 10.0 ** rng.uniform(-18, 2, nr)
    k, rhs = rng.standard_normal(n) * V, rng.standard_normal(n)
    w = coop_walk.Walk(m, True, 4, V, F, K, 1.0 / (30.0 * 0.5), rhs)
    u, t, vt, hl, mu = w.adjoint_stage(Vs, k, rhs)

    _, L, U = coop_walk.dense(m, w)
    ref = solve_triangular(L.T, solve_triangular(U.T, rhs, lower=True), unit_diagonal=True)
    cL, cU = coop_walk.comparison(L, U)
    bound = np.abs(U).T @ np.abs(L).T
    reach = solve_triangular(cL.T, solve_triangular(cU.T, bound @ np.abs(ref) + np.abs(rhs), lower=True))
    assert (np.abs(u - ref) <= gamma(8 * n) * reach).all()

    S = np.zeros((nr, n))
    for i, j, v in m["stoich"]:
        S[j, i] += float(codegen.literal(v))
    most = int((S != 0).sum(1).max()) + 8
    assert (np.abs(t - S @ u) <= 2 * gamma(most) * (np.abs(S) @ np.abs(u))).all()

    want = {x: np.zeros(n) for x in ("vt", "vt+", "hl", "hl+")}
    wmu, amu = np.zeros(nr), np.zeros(nr)
    used = np.zeros(n, int)
    for j, (kj, lit, vs, fs) in enumerate(rates(m)):
        c = lit * (K[kj] if kj is not None else 1.0) * np.prod(F[fs])
        along, most_along = 0.0, 0.0
        for q, i in enumerate(vs):
            rest = vs[:q] + vs[q + 1:]
            d = c * np.prod(Vs[rest])
            want["vt"][i] += t[j] * d
            want["vt+"][i] += abs(t[j]) * abs(d)
            used[i] += 1
            for r, x in enumerate(rest):
                h = c * k[x] * np.prod(V[rest[:r] + rest[r + 1:]])
                want["hl"][i] += t[j] * h
                want["hl+"][i] += abs(t[j] * h)
            along += c * k[i] * np.prod(V[rest])
            most_along += abs(c * k[i] * np.prod(V[rest]))
        if kj is not None:
            wmu[j] = t[j] * (c * np.prod(Vs[vs]) + along)
            amu[j] = abs(t[j]) * (abs(c) * np.prod(Vs[vs]) + most_along)
    most = int(used.max()) + 16
    assert (np.abs(vt - want["vt"]) <= 2 * gamma(most) * want["vt+"]).all()
    assert (np.abs(hl - want["hl"]) <= 2 * gamma(most) * want["hl+"]).all()
    assert (np.abs(mu - wmu) <= 2 * gamma(16) * amu).all()
    assert (amu > 0).sum() > nr // 2
