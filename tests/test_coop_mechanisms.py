"""The cooperative kernel's generator on mechanisms other than the shipped
ones: where it gives programs, they compute the mechanism's Fun, Jacobian,
factors and solves -- bit for bit without split sums, within rounding with
them -- and no offset of a word spills into its neighbour."""
import numpy as np
import pytest

import coop_walk
from mechanism import codegen, coop, synthetic


def mechanism(nspec, nreact, seed=7):
    return codegen.finalize(synthetic.generate(seed, nspec, nreact))


def agrees(m, split, nw, seed=3):
    """Walk the programs against the plain evaluation; False without programs."""
    rng = np.random.default_rng(seed)
    V = 10.0 ** rng.uniform(0, 6, m["nvar"])
    F = 10.0 ** rng.uniform(15, 19, m["nfix"])
    K = 10.0 ** rng.uniform(-18, 2, m["nreact"])
    rhs = rng.standard_normal(m["nvar"]) * 1e5
    ghinv = 1.0 / (30.0 * 0.5)
    w = coop_walk.Walk(m, split, nw, V, F, K, ghinv, rhs)
    if w.p is None:
        return False
    if split:
        coop_walk.check_split(m, w, V, F, K, ghinv, rhs)
    else:
        for g, r in zip((w.fun, w.G0, w.lu, w.x), coop_walk.reference(m, V, F, K, ghinv, rhs)):
            assert np.array_equal(g + 0.0, r + 0.0)      # but for the sign of zeros
    return True


@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("name", ["synth120", "fullchem"])
def test_shipped_mechanisms(name, split):
    assert agrees(codegen.load(name), split, 4)


@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("nspec,nreact,what", [(30, 3000, "buffer"), (135, 450, "factors")])
def test_offsets_beyond_16_bits(nspec, nreact, what, split):
    """30 species in 3,000 reactions: the long sums' products (production
    build) need more than 8,192 places.  135 species in 450 reactions: 9,138
    factors, 73 KB."""
    m = mechanism(nspec, nreact)
    assert agrees(m, split, 4)
    p = coop.level_programs(m, split, 4)
    wide = p["buffer"] > 8191 if what == "buffer" else p["ng"] > 8191
    assert wide == (split or what == "factors")
    assert p["unit"] == (1 if wide else 8)


def test_cell_within_shared_memory():
    """A cell that shared memory does not hold gets fewer inverses of the sweeps'
    parts; one whose factors alone are too many gets no programs."""
    m = mechanism(80, 200)
    p = coop.level_programs(m, True, 4)
    full = coop.SHARED
    try:
        coop.SHARED = p["cell"] + len(p["coef"]) - 200
        q = coop.level_programs(m, True, 4)
        assert q is not None and q["ng"] < p["ng"]
        assert q["cell"] + len(q["coef"]) <= coop.SHARED
        coop.SHARED = m["nnz"]
        assert coop.level_programs(m, True, 4) is None
        assert "shared memory" in coop.coop_inc(m)
    finally:
        coop.SHARED = full


def with_dest(m, terms):
    """The mechanism with other destruction sums for its first species."""
    return dict(m, dest=[e if e is not None else d for e, d in
                         zip(list(terms) + [None] * (m["nvar"] - len(terms)), m["dest"])])


@pytest.mark.parametrize("split", [False, True])
def test_destruction_sums_of_every_form(split):
    """Negative terms, with and without literals, and products of four factors."""
    m = mechanism(24, 90)
    k, v, num, mul = (lambda j: ["k", j]), (lambda i: ["v", i]), (lambda x: ["n", x]), (lambda a, b: ["*", a, b])
    m = with_dest(m, [
        ["-", ["+", k(0), mul(k(1), v(2))], mul(k(3), v(4))],
        ["+", ["neg", mul(mul(k(5), num("2")), v(1))], k(6)],
        ["-", mul(mul(mul(k(7), v(3)), v(4)), v(5)), mul(num("3"), v(6))],
        ["-", ["neg", v(7)], mul(mul(k(8), num("0.5")), v(9))],
    ])
    assert agrees(m, split, 4)


@pytest.mark.parametrize("split", [False, True])
def test_partial_of_several_columns(split):
    """An entry that reads a partial of another column."""
    m = mechanism(24, 90)
    jvs, icol = list(m["jvs"]), m["lu_icol"]
    first = next(p for p, e in enumerate(jvs) if codegen._refs(e, "b"))
    b = codegen._refs(jvs[first], "b")[0]
    others = [p for p in range(m["nnz"]) if icol[p] != icol[first] and codegen._refs(jvs[p], "b")]
    for p in others[:3]:
        jvs[p] = ["+", jvs[p], ["b", b]]
    jvs[others[3]] = ["-", jvs[others[3]], ["*", ["n", "2"], ["b", b]]]
    assert agrees(dict(m, jvs=jvs), split, 4)


@pytest.mark.parametrize("nreact,tail", [(63, 0), (64, 32)])
def test_fewer_rates_than_two_tail_rows(nreact, tail):
    """The tail block's elimination hands its pivot rows over in the rates'
    scratch array; a mechanism with fewer rates goes without the block."""
    m = mechanism(60, nreact)
    assert agrees(m, True, 4)
    assert coop.level_programs(m, True, 4)["tail"] == tail


def test_more_long_sums_than_lanes():
    """40 species in 1,400 reactions: production sums of more than 60 terms take
    two rounds of a warp's lanes."""
    m = mechanism(40, 1400)
    assert agrees(m, True, 4)
    p = coop.level_programs(m, True, 4)
    assert len(p["chains"][1]) > 32
    assert "#define COOP_CHAINS 2" in coop.coop_inc(m)


@pytest.mark.parametrize("name,split,lu,sweep", [
    ("fullchem", False, 61, 69), ("fullchem", True, 13, 9), ("synth120", False, 140, 143), ("synth120", True, 20, 5)])
def test_barriers_of_a_factorisation_and_a_solve(name, split, lu, sweep):
    """The level counts that the kernel's comments state."""
    p = coop.level_programs(codegen.load(name), split, 4)
    for seg, want in (("lu", lu), ("sweep", sweep)):
        for ops in p["segs"][seg].ops:
            assert sum(op[0][1] >> coop.L_SYNC for op in ops) == want
