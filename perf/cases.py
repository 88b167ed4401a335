"""The work that a model hands to this framework, as measurable cases.

Every case is one call sequence of the public Python API on the production
(FMA) libraries with the default launch settings:

* ``device``   Solver.integrate_device: the stream-ordered solve of a batch
               whose arrays live on the GPU;
* ``retry``    Solver.integrate_device_retry: the same with the model's retry
               protocol;
* ``host``     Solver.integrate_batch: the legacy entry that a Fortran host
               model binds, on host arrays (copies in and out included);
* ``grid``     GridChemistry.step: the model's whole batch path on device
               grid fields (pre-scan sort, gather, solve with retry, scatter);
* ``adjoint``  chemistry_step forward and backward: final state and the
               gradients with respect to the initial state and ln RCONST.

Cell states follow the distributions documented in the package's workloads
module (a cold 1200 s step from random states, half of the cells at night),
drawn on the GPU.  ``exact`` integrates small batches of cells with a plain
torch float64 Rodas3 (dense LAPACK solves) from the mechanism's reaction
list."""
import functools
import importlib
import json
import math
import os

import numpy as np
import torch

PKG = importlib.import_module("geos-chem-gpu-hybrid_b200")
ADJ = importlib.import_module("geos-chem-gpu-hybrid_b200.adjoint")
GRID = importlib.import_module("geos-chem-gpu-hybrid_b200.gridstep")
W = PKG.workloads
DEV = "cuda:0"
F64, I32 = torch.float64, torch.int32

# log10 ranges of the rate constants by reaction class (1 first order and
# photolysis, 2 second, 3 third order, 4 with a fixed species, 5 zero order)
K_RANGE = {1: (-6.0, -2.0), 2: (-17.0, -10.0), 3: (-34.0, -31.0), 4: (-17.0, -11.0), 5: (-25.0, -20.0)}
# internal steps of a cold step (the synthetic mechanism over a hundredth of its
# normalised time unit), and floating-point operations per internal step (3 Fun,
# Jac, factorisation, 4 solves)
STEPS = {"fullchem": 78, "synth120": 35}
FLOPS = {"fullchem": 142000, "synth120": 322000}
# most cells of a drawn case, by entry
MOST = {"device": 15000, "retry": 15000, "host": 8000, "adjoint": 100}


def listed():
    return [
        # one cell: a box model or a column debugger calling the solver (smallest call)
        {"name": "box 1 cell", "entry": "device", "mech": "fullchem", "n": 1},
        # one vertical column of 72 levels, as a single-column model has it, retry protocol on
        {"name": "column 72 cells", "entry": "retry", "mech": "fullchem", "n": 72},
        # one MPI rank's small share of a cubed-sphere face through the Fortran entry, odd size,
        # with the options a host may set: non-autonomous, negatives clamped in the solve
        {"name": "host 1001 nonauto", "entry": "host", "mech": "fullchem", "n": 1001, "nonauto": True},
        # a regional grid step with cells outside the chemistry domain: sort, gather, solve, scatter
        {"name": "grid 12x10x36 masked", "entry": "grid", "mech": "fullchem", "nx": 12, "ny": 10, "nz": 36, "mask": True},
        # a share of the 4x5 degree grid (one GPU of several): the largest call
        {"name": "4x5 share 26x16x72", "entry": "device", "mech": "fullchem", "nx": 26, "ny": 16, "nz": 72},
        # sensitivities of a few levels over a 60 s chemistry step: forward and backward
        {"name": "adjoint 24 cells", "entry": "adjoint", "mech": "fullchem", "n": 24, "tend": 60.0},
        # the synthetic stiff mechanism (nearly dense factors) with retry
        {"name": "stiff 1500 cells", "entry": "retry", "mech": "synth120", "n": 1500, "tend": 0.01},
    ]


def _log_size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    entry = rng.choice(["device", "device", "retry", "retry", "host", "grid", "adjoint"])
    case = {"entry": entry, "mech": "fullchem"}
    if entry == "grid":
        case.update(nx=rng.randint(2, 16), ny=rng.randint(2, 12), nz=rng.randint(5, 72), mask=rng.random() < 0.5)
        return case
    if entry == "retry" and rng.random() < 0.5:
        case.update(mech="synth120", n=_log_size(rng, 2, 2000), tend=0.01)
        return case
    case["n"] = _log_size(rng, 2, MOST[entry])
    if entry == "adjoint":
        case["tend"] = rng.choice([60.0, 300.0])
    else:
        case["nonauto"] = rng.random() < 0.25
    return case


def _tend(case):
    return case.get("tend", 1200.0)


def _cells(case):
    return case["n"] if "n" in case else case["nx"] * case["ny"] * case["nz"]


@functools.lru_cache(maxsize=None)
def _info(mech):
    return W.mechanism_info(mech)


def _uniform(g, lo, hi, *shape):
    return torch.rand(*shape, generator=g, dtype=F64, device=DEV) * (hi - lo) + lo


@functools.lru_cache(maxsize=None)
def _rate_table(mech):
    """Per reaction: rate constant at 298 K and E/R, fixed for a mechanism."""
    info = _info(mech)
    rng = np.random.default_rng(1234567)
    k0, ea = np.zeros(info.nreact), np.zeros(info.nreact)
    for c, (lo, hi) in K_RANGE.items():
        sel = info.klass == c
        k0[sel] = 10.0 ** rng.uniform(lo, hi, sel.sum())
    sel = info.klass == 2
    ea[sel] = rng.uniform(-500.0, 2000.0, sel.sum())
    return k0, ea


def _states(case, seed):
    """C (n, NSPEC) and RCONST (n, NREACT) of the case's cells."""
    info, n = _info(case["mech"]), _cells(case)
    g = torch.Generator(device=DEV).manual_seed(int(seed) + 17)
    if case["mech"] != "fullchem":
        k0 = 10.0 ** np.random.default_rng(7654321).uniform(-20.0, 4.0, info.nreact)
        R = torch.as_tensor(k0, device=DEV) * 10.0 ** _uniform(g, -2.0, 2.0, n, 1)
        R = R * 10.0 ** _uniform(g, -0.05, 0.05, n, info.nreact)
        return 10.0 ** _uniform(g, -6.0, 0.0, n, info.nvar + info.nfix), R
    if "n" in case:
        T = _uniform(g, 190.0, 310.0, n)
        P = 10.0 ** _uniform(g, 3.0, math.log10(101300.0), n)
        h2o = 10.0 ** _uniform(g, -6.0, math.log10(3e-2), n)
        o3 = 10.0 ** _uniform(g, -8.0, -5.0, n)
        night = _uniform(g, 0.0, 1.0, n) < 0.5
        sun = torch.where(night, 0.0, _uniform(g, 0.0, 1.0, n) * _uniform(g, 0.0, 1.0, n))
    else:
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        lon = ((torch.arange(nx, device=DEV, dtype=F64) + 0.5) / nx * 360.0 - 180.0)[:, None, None].expand(nx, ny, nz).reshape(-1)
        lat = ((torch.arange(ny, device=DEV, dtype=F64) + 0.5) / ny * 180.0 - 90.0)[None, :, None].expand(nx, ny, nz).reshape(-1)
        lev = torch.arange(nz, device=DEV, dtype=F64)[None, None, :].expand(nx, ny, nz).reshape(-1)
        surf = 300.0 - 40.0 * (lat.abs() / 90.0) ** 1.5 + _uniform(g, -3.0, 3.0, nx * ny).repeat_interleave(nz)
        trop = 16.0 - 4.0 * lat.abs() / 90.0
        z = 0.06 + 79.9 * (lev / max(nz - 1, 1)) ** 2.2
        T = torch.where(z < trop, surf - 6.5 * z, surf - 6.5 * trop + (z - trop)).clamp(185.0, 320.0)
        P = 101325.0 * torch.exp(-z / (29.3 * 0.5 * (surf + T) / 1000.0))
        h2o = torch.where(z < trop, 10.0 ** (math.log10(2e-2) - 4.0 * z / trop), 5e-6)
        h2o = (h2o * 10.0 ** _uniform(g, -0.3, 0.3, n)).clamp(1e-6, 3e-2)
        o3 = torch.where(z < trop, 10.0 ** _uniform(g, -8.0, -7.0, n), 10.0 ** _uniform(g, -6.0, -5.0, n))
        sun = (torch.cos(torch.deg2rad(lat)) * torch.cos(torch.deg2rad(lon))).clamp(0.0, 1.0) * _uniform(g, 0.5, 1.0, n)
    M = P / (W.KB * T) * 1e-6
    vmr = 10.0 ** _uniform(g, -15.0, -6.0, n, info.nvar)
    sp = info.species
    vmr[:, sp["O3"]] = o3
    vmr[:, sp["CO"]] = 10.0 ** _uniform(g, math.log10(5e-8), math.log10(3e-7), n)
    vmr[:, sp["CH4"]] = 1.8e-6
    vmr[:, sp["H2O"]] = h2o
    fix = torch.tensor([f for _, f in info.fixed], dtype=F64, device=DEV)
    C = torch.cat([vmr, fix.expand(n, -1)], 1) * M[:, None]
    k0, ea = _rate_table(case["mech"])
    klass = torch.as_tensor(info.klass, device=DEV)
    R = 10.0 ** _uniform(g, -0.1, 0.1, n, info.nreact)
    R *= torch.exp(torch.as_tensor(-ea, device=DEV) * (1.0 / T - 1.0 / 298.0)[:, None])
    R *= torch.where(klass == 1, sun[:, None], 1.0)
    R *= torch.as_tensor(k0, device=DEV)
    return C.contiguous(), R.contiguous()


def _controls(case):
    """One cell's ICNTRL and RCNTRL, and the tolerances of all."""
    ic = np.zeros(20, np.int32)
    ic[[0, 2, 6, 14]] = (0 if case.get("nonauto") else 1, 4, 1, -1)
    ic[15] = 1 if case.get("nonauto") else 0          # clamp negatives inside the solve
    synth = case["mech"] != "fullchem"
    nvar = _info(case["mech"]).nvar
    return ic, np.zeros(20), np.full(nvar, 1e-8 if synth else W.ATOL_DEFAULT), np.full(nvar, 1e-3 if synth else W.RTOL_DEFAULT)


def prepare(case, seed):
    s = PKG.solver(case["mech"], "fma")
    n, entry = _cells(case), case["entry"]
    C, R = _states(case, seed)
    ic, rc, atol, rtol = _controls(case)
    st = {"case": case, "s": s}
    if entry == "host":
        st["batch"] = W.Batch(np.asfortranarray(C.cpu().numpy().T), np.asfortranarray(R.cpu().numpy().T), atol, rtol,
                              np.asfortranarray(np.tile(ic[:, None], (1, n))), np.asfortranarray(np.tile(rc[:, None], (1, n))))
        return st
    if entry == "grid":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        st["conc0"] = C.T.reshape(s.nspec, nx, ny, nz).permute(0, 3, 2, 1).contiguous()
        rgrid = R.T.reshape(s.nreact, nx, ny, nz).permute(0, 3, 2, 1).contiguous()
        inside = None
        if case["mask"]:                              # the top quarter of the levels has no chemistry
            inside = np.ones((nz, ny, nx), np.int32)
            inside[nz - nz // 4:] = 0
        st["grid"] = GRID.GridChemistry(s, st["conc0"].clone(), np.arange(1, s.nspec + 1), rgrid, atol, rtol, in_chem=inside)
        return st
    if entry == "adjoint":
        b = W.Batch(np.empty((0, n)), np.empty((0, n)), atol, rtol, np.tile(ic[:, None], (1, n)), np.tile(rc[:, None], (1, n)),
                    0.0, _tend(case))
        st["ctl"] = ADJ.Controls(b, torch.device(DEV))
        st["C0"] = C.requires_grad_(True)
        st["logk"] = torch.log(R.clamp(min=1e-300)).requires_grad_(True)
        w = torch.zeros(n, s.nspec, dtype=F64, device=DEV)
        w[:, : s.nvar] = torch.as_tensor(ADJ.loss_weights(n, s.nvar, int(seed) % 1000), device=DEV)
        st["w"] = w
        return st
    st.update(C0=C, C=C.clone(), R=R, A=torch.as_tensor(atol, device=DEV), T=torch.as_tensor(rtol, device=DEV),
              IC=torch.as_tensor(np.tile(ic, (n, 1)), device=DEV), RC=torch.zeros(n, 20, dtype=F64, device=DEV),
              order=torch.arange(n, dtype=I32, device=DEV), IST=torch.zeros(n, 8, dtype=I32, device=DEV),
              RST=torch.zeros(n, 3, dtype=F64, device=DEV), IE=torch.zeros(n, dtype=I32, device=DEV),
              nfail=torch.zeros(2, dtype=I32, device=DEV))
    s.reserve(n)
    return st


def run(st):
    s, entry = st["s"], st["case"]["entry"]
    if entry == "host":
        C, ist, rst, ierr, _, _ = s.integrate_batch(st["batch"])
        return [C, ist, rst, ierr]
    if entry == "grid":
        g = st["grid"]
        g.conc.copy_(st["conc0"])                     # the fields as transport left them
        g.kpph.zero_()
        g.prev.zero_()
        g.step()
        return [g.conc, g.kpph, g.prev, g.diag]
    if entry == "adjoint":
        Cf = ADJ.chemistry_step(st["C0"], st["logk"], s, st["ctl"], 256)
        gC, gk = torch.autograd.grad((Cf * st["w"]).sum(), (st["C0"], st["logk"]))
        return [Cf.detach(), gC, gk]
    st["C"].copy_(st["C0"])
    args = [st[k] for k in ("C", "R", "A", "T")]
    rest = [st[k] for k in ("IC", "RC", "order", "IST", "RST", "IE")]
    if entry == "retry":
        s.integrate_device_retry(*args, st["A"], st["T"], *rest, st["nfail"], 0.0, _tend(st["case"]))
    else:
        s.integrate_device(*args, *rest, 0.0, _tend(st["case"]))
    return [st["C"], st["IST"], st["RST"], st["IE"]]


def work(case):
    info, n = _info(case["mech"]), _cells(case)
    if case["entry"] == "grid" and case["mask"]:
        n -= case["nx"] * case["ny"] * (case["nz"] // 4)
    nspec = info.nvar + info.nfix
    b = 8 * (2 * nspec + info.nreact) + 20 * 12 + 8 * 4 + 3 * 8 + 8
    f = STEPS[case["mech"]] * FLOPS[case["mech"]]
    if case["entry"] == "adjoint":
        b, f = b + 8 * (2 * nspec + info.nreact), 3 * f
    return {"bytes": n * b, "flops": n * f}


@functools.lru_cache(maxsize=None)
def _reactions(mech):
    """The mechanism file's reaction list as dense arrays."""
    with open(os.path.join(W.HERE, "mechanism", mech + ".json")) as fh:
        m = json.load(fh)

    def leaves(e):
        return leaves(e[1]) + leaves(e[2]) if e[0] == "*" else [e]

    rate = []
    for e in m["rates"]:
        fs = leaves(e)
        rate.append(([f[1] for f in fs if f[0] == "k"], math.prod(float(f[1].lower().replace("d", "e")) for f in fs if f[0] == "n"),
                     [f[1] for f in fs if f[0] == "v"], [f[1] for f in fs if f[0] == "f"]))
    S = torch.zeros(m["nvar"], m["nreact"], dtype=F64)
    for i, j, v in m["stoich"]:
        S[i, j] += float(v.lower().replace("d", "e"))
    one = m["nvar"] + m["nfix"]                       # index of a constant 1 behind the species
    idx = torch.full((m["nreact"], 5), one, dtype=torch.long)
    for j, (_, _, v, f) in enumerate(rate):
        idx[j, : len(v)] = torch.tensor(v, dtype=torch.long)
        idx[j, 3: 3 + len(f)] = torch.tensor([m["nvar"] + x for x in f], dtype=torch.long)
    lit = torch.tensor([r[1] for r in rate], dtype=F64)
    usek = torch.tensor([bool(r[0]) for r in rate])
    return S.to(DEV), idx.to(DEV), lit.to(DEV), usek.to(DEV)


def exact(case, seed):
    n = _cells(case)
    if case["entry"] not in ("device", "retry") or case["mech"] != "fullchem" or n > 100 or case.get("nonauto"):
        return None
    C, R = _states(case, seed)
    S, idx, lit, usek = _reactions(case["mech"])
    nvar, nreact = S.shape
    k = torch.where(usek, R, 1.0) * lit
    fixed = torch.cat([C[:, nvar:], torch.ones(n, 1, dtype=F64, device=DEV)], 1)

    def factors(y, kk, fx):
        return torch.cat([y, fx], 1)[:, idx]          # (n, NREACT, 5)

    def fun(y, kk, fx):
        return (factors(y, kk, fx).prod(2) * kk) @ S.T

    def jac(y, kk, fx):
        f = factors(y, kk, fx)
        D = torch.zeros(len(y), nreact, nvar + fixed.shape[1], dtype=F64, device=DEV)
        for p in range(3):
            rest = torch.cat([f[:, :, :p], f[:, :, p + 1:]], 2).prod(2) * kk
            D.scatter_add_(2, idx[:, p].expand(len(y), nreact)[:, :, None], rest[:, :, None])
        return S @ D[:, :, :nvar]

    y, tend = C[:, :nvar].clone(), _tend(case)
    t = torch.zeros(n, dtype=F64, device=DEV)
    h = torch.full((n,), 1e-5, dtype=F64, device=DEV)
    rst = torch.zeros(n, 3, dtype=F64, device=DEV)
    rej, rej2 = torch.zeros(n, dtype=torch.bool, device=DEV), torch.zeros(n, dtype=torch.bool, device=DEV)
    eye = torch.eye(nvar, dtype=F64, device=DEV)
    while True:
        a = torch.nonzero((t - tend) + 2.0 ** -52 <= 0.0)[:, 0]
        if not len(a):
            break
        kk, fx, ya = k[a], fixed[a], y[a]
        new = torch.minimum(h[a], (tend - t[a]).abs())
        hh = torch.where(rej[a], h[a], new)           # the step is clipped where it is first tried
        H = hh[:, None]
        f0 = fun(ya, kk, fx)
        lu = torch.linalg.lu_factor(eye / (0.5 * H[:, :, None]) - jac(ya, kk, fx))

        def solve(b):
            return torch.linalg.lu_solve(*lu, b[:, :, None])[:, :, 0]

        k1 = solve(f0)
        k2 = solve(f0 + 4.0 / H * k1)
        k3 = solve(fun(ya + 2.0 * k1, kk, fx) + (k1 - k2) / H)
        k4 = solve(fun(ya + 2.0 * k1 + k3, kk, fx) + (k1 - k2 - 8.0 / 3.0 * k3) / H)
        yn = ya + 2.0 * k1 + k3 + k4
        scal = W.ATOL_DEFAULT + W.RTOL_DEFAULT * torch.maximum(ya.abs(), yn.abs())
        err = ((k4 / scal) ** 2).mean(1).sqrt().clamp(min=1e-10)
        hn = hh * (0.9 / err ** (1.0 / 3.0)).clamp(0.2, 6.0)
        ok = err <= 1.0
        good = torch.where(rej[a], torch.minimum(hn.clamp(max=tend), hh), hn.clamp(max=tend))
        bad = torch.where(rej2[a], hh * 0.1, hn)
        y[a] = torch.where(ok[:, None], yn, ya)
        t[a] = torch.where(ok, t[a] + hh, t[a])
        rst[a] = torch.where(ok[:, None], torch.stack([t[a], hh, good], 1), rst[a])
        h[a] = torch.where(ok, good, bad)
        rej2[a] = ~ok & rej[a]
        rej[a] = ~ok
    return [torch.cat([y, C[:, nvar:]], 1), None, rst, None]
