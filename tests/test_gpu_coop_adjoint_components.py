"""The backward sweep with one thread block per cell against the one with one
thread per cell, component by component.

A row's largest gradient says nothing about the others: most reactions' are
below 1e-8 of it.  Every component is a sum over the steps, and is compared
with the size of that sum's terms: t_j is h |S_j| times the adjoint state, so
d/d ln k_j has terms of lambda_max |S_j| h A_j, and d/dC_i of lambda_max (1 +
sum_j |S_j| h dA_j/dV_i).  The rates are taken at the checkpoints on either side
of a step, lambda_max from the two ends of the sweep.  Against these sizes the
two sweeps, two roundings of the same sums, must agree to 1e-8, a thousand times
better than the finite-difference tests hold each of them to.  A wrong partial,
coefficient or t_j shows in a component of more than 1e-6 of its size; that most
are is asserted too."""
import importlib

import numpy as np
import pytest

from mechanism import codegen
from test_coop_adjoint_programs import rates

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(600)]

TOL = 1e-8


def sizes(m, C, R, ck, nacc, lam_max):
    """Sizes of the terms behind a cell's d/d ln k and d/dC (numpy)."""
    n = m["nvar"]
    absS = np.zeros(m["nreact"])
    for i, j, v in m["stoich"]:
        absS[j] += abs(float(codegen.literal(v)))
    y, h = ck[:nacc, :n], ck[:nacc, n]
    y = np.maximum(y, np.concatenate([y[1:], y[-1:]]))       # either side of the step
    gk, gc = np.zeros(m["nreact"]), np.ones(n)
    for j, (kj, lit, vs, fs) in enumerate(rates(m)):
        c = abs(lit) * (R[kj] if kj is not None else 1.0) * np.prod(C[n:][fs]) * absS[j]
        if kj is not None:
            gk[j] = (h * c * np.prod(y[:, vs], axis=1)).sum()
        for q, i in enumerate(vs):
            gc[i] += (h * c * np.prod(y[:, vs[:q] + vs[q + 1:]], axis=1)).sum()
    return lam_max * gk, lam_max * gc


@pytest.mark.parametrize("mech,n,tend", [("fullchem", 10, 60.0), ("fullchem", 6, 1200.0), ("synth120", 10, 0.01)])
def test_components(pkg, mech, n, tend):
    import torch
    adj = importlib.import_module("geos-chem-gpu-hybrid_b200.adjoint")
    w = pkg.workloads
    b = w.plain_small(n, seed=8) if mech == "fullchem" else w.synthetic_stiff(n, seed=8)
    s = pkg.solver(mech, "fma")
    dev = torch.device("cuda:0")
    ctl = adj.Controls(b, dev)
    C0 = torch.from_numpy(np.ascontiguousarray(b.C.T)).to(dev)
    R = torch.from_numpy(np.ascontiguousarray(b.RCONST.T)).to(dev)
    ckmax = 400
    ist = torch.zeros((n, 8), dtype=torch.int32, device=dev)
    rst = torch.zeros((n, 3), dtype=torch.float64, device=dev)
    ie = torch.zeros(n, dtype=torch.int32, device=dev)
    ck = torch.zeros(n * ckmax * (s.nvar + 1), dtype=torch.float64, device=dev)
    s.set_launch(pkg.PERSISTENT)
    s.integrate_device_ckpt(C0.clone(), R, ctl.ATOL, ctl.RTOL, ctl.ICNTRL, ctl.RCNTRL,
                            torch.arange(n, dtype=torch.int32, device=dev), ist, rst, ie, ck, ckmax,
                            0.0, tend)
    lam = torch.from_numpy(np.random.default_rng(4).uniform(0.1, 1.0, (n, s.nspec))).to(dev)
    out = {}
    for mode in (pkg.PLAIN_FUSED, pkg.COOP):
        s.set_launch(mode, 128)
        g, k = torch.empty_like(C0), torch.empty_like(R)
        err = torch.zeros(n, dtype=torch.int32, device=dev)
        s.adjoint_device(C0, R, ist, ck, ckmax, lam, g, k, err)
        torch.cuda.synchronize()
        assert bool((err == 1).all())
        out[mode] = (g.cpu().numpy(), k.cpu().numpy())
    s.set_launch(pkg.PERSISTENT)
    m = codegen.load(mech)
    ck, nacc = ck.cpu().numpy().reshape(n, ckmax, -1), ist[:, 3].tolist()
    (g0, k0), (g1, k1) = out[pkg.PLAIN_FUSED], out[pkg.COOP]
    shown = possible = 0
    for c in range(n):
        lam_max = max(float(lam[c].max()), np.abs(g0[c]).max())
        gk, gc = sizes(m, b.C[:, c], b.RCONST[:, c], ck[c], nacc[c], lam_max)
        assert (np.abs(k0[c] - k1[c]) <= TOL * gk).all()
        assert (np.abs(g0[c] - g1[c])[:s.nvar] <= TOL * gc).all()
        assert (g1[c, s.nvar:] == 0.0).all()
        possible += int((gk > 0).sum())
        shown += int((np.abs(k0[c]) > 100 * TOL * gk).sum())
    assert shown > possible // 2, (shown, possible)
