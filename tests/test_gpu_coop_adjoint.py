"""The backward sweep with one thread block per cell against the one with one
thread per cell, on the same checkpoints.

Both apply the same exact adjoint of the recorded steps and differ in the
order of sums and in the solves (inverses of diagonal blocks).  The
finite-difference tests hold each to 1e-5; two roundings of the same sums must
agree a thousand times better.  Batch sizes below, at and above one cell per
SM; a checkpoint overflow gives -101 and NaN in either."""
import importlib

import numpy as np
import pytest

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(600)]


@pytest.mark.parametrize("mech,n,tend", [("fullchem", 1, 1200.0), ("fullchem", 149, 60.0),
                                         ("fullchem", 301, 1.0), ("synth120", 17, 0.01)])
def test_block_per_cell_matches_thread_per_cell(pkg, mech, n, tend):
    import torch
    adj = importlib.import_module("geos-chem-gpu-hybrid_b200.adjoint")
    w = pkg.workloads
    b = w.plain_small(n, seed=8) if mech == "fullchem" else w.synthetic_stiff(n, seed=8)
    s = pkg.solver(mech, "fma")
    s.set_launch(pkg.PERSISTENT)
    dev = torch.device("cuda:0")
    ctl = adj.Controls(b, dev)
    C0 = torch.from_numpy(np.ascontiguousarray(b.C.T)).to(dev)
    R = torch.from_numpy(np.ascontiguousarray(b.RCONST.T)).to(dev)
    ckmax = 400
    ist = torch.zeros((n, 8), dtype=torch.int32, device=dev)
    rst = torch.zeros((n, 3), dtype=torch.float64, device=dev)
    ie = torch.zeros(n, dtype=torch.int32, device=dev)
    ck = torch.zeros(n * ckmax * (s.nvar + 1), dtype=torch.float64, device=dev)
    s.integrate_device_ckpt(C0.clone(), R, ctl.ATOL, ctl.RTOL, ctl.ICNTRL, ctl.RCNTRL,
                            torch.arange(n, dtype=torch.int32, device=dev), ist, rst, ie, ck, ckmax,
                            0.0, tend)
    lam = torch.from_numpy(np.random.default_rng(4).uniform(0.1, 1.0, (n, s.nspec))).to(dev)
    out = {}
    for mode in (pkg.PLAIN_FUSED, pkg.COOP):
        for cap in (ckmax, int(ist[:, 3].max()) - 1):
            s.set_launch(mode, 128)
            g, k = torch.empty_like(C0), torch.empty_like(R)
            err = torch.zeros(n, dtype=torch.int32, device=dev)
            s.adjoint_device(C0, R, ist, ck if cap == ckmax else ck.view(n, ckmax, -1)[:, :cap].contiguous(),
                             cap, lam, g, k, err)
            out[mode, cap == ckmax] = (g, k, err)
    s.set_launch(pkg.PERSISTENT)
    for full in (True, False):
        (g0, k0, e0), (g1, k1, e1) = out[pkg.PLAIN_FUSED, full], out[pkg.COOP, full]
        assert torch.equal(e0, e1) and (bool((e0 == 1).all()) if full else bool((e0 == -101).any()))
        ok = e0 == 1
        assert torch.isnan(g1[~ok][:, :s.nvar]).all() and torch.isnan(k1[~ok]).all()
        for x, y in ((g0, g1), (k0, k1)):
            scale = x[ok].abs().amax(1, keepdim=True)
            assert bool(((x[ok] - y[ok]).abs() <= 1e-8 * scale).all())
