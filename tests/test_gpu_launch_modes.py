"""The automatic launch mode as a setting, and what naming a kernel promises.

A process that has named a kernel can go back to the choice by the number of
cells; threads and blocks set in that mode are the persistent kernel's.  The
model's paths (grid step, chain, retry) give the oracle's bits in it.  One
named kernel gives a cell the same bits in a call of any size, with one cell
per block and with two."""
import importlib

import numpy as np
import pytest

import test_gpu_chain
import test_gpu_gridstep
import test_gpu_retry

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(600)]


def solve(pkg, s, b, tend=1200.0):
    import torch
    dev = torch.device("cuda:0")
    ctl = importlib.import_module("geos-chem-gpu-hybrid_b200.adjoint").Controls(b, dev)
    C = torch.from_numpy(np.ascontiguousarray(b.C.T)).to(dev)
    R = torch.from_numpy(np.ascontiguousarray(b.RCONST.T)).to(dev)
    ist = torch.zeros((b.n, 8), dtype=torch.int32, device=dev)
    rst = torch.zeros((b.n, 3), dtype=torch.float64, device=dev)
    ie = torch.zeros(b.n, dtype=torch.int32, device=dev)
    s.integrate_device(C, R, ctl.ATOL, ctl.RTOL, ctl.ICNTRL, ctl.RCNTRL,
                       torch.arange(b.n, dtype=torch.int32, device=dev), ist, rst, ie, 0.0, tend)
    torch.cuda.synchronize()
    assert bool((ie == 1).all())
    return C, ist, rst


def equal(a, b):
    import torch
    return all(torch.equal(x, y) for x, y in zip(a, b))


def batch(pkg, mech, n, seed):
    w = pkg.workloads
    return (w.plain_small if mech == "fullchem" else w.synthetic_stiff)(n, seed=seed)


def test_automatic_mode_after_a_named_kernel(pkg):
    s = pkg.solver("fullchem", "fma")
    b = batch(pkg, "fullchem", 40, 5)
    s.set_launch(pkg.COOP, 128)
    coop = solve(pkg, s, b, 60.0)
    s.set_launch(pkg.PERSISTENT)
    assert s.workspace_slots(40) > 0
    for settings in ((pkg.AUTO,), (), (pkg.AUTO, 64, 1), (pkg.AUTO, 256)):
        s.set_launch(*settings)
        assert s.workspace_slots(16000) == 0
        # the small call: 128 threads per cell whatever the setting
        assert equal(coop, solve(pkg, s, b, 60.0))
        # the large one: the persistent grid of the given blocks
        big = s.workspace_slots(10 ** 7)
        s.set_launch(pkg.PERSISTENT, *settings[1:])
        assert big == s.workspace_slots(10 ** 7)
    s.set_launch(threads=192)
    assert s.workspace_slots(16000) == 0 and s.workspace_slots(16001) % 192 == 0
    with pytest.raises(ValueError):
        s.set_launch(-2)
    with pytest.raises(ValueError):
        s.set_launch(pkg.AUTO, 48)
    s.set_launch(pkg.PERSISTENT)


@pytest.fixture
def automatic(pkg, monkeypatch):
    """Every set_launch of a test selects the automatic mode."""
    cls = type(pkg.solver("fullchem", "nofma"))
    named = cls.set_launch

    def auto(self, *args, **kwargs):
        named(self, pkg.AUTO)
        assert self.workspace_slots(4000) == 0

    monkeypatch.setattr(cls, "set_launch", auto)
    yield
    monkeypatch.undo()
    pkg.solver("fullchem", "nofma").set_launch(pkg.PERSISTENT)


@pytest.mark.parametrize("graph", [False, True], ids=["eager", "graph"])
def test_gridstep_automatic(pkg, orc, automatic, graph):
    test_gpu_gridstep.test_gridstep_matches_host_path(pkg, orc, graph)


def test_chain_automatic(pkg, orc, automatic):
    test_gpu_chain.test_chain_eager_graph_oracle(pkg, orc)


@pytest.mark.parametrize("max_steps,rtol,want_both", [(140, 2e-3, 0), (120, 3e-3, 7)])
def test_retry_automatic(pkg, orc, automatic, max_steps, rtol, want_both):
    test_gpu_retry.test_retry_bitexact(pkg, orc, max_steps, rtol, want_both, pkg.PERSISTENT)


@pytest.mark.parametrize("mech,tend", [("fullchem", 60.0), ("synth120", 0.1)])
@pytest.mark.parametrize("kernel,threads", [("COOP", 128), ("COOP", 256), ("PERSISTENT", 128)])
def test_named_kernel_bits_do_not_depend_on_the_call(pkg, mech, tend, kernel, threads):
    """600 cells: two cells per block of the cooperative kernel on any GPU with
    fewer than 300 one-cell blocks of it; 37 of them alone: one cell per block."""
    s = pkg.solver(mech, "fma")
    b = batch(pkg, mech, 600, 9)
    mode = getattr(pkg, kernel)
    s.set_launch(mode, threads)
    whole = solve(pkg, s, b, tend)
    few = solve(pkg, s, pkg.workloads.subset(b, np.arange(37)), tend)
    assert equal([x[:37] for x in whole], few)
    if mode == pkg.COOP:
        s.set_launch(mode, threads, 1)             # one cell per block, one block per SM
        assert equal(whole, solve(pkg, s, b, tend))
    s.set_launch(pkg.PERSISTENT)


@pytest.mark.parametrize("threads", [128, 256])
@pytest.mark.parametrize("mech,tend", [("fullchem", 60.0), ("synth120", 0.1)])
def test_two_cells_per_block_bits_nofma(pkg, mech, tend, threads):
    """The --fmad=false build's kernels agree bit for bit; more cells than
    one-cell blocks fit on the GPU."""
    s = pkg.solver(mech, "nofma")
    b = batch(pkg, mech, 601, 10)
    s.set_launch(pkg.PERSISTENT)
    ref = solve(pkg, s, b, tend)
    s.set_launch(pkg.COOP, threads)
    got = solve(pkg, s, b, tend)
    s.set_launch(pkg.PERSISTENT)
    assert equal(ref, got)
