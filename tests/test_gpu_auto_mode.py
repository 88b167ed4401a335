"""The kernel a process gets that has named none: one thread block per cell up
to 16,000 fullchem cells (4,000 in the --fmad=false build, any number where the
factorisation is not generated), one thread per cell above.  On either side of
the line the default must give the bits of the kernel it is said to be."""
import os
import subprocess
import sys

import pytest

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(600)]

_CHILD = """
import importlib, sys, torch
pkg = importlib.import_module("geos-chem-gpu-hybrid_b200")
mech, variant, n, tend, coop = sys.argv[1], sys.argv[2], int(sys.argv[3]), float(sys.argv[4]), sys.argv[5] == "1"
b = pkg.workloads.plain_small(n, seed=12) if mech == "fullchem" else pkg.workloads.synthetic_stiff(n, seed=12)
s = pkg.solver(mech, variant)
dev = torch.device("cuda:0")
ctl = importlib.import_module("geos-chem-gpu-hybrid_b200.adjoint").Controls(b, dev)
up = lambda x: torch.from_numpy(x).to(dev)
def run():
    C, R = up(b.C.T.copy()), up(b.RCONST.T.copy())
    ist = torch.zeros((n, 8), dtype=torch.int32, device=dev)
    rst = torch.zeros((n, 3), dtype=torch.float64, device=dev)
    ie = torch.zeros(n, dtype=torch.int32, device=dev)
    s.integrate_device(C, R, ctl.ATOL, ctl.RTOL, ctl.ICNTRL, ctl.RCNTRL,
                       torch.arange(n, dtype=torch.int32, device=dev), ist, rst, ie, 0.0, tend)
    torch.cuda.synchronize()
    return C, ist, rst, ie
assert (s.workspace_slots(n) == 0) == coop
got = run()
s.set_launch(pkg.COOP if coop else pkg.PERSISTENT, 128)
assert (s.workspace_slots(n) == 0) == coop
assert bool((got[3] == 1).all())
for x, y in zip(got, run()):
    assert torch.equal(x, y)
"""


@pytest.mark.parametrize("mech,variant,n,tend,coop", [
    ("fullchem", "fma", 16000, 1e-3, True), ("fullchem", "fma", 16001, 1e-3, False),
    ("fullchem", "nofma", 4000, 1e-3, True), ("fullchem", "nofma", 4001, 1e-3, False),
    ("synth120", "fma", 16001, 1e-6, True), ("synth120", "nofma", 4001, 1e-6, False)])
def test_default_kernel(mech, variant, n, tend, coop):
    env = {k: v for k, v in os.environ.items() if k != "GCCHEM_B200_MODE"}
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _CHILD, mech, variant, str(n), str(tend), str(int(coop))],
                       cwd=root, env=env, capture_output=True, text=True, timeout=500)
    assert r.returncode == 0, r.stderr[-3000:]
