"""The cooperative kernel's cube root of the error norm (csrc/gc_root.h) under
the contraction of the production build's flags.

Its corrections carry a relative error of a few roundings and are at most a few
ulp of the result near 1 (115 ulp at the ends of the range, from the difference
between 1/3 and the double nearest it), so before the last addition the value
is known to better than 1e-12 ulp: it is the correctly rounded one, gc_pow's,
but where x**(1/3) lies that close to a midpoint of two doubles (1e-6 expected
cases in 200,000 arguments)."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(600)]

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "geos-chem-gpu-hybrid_b200", "csrc")
SOURCE = """
#include "gc_root.h"
__global__ void roots(const double* x, double* y, double* z, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) { y[i] = gc_root3(x[i]); z[i] = gc_pow(x[i], 1.0 / 3.0); }
}
extern "C" int run(const void* x, void* y, void* z, int n) {
  roots<<<(n + 127) / 128, 128>>>((const double*)x, (double*)y, (double*)z, n);
  return (int)cudaDeviceSynchronize();
}
"""


def test_root_is_correctly_rounded(tmp_path):
    import torch
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    src, lib = tmp_path / "root.cu", tmp_path / "root.so"
    src.write_text(SOURCE)
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "--fmad=true", "-shared",
                    "-Xcompiler", "-fPIC", "-I", CSRC, "-o", str(lib), str(src)], check=True)
    rng = np.random.default_rng(17)
    # Err starts at 1e-10; most attempts are near 1
    x = np.concatenate([10.0 ** rng.uniform(-10, 10, 100000), 10.0 ** rng.uniform(-2, 2, 80000),
                        10.0 ** rng.uniform(10, 299, 19996), [1e-10, 1.0, 8.0, 9.99e299]])
    dx = torch.from_numpy(x).cuda()
    y, z = torch.empty_like(dx), torch.empty_like(dx)
    run = ctypes.CDLL(str(lib)).run
    run.argtypes = [ctypes.c_void_p] * 3 + [ctypes.c_int]
    torch.cuda.synchronize()
    assert run(dx.data_ptr(), y.data_ptr(), z.data_ptr(), len(x)) == 0
    assert torch.equal(y, z)
