"""A user model's infinite log-likelihood is an error at every size: one block
(up to 1024 particles) and many."""
import ctypes
import os
import subprocess

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")


@pytest.fixture(scope="module")
def run(vc, tmp_path_factory):
    from vsmc_gb300 import build
    libdir = os.path.dirname(build.build())
    out = tmp_path_factory.mktemp("infinite_weight") / "lib.so"
    r = subprocess.run(
        [NVCC, "-std=c++17", "-O2", "-gencode",
         "arch=compute_103a,code=sm_103a", "-Xcompiler", "-fPIC", "-shared",
         "-I", os.path.join(ROOT, "include"),
         os.path.join(ROOT, "tests", "cpp", "infinite_weight.cu"), "-o",
         str(out), "-L", libdir, "-lvsmc_cuda", f"-Xlinker=-rpath={libdir}"],
        capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    L = ctypes.CDLL(str(out))
    L.infinite_weight_run.argtypes = [ctypes.c_size_t, ctypes.c_size_t,
                                      ctypes.c_float]
    return L.infinite_weight_run


@pytest.mark.parametrize("T", [1, 3])
@pytest.mark.parametrize("n", [50, 1000, 1024, 1025, 100003])
def test_infinite_log_likelihood_is_reported(vc, run, n, T):
    assert run(n, T, -1.0) == 0  # no particle
    for which in (0, n // 2, n - 1):
        assert run(n, T, float(which)) == vc.ERR_NONFINITE, which
