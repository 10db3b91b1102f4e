"""The FP64 filter's copy after a resample (k_select64): particles, weights and
mean for a valid index, and after an error of the passes before it (their index
may be an earlier one) the particles as they were."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT, dev, host

pytestmark = pytest.mark.gpu

NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")


@pytest.fixture(scope="module")
def lib(vc, tmp_path_factory):
    from vsmc_gb300 import build
    libdir = os.path.dirname(build.build())
    out = tmp_path_factory.mktemp("select64") / "libselect64.so"
    r = subprocess.run(
        [NVCC, "-std=c++17", "-O2", "--expt-relaxed-constexpr", "-gencode",
         "arch=compute_103a,code=sm_103a", "-Xcompiler", "-fPIC", "-shared",
         "-I", build.CSRC, "-I", os.path.join(ROOT, "include"),
         os.path.join(ROOT, "tests", "cpp", "select64.cu"), "-o", str(out),
         "-L", libdir, "-lvsmc_cuda", f"-Xlinker=-rpath={libdir}"],
        capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    L = ctypes.CDLL(str(out))
    L.select64.argtypes = [ctypes.c_uint32] * 2 + [ctypes.c_void_p] * 8
    return L


@pytest.mark.parametrize("err", [0, 2])
@pytest.mark.parametrize("n", [1, 127, 129, 40001])
def test_copy_only_without_an_error(lib, n, err):
    rng = np.random.default_rng(n)
    ld = (n + 255) // 256 * 256
    s0 = rng.normal(0, 1, (4, ld))
    # parents keep their slots, the others copy one of them
    parent = rng.random(n) < 0.4
    parent[0] = True
    idx = np.where(parent, np.arange(n), rng.choice(np.flatnonzero(parent), n))
    words = np.zeros(8, np.uint32)
    words[0] = err
    words[4] = 17  # the uniforms left, handed on to the host
    state, W = dev(s0), dev(np.zeros(n))
    scal = dev(np.array([0, 0, 1.0 / n, 0, 0, 0, 0, 0]))
    e, part = dev(words.view(np.int32)), dev(np.zeros(2 * 4096))
    assert 2 * lib.select64_blocks(n) <= len(part)
    out, h = dev(np.zeros(2)), dev(np.zeros(3, np.int32))
    assert lib.select64(n, ld, state.data_ptr(), W.data_ptr(),
                        dev(idx.astype(np.int32)).data_ptr(), scal.data_ptr(),
                        e.data_ptr(), part.data_ptr(), out.data_ptr(),
                        h.data_ptr()) == 0
    want = s0.copy()
    if err == 0:
        want[:, :n] = s0[:, idx]
    assert np.array_equal(host(state), want)
    assert (host(W) == 1.0 / n).all()
    np.testing.assert_allclose(host(out), want[:2, :n].mean(axis=1),
                               rtol=1e-12, atol=1e-14)
    assert host(h).tolist() == [err, 0, 17]
    assert host(e)[5] == 0  # the ticket, for the next launch
