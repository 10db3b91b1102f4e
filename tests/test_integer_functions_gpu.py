"""The integer radius, sine and cosine, exponential, logarithm and quotient as
the kernels compile them, against extended precision: the points and bounds of
the host tests (test_normal64_cpu.py, test_explog64_cpu.py)."""
import ctypes
import os
import pathlib
import subprocess

import numpy as np
import pytest

import test_explog64_cpu as explog
import test_normal64_cpu as normal
from conftest import dev, host

pytestmark = pytest.mark.gpu

LD = np.longdouble
HERE = pathlib.Path(__file__).resolve().parent
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")


@pytest.fixture(scope="module")
def lib(vc, tmp_path_factory):
    from vsmc_gb300 import build
    if np.finfo(LD).nmant < 63:
        pytest.skip("no extended precision to compare with")
    so = tmp_path_factory.mktemp("integer_functions") / "f.so"
    r = subprocess.run(
        [NVCC, "-std=c++17", "-O3", "--expt-relaxed-constexpr", "-gencode",
         "arch=compute_103a,code=sm_103a", "-Xcompiler", "-fPIC", "-shared",
         "-I", build.CSRC, str(HERE / "cpp" / "integer_functions.cu"), "-o",
         str(so)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    return ctypes.CDLL(str(so))


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("which", ["random", "small", "near one", "edges"])
def test_radius_sine_cosine(lib, which):
    u = normal._points(which)
    r, s, c = (dev(np.zeros(len(u))) for _ in range(3))
    assert lib.polar(_p(dev(u.view(np.int64))), ctypes.c_size_t(len(u)),
                     _p(r), _p(s), _p(c)) == 0
    r, s, c = host(r), host(s), host(c)
    comp = np.uint64(0) - u
    ln = np.where(u >> np.uint64(63) == 1,
                  np.log1p(-normal._fraction(comp)),
                  np.log(normal._fraction(u)))
    assert normal._ulps(r, np.sqrt(-2 * ln)).max() <= 1.05
    k = (u & np.uint64(2047)) == 0
    th = ((2 * np.pi) * normal._fraction(u[k]).astype(np.float64)).astype(LD)
    for got, want in ((s[k], np.sin(th)), (c[k], np.cos(th))):
        ulp = np.spacing(np.abs(want.astype(np.float64))).astype(LD)
        err = np.abs(got.astype(LD) - want)
        assert np.all(err <= LD(0.55) * ulp + LD(2) ** -91)


class _Device:
    """The host tests' function, by the device; in their op numbers.  Arguments
    that are not for the integer form give -1 there: not asked here."""

    def __init__(self, lib):
        self.lib = lib

    def __call__(self, op, x=None, w=None, d=None):
        n = len(x if x is not None else w)
        r = dev(np.zeros(n))
        args = [dev(a.view(np.int32) if a.dtype == np.uint32 else a)
                if a is not None else None for a in (x, w, d)]
        assert self.lib.explog(op, *[_p(a) if a is not None else None
                                     for a in args], ctypes.c_size_t(n),
                               _p(r)) == 0
        return host(r)


def test_exp(lib):
    rng = np.random.default_rng(1)
    edge = np.arange(0, 65000, 7) * np.log(2) / 64
    x = np.concatenate([
        rng.exponential(3, 30000), rng.random(20000) * 704,
        2.0 ** rng.uniform(-1060, 9, 20000), edge, np.nextafter(edge, 0),
        np.nextafter(edge, 1000), [0.0, 5e-324, 1e-300, 704.0]])
    x = np.minimum(x, 704.0)
    got = _Device(lib)(0, x)
    assert explog._ulps(got, np.exp(-x.astype(LD))).max() <= 0.55
    # CUDA's function past the range: zero, one and what is not a number
    far = _Device(lib)(0, np.array([800.0, np.inf, np.nan]))
    assert far[0] == 0 and far[1] == 0 and np.isnan(far[2])


def test_log(lib):
    rng = np.random.default_rng(2)
    iv = (128 + np.arange(129)) / 256
    x = np.concatenate([
        rng.random(30000), 2.0 ** rng.uniform(-1022, 0, 30000), iv,
        np.nextafter(iv, 0), np.nextafter(iv, 1), iv * 2.0 ** -40,
        1 - 2.0 ** -rng.uniform(1, 53, 20000), [2.0 ** -1022]])
    x = x[(x < 1) & (x >= 2.0 ** -1022)]
    got = _Device(lib)(1, x)
    want = -np.log(x.astype(LD))
    near = x > 0.5
    want[near] = -np.log1p(-(1 - x[near].astype(LD)))
    assert explog._ulps(got, want).max() <= 0.55
    far = _Device(lib)(1, np.array([0.0, 1.0, np.inf, np.nan, -0.5]))
    assert far[0] == np.inf and far[1] == 0 and far[2] == -np.inf
    assert np.isnan(far[3:]).all()


def test_log_over(lib):
    explog.test_log_over(_Device(lib))
