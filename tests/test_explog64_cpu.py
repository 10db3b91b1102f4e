"""The integer exponential, logarithm and quotient (explog64.cuh) compiled for
the host, against extended precision: edges of the tables' intervals, the ends
of the ranges and random arguments.

Bounds: half an ulp of the rounding and 0.05 of the fixed-point errors (the
logarithm's 2^-55 relative at worst).  The quotient rounds a rounded logarithm:
0.55 ulp of it, at most doubled by the change of binade, and 0.51."""
import ctypes
import pathlib
import subprocess

import numpy as np
import pytest

CSRC = pathlib.Path(__file__).resolve().parent.parent / "vsmc_gb300" / "csrc"
LD = np.longdouble

SRC = """
#include <cstddef>
#include "explog64.cuh"
using namespace vsmc_cuda;
extern "C" void f(int op, const double *x, const uint32_t *w,
    const uint32_t *d, size_t n, double *r)
{
    for (size_t i = 0; i < n; ++i) {
        if (op == 0)
            r[i] = n64_exp_ok(n64_bits(x[i])) ? n64_exp_neg(n64_bits(x[i]))
                                              : -1.0;
        else if (op == 1)
            r[i] = n64_log_ok(n64_bits(x[i]))
                ? n64_neg_log_double(n64_bits(x[i]))
                : -1.0;
        else
            r[i] = n64_neg_log_over(w[i], d[i]);
    }
}
"""


@pytest.fixture(scope="module")
def fn(tmp_path_factory):
    if np.finfo(LD).nmant < 63:
        pytest.skip("no extended precision to compare with")
    t = tmp_path_factory.mktemp("explog64")
    (t / "f.cpp").write_text(SRC)
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-shared", "-fPIC",
                           f"-I{CSRC}", "-o", str(t / "f.so"),
                           str(t / "f.cpp")])
    lib = ctypes.CDLL(str(t / "f.so"))

    def call(op, x=None, w=None, d=None):
        n = len(x if x is not None else w)
        r = np.zeros(n)
        ptr = [None if a is None else a.ctypes.data_as(ctypes.c_void_p)
               for a in (x, w, d)]
        lib.f(op, *ptr, ctypes.c_size_t(n),
              r.ctypes.data_as(ctypes.c_void_p))
        return r
    return call


def _ulps(got, want):
    sp = np.spacing(np.abs(want.astype(np.float64))).astype(LD)
    return np.abs(got.astype(LD) - want) / sp


def test_exp(fn):
    rng = np.random.default_rng(1)
    edge = np.arange(0, 65000, 7) * np.log(2) / 64
    x = np.concatenate([
        rng.exponential(3, 30000), rng.random(20000) * 704,
        2.0 ** rng.uniform(-1060, 9, 20000), edge, np.nextafter(edge, 0),
        np.nextafter(edge, 1000), [0.0, -0.0, 5e-324, 1e-300, 704.0]])
    x = np.minimum(x, 704.0)
    got = fn(0, -x)
    assert np.array_equal(got, fn(0, x))  # the sign is ignored
    assert _ulps(got, np.exp(-x.astype(LD))).max() <= 0.55
    assert (fn(0, np.array([704.1, -1e9, np.inf, np.nan])) == -1).all()


def test_log(fn):
    rng = np.random.default_rng(2)
    iv = (128 + np.arange(129)) / 256
    x = np.concatenate([
        rng.random(30000), 2.0 ** rng.uniform(-1022, 0, 30000), iv,
        np.nextafter(iv, 0), np.nextafter(iv, 1), iv * 2.0 ** -40,
        1 - 2.0 ** -rng.uniform(1, 53, 20000), [2.0 ** -1022]])
    x = x[(x < 1) & (x >= 2.0 ** -1022)]
    got = fn(1, x)
    want = -np.log(x.astype(LD))
    near = x > 0.5
    want[near] = -np.log1p(-(1 - x[near].astype(LD)))
    assert _ulps(got, want).max() <= 0.55
    bad = np.array([0.0, -0.0, 1.0, 2.0, 1e-310, -0.5, np.inf, np.nan])
    assert (fn(1, bad) == -1).all()


def test_log_over(fn):
    rng = np.random.default_rng(3)
    w = np.concatenate([rng.integers(1, 2 ** 32, 40000),
                        2 ** rng.integers(0, 32, 4000),
                        2 ** 32 - 2 ** rng.integers(0, 31, 4000),
                        (128 + np.arange(128)) << 24]).astype(np.uint32)
    d = (2 ** rng.uniform(0, 32, len(w))).astype(np.uint64)
    d[::5] = 2 ** rng.integers(0, 32, len(d[::5]))
    d[1::5] = 2 ** 32 - 1 - rng.integers(0, 4, len(d[1::5]))
    d = np.maximum(d, 1).astype(np.uint32)
    u = w.astype(LD) / LD(2) ** 32
    ln = np.where(u > 0.5, -np.log1p(-(1 - u)), -np.log(u))
    assert _ulps(fn(2, None, w, d), ln / d.astype(LD)).max() <= 1.61
