"""The integer Box-Muller functions (radius, sine, cosine of 64-bit uniforms)
compiled for the host, against extended precision: table interval edges,
octant edges, uniforms next to 0 and 1 and random ones.

Bounds.  Radius: the logarithm is rounded to FP64 with an error of 0.54 ulp
(its fixed point is good to 2^-55 relative), which the root turns into at most
0.54 ulp, and its own rounding adds 0.5.  Sine and cosine of the FP64 angle:
0.5 of the rounding and 0.04 of the fixed point, and next to an axis the
angle's last bits (three errors of 2^-96 turns, below 2^-91).  0.01 for the comparison's
own arithmetic."""
import ctypes
import pathlib
import subprocess

import numpy as np
import pytest

CSRC = pathlib.Path(__file__).resolve().parent.parent / "vsmc_gb300" / "csrc"
LD = np.longdouble

SRC = """
#include <cstddef>
#include "normal64.cuh"
extern "C" void n64(const uint64_t *u, size_t n, double *r, double *s,
    double *c)
{
    for (size_t i = 0; i < n; ++i) {
        r[i] = vsmc_cuda::n64_radius(u[i]);
        vsmc_cuda::n64_sincos(u[i], s[i], c[i]);
    }
}
"""


def _points(which):
    rng = np.random.default_rng(7)
    big = [int(x) for x in rng.integers(0, 2 ** 64, 20000, dtype=np.uint64)]
    sh = [int(k) for k in rng.integers(0, 64, 20000)]
    big += [x >> 11 << 11 for x in big]
    sh += sh
    if which == "random":
        u = big
    elif which == "small":
        u = [x >> k for x, k in zip(big, sh)]
    elif which == "near one":
        u = [2 ** 64 - max(1, x >> k) for x, k in zip(big, sh)]
    else:
        u = [(1 << 63) + (i << 56) + d for i in range(128) for d in (-1, 0, 1)]
        u += [(o << 61) + d for o in range(9)
              for k in range(60) for d in (-(1 << k), 0, (1 << k))]
        u += [(1 << k) + d for k in range(64) for d in (-1, 0, 1)]
        u += [x >> 11 << 11 for x in u if x > 0]
    return np.array(sorted({x for x in u if 0 < x < 2 ** 64}), np.uint64)


def _fraction(u):
    """u 2^-64, exact where the type has 64 bits of mantissa."""
    hi, lo = u >> np.uint64(32), u & np.uint64(0xFFFFFFFF)
    return (hi.astype(LD) * LD(2) ** 32 + lo.astype(LD)) / LD(2) ** 64


def _ulps(got, want):
    """Errors in ulps of the wanted value's own binade."""
    w = want.astype(np.float64)
    return np.abs(got.astype(LD) - want) / np.spacing(np.abs(w)).astype(LD)


@pytest.mark.parametrize("which", ["random", "small", "near one", "edges"])
def test_within_rounding(tmp_path, which):
    if np.finfo(LD).nmant < 63:
        pytest.skip("no extended precision to compare with")
    (tmp_path / "n64.cpp").write_text(SRC)
    so = tmp_path / "n64.so"
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-shared", "-fPIC",
                           f"-I{CSRC}", "-o", str(so),
                           str(tmp_path / "n64.cpp")])
    u = _points(which)
    r, s, c = (np.zeros(len(u)) for _ in range(3))
    ptr = [a.ctypes.data_as(ctypes.c_void_p) for a in (u, r, s, c)]
    ctypes.CDLL(str(so)).n64(ptr[0], ctypes.c_size_t(len(u)), *ptr[1:])
    # next to 1: the logarithm of the exact complement
    comp = np.uint64(0) - u
    ln = np.where(u >> np.uint64(63) == 1, np.log1p(-_fraction(comp)),
                  np.log(_fraction(u)))
    assert _ulps(r, np.sqrt(-2 * ln)).max() <= 1.05
    # the FP64 angle of a 53-bit uniform
    k = (u & np.uint64(2047)) == 0
    th = ((2 * np.pi) * _fraction(u[k]).astype(np.float64)).astype(LD)
    for got, want in ((s[k], np.sin(th)), (c[k], np.cos(th))):
        ulp = np.spacing(np.abs(want.astype(np.float64))).astype(LD)
        err = np.abs(got.astype(LD) - want)
        assert np.all(err <= LD(0.55) * ulp + LD(2) ** -91)
