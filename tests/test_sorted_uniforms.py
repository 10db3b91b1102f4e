"""The sorted uniforms' running maximum, found among the predecessors whose
sums are within 2^-50 (n64_sorted_max): compiled for the host against the
sequential maximum of the same uniforms, and on the GPU for engines whose
uniforms come that near, or whose sum becomes infinite, counts and time."""
import ctypes
import pathlib
import subprocess
import time

import numpy as np
import pytest

from conftest import P, dev, host

CSRC = pathlib.Path(__file__).resolve().parent.parent / "vsmc_gb300" / "csrc"

SRC = """
#include <cstddef>
#include "explog64.cuh"
using namespace vsmc_cuda;
// 1 - exp(-s) with the exponential's last bit up or down, as an exponential
// within an ulp may have it
struct Shaky {
    double operator()(double s) const
    {
        const double e = exp_of_negative(-s);
        const uint64_t h = n64_bits(s) * 0x9E3779B97F4A7C15ull >> 62;
        return 1.0 - (h == 0 ? std::nextafter(e, 2.0)
                             : (h == 1 ? std::nextafter(e, 0.0) : e));
    }
};
template <class F>
static void all(int max, const double *s, size_t n, double *u, const F &f)
{
    for (size_t j = 0; j < n; ++j)
        u[j] = max ? n64_sorted_max(s, j, f) : f(s[j]);
}
extern "C" void f(int shaky, int max, const double *s, size_t n, double *u)
{
    if (shaky)
        all(max, s, n, u, Shaky());
    else
        all(max, s, n, u, SortedUniform());
}
"""


@pytest.fixture(scope="module")
def fn(tmp_path_factory):
    t = tmp_path_factory.mktemp("sorted")
    (t / "f.cpp").write_text(SRC)
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-shared", "-fPIC",
                           f"-I{CSRC}", "-o", str(t / "f.so"),
                           str(t / "f.cpp")])
    lib = ctypes.CDLL(str(t / "f.so"))

    def call(mx, s, shaky=0):
        u = np.zeros(len(s))
        lib.f(shaky, mx, P(s), ctypes.c_size_t(len(s)), P(u))
        return u
    return call


@pytest.mark.parametrize("shaky", [0, 1])
@pytest.mark.parametrize("base", [0.0, 1e-17, 3e-9, 0.1, 0.7, 1.0, 5.0, 30.0,
                                  36.7, 37.5, 38.0, 700.0, 703.99, 1000.0,
                                  1023.9, 1024.0, 3000.0])
def test_local_maximum_is_the_sequential_one(fn, base, shaky):
    """Runs of neighbouring sums, equal or a few units apart, around base."""
    rng = np.random.default_rng(int(base * 16) + 1)
    unit = max(np.spacing(base), 2.0 ** -53)
    back = 0
    for step in (1, 3, 12):
        d = rng.integers(0, step + 1, 4000) * unit
        s = np.ascontiguousarray(np.cumsum(np.concatenate([[base], d])))
        assert (np.diff(s) >= 0).all()
        u = fn(0, s, shaky)
        back += (np.diff(u) < 0).sum()
        assert np.array_equal(fn(1, s, shaky), np.maximum.accumulate(u))
    # (from e < 1/4 on, the subtraction's rounding hides e's last bit)
    if shaky and 0.05 < base < 1.2:
        assert back > 100  # there is something to put right


def test_infinite_sums(fn):
    s = np.array([0.1, 0.1, 2.0, 2.0, np.inf, np.inf, np.inf])
    u = fn(1, s)
    assert (u[4:] == 1.0).all() and (np.diff(u) >= 0).all()


N = 1 << 20
# Philox key {seed, 0}: no two sums within 2^-50; one pair (term 35668); a word
# that is 0 (term 344899), after which every sum is infinite
SEEDS = {"plain": 1, "near": 1667, "zero": 10751}


def _call(vc, seed, w, rep):
    r = vc.rng(vc.PHILOX4X32, key=[seed, 0], ctr=[0, 0, 0, 0])
    vc.call("vsmc_cuda_resample", N, N, ctypes.byref(r), w.data_ptr(),
            rep.data_ptr(), vc.MULTINOMIAL, None)
    return r


@pytest.mark.gpu
@pytest.mark.parametrize("which", ["plain", "near", "zero"])
def test_counts_equal_the_oracle(vc, port, which):
    import torch
    seed = SEEDS[which]
    rng = np.random.default_rng(seed)
    w = rng.random(N)
    w /= w.sum()
    rep_ref = np.zeros(N, np.int32)
    next_ref = np.zeros(4, np.uint32)
    port.vo_resample_words(0, N, N, P(np.array([seed, 0], np.uint32)),
                           P(np.zeros(4, np.uint32)), P(w), P(rep_ref),
                           P(next_ref))
    rep = torch.zeros(N, dtype=torch.int32, device="cuda")
    r = _call(vc, seed, dev(w), rep)
    nxt = torch.zeros(4, dtype=torch.int32, device="cuda")
    vc.call("vsmc_cuda_rng_rand", ctypes.byref(r), 4, nxt.data_ptr(), None)
    assert np.array_equal(host(rep), rep_ref)
    assert np.array_equal(host(nxt).view(np.uint32), next_ref)


@pytest.mark.gpu
def test_near_sums_cost_no_extra_pass(vc):
    """A call with such a pair, or an infinite sum, takes no longer than
    another (a walk over all uniforms by one block took 7 times the call)."""
    import torch
    w = dev(np.full(N, 1.0 / N))
    rep = torch.zeros(N, dtype=torch.int32, device="cuda")
    us = {}
    for which in ("plain", "near", "zero"):
        best = np.inf
        for _ in range(8):
            torch.cuda.synchronize()
            t = time.perf_counter()
            _call(vc, SEEDS[which], w, rep)
            best = min(best, time.perf_counter() - t)
        us[which] = 1e6 * best
    assert us["near"] < 2.5 * us["plain"], us
    assert us["zero"] < 2.5 * us["plain"], us
