"""The library's scratch memory: kept between calls up to a bound, given back
on request, and not used past a device reset."""
import ctypes
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT, dev, host

pytestmark = pytest.mark.gpu


def _stratified(vc, n, w, rep):
    r = vc.rng(vc.PHILOX4X32, 3)
    vc.call("vsmc_cuda_resample_stratified", n, n, ctypes.byref(r),
            w.data_ptr(), rep.data_ptr(), None)


def test_trim_gives_the_memory_back(vc):
    """A call at 2^23 takes about 200 MB of scratch; after a trim the device
    has as much free memory as before (within 32 MB), and a call still
    works."""
    import torch
    n = 1 << 23
    w = dev(np.full(n, 1.0 / n))
    rep = torch.zeros(n, dtype=torch.int32, device="cuda")
    small = 1000
    _stratified(vc, small, dev(np.full(small, 1.0 / small)), rep)  # loads code
    torch.cuda.synchronize()
    vc.call("vsmc_cuda_trim_scratch")
    before = torch.cuda.mem_get_info()[0]
    _stratified(vc, n, w, rep)
    first = host(rep).copy()
    torch.cuda.synchronize()
    kept = before - torch.cuda.mem_get_info()[0]
    assert kept <= (1 << 30) + (32 << 20)
    vc.call("vsmc_cuda_trim_scratch")
    assert abs(before - torch.cuda.mem_get_info()[0]) <= 32 << 20, kept
    _stratified(vc, n, w, rep)
    assert np.array_equal(host(rep), first) and first.sum() == n


CHILD = """
import ctypes
import numpy as np
import vsmc_gb300 as vc
rt = ctypes.CDLL("libcudart.so.13")
n = 100000
x = np.random.default_rng(1).random(n)
want = np.cumsum(x)[-1]


def call():
    p = ctypes.c_void_p()
    assert rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(8 * n + 8)) == 0
    assert rt.cudaMemcpy(p, x.ctypes.data_as(ctypes.c_void_p),
                         ctypes.c_size_t(8 * n), 1) == 0
    total = ctypes.c_void_p(p.value + 8 * n)
    vc.call("vsmc_cuda_sequential_sum", n, p, None, total, None)
    got = ctypes.c_double()
    assert rt.cudaMemcpy(ctypes.byref(got), total, ctypes.c_size_t(8), 2) == 0
    assert got.value == want, (got.value, want)


for _ in range(3):
    call()
    vc.call("vsmc_cuda_trim_scratch")
    call()
    assert rt.cudaDeviceReset() == 0
print("done")
"""


def test_calls_after_a_device_reset(vc):
    """A reset ends the pool with everything else of its context; the next call
    makes another (in a process of its own)."""
    r = subprocess.run([sys.executable, "-c", CHILD], capture_output=True,
                       text=True, cwd=ROOT)
    assert r.returncode == 0 and "done" in r.stdout, r.stderr[-2000:]
