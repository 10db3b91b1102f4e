"""The library's scratch memory: kept between calls up to a bound, given back
on request."""
import ctypes

import numpy as np
import pytest

from conftest import dev, host

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
