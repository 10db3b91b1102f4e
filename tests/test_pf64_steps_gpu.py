"""The FP64 filter stepped by its caller: weights written between steps, and
what a step leaves behind when it returns."""
import numpy as np
import pytest

from conftest import dev

pytestmark = pytest.mark.gpu


class _View:
    def __init__(self, owner, ptr, count):
        self.owner = owner
        self.__cuda_array_interface__ = {
            "data": (ptr, False), "shape": (count,), "strides": None,
            "typestr": "<f8", "version": 3}


def _views(pf, n):
    import torch
    s, w = pf.state_ptrs()
    ld = (n + 255) // 256 * 256
    state = torch.as_tensor(_View(pf, s, 4 * ld), device="cuda")
    weight = torch.as_tensor(_View(pf, w, n), device="cuda")
    return state.reshape(4, ld)[:, :n], weight


@pytest.mark.parametrize("n", [3000, 16384, 20000])
@pytest.mark.parametrize("threshold", [0.0, 1.1])
def test_weights_written_between_steps_count(vc, n, threshold):
    """The evidence of a step from equal weights is the mean of those from
    all weight on the first half and on the second: whatever the step before
    did (1.1: it resampled), the weights in memory are the ones used.  The
    three increments are within 1e-12 (sums of n terms, 3e-15 each way)."""
    import torch
    obs = np.array([[0.3, -0.2], [0.5, 0.1]])
    d = dev(obs)
    inc = []
    for part in (slice(0, n), slice(0, n // 2), slice(n // 2, n)):
        pf = vc.ParticleFilter(n, 64, vc.SYSTEMATIC, threshold, seed=3,
                               max_steps=2)
        vc.call("vsmc_cuda_pf_initialize", pf.handle, d[0].data_ptr())
        torch.cuda.synchronize()
        w = torch.zeros(n, dtype=torch.float64, device="cuda")
        w[part] = 1.0 / len(range(n)[part])
        _views(pf, n)[1].copy_(w)
        torch.cuda.synchronize()
        vc.call("vsmc_cuda_pf_iterate", pf.handle, d[1].data_ptr())
        h = pf.history(2)
        assert h["resampled"][0] == (threshold > 1)
        inc.append(h["logz"][1] - h["logz"][0])
        pf.close()
    assert inc[1] != inc[2]
    want = np.log(0.5 * (np.exp(inc[1]) + np.exp(inc[2])))
    assert abs(inc[0] - want) < 1e-12
