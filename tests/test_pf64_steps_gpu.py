"""The FP64 filter stepped by its caller: weights written between steps, and
what a step leaves behind when it returns."""
import math

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


def _log_likelihood(model, obs, x, y):
    """Student-t log-density of both coordinates, in the filter's order."""
    nu, sc = model.nu, model.obs_scale
    c2 = 2 * (math.lgamma(0.5 * (nu + 1)) - math.lgamma(0.5 * nu) -
              0.5 * math.log(nu * math.pi) - math.log(sc))
    q = [((o - v) * (1 / sc)) ** 2 * (1 / nu) for o, v in zip(obs, (x, y))]
    return c2 - 0.5 * (nu + 1) * (np.log1p(q[0]) + np.log1p(q[1]))


@pytest.mark.parametrize("n", [1500, 16384, 1 << 20])
def test_evidence_increments_are_accurate(vc, n):
    """An increment is max l + log(sum W exp(l - max l)), the sum a tree: no
    error that grows with n.  Left over are one rounding of the logarithm (1
    ulp at most, of a number below 4: 4.4e-16 to 8.9e-16) and of each addition
    (half an ulp of a total below 32: 1.8e-15): 3e-15 for the first increment
    and an ulp of the total more for the second, on the mean over the seeds
    (the particles' own rounding errors average out).  Left-to-right sums
    had 2.4e-14 at 2^20."""
    import torch
    obs = np.array([[0.3, -0.2], [0.5, 0.1]])
    d = dev(obs)
    e0, e1, ulp = [], [], []
    for seed in range(8):
        pf = vc.ParticleFilter(n, 64, vc.SYSTEMATIC, 0.0, seed=seed,
                               max_steps=2)
        vc.call("vsmc_cuda_pf_initialize", pf.handle, d[0].data_ptr())
        torch.cuda.synchronize()
        s0, w0 = (v.cpu().numpy() for v in _views(pf, n))
        vc.call("vsmc_cuda_pf_iterate", pf.handle, d[1].data_ptr())
        logz = pf.history(2)["logz"]
        s1 = _views(pf, n)[0].cpu().numpy()
        inc = []
        for w, o, s in ((np.full(n, 1.0), obs[0], s0), (w0, obs[1], s1)):
            ll = _log_likelihood(pf.model, o, s[0], s[1])
            m = ll.max()
            mass = math.fsum(w * np.exp(ll - m))
            if s is s0:
                mass /= n
            inc.append(np.longdouble(m) + np.log(np.longdouble(mass)))
        e0.append(abs(float(np.longdouble(logz[0]) - inc[0])))
        e1.append(abs(float(np.longdouble(logz[1]) - np.longdouble(logz[0]) -
                            inc[1])))
        ulp.append(np.spacing(abs(logz[1])))
        pf.close()
    assert np.mean(e0) < 3e-15, e0
    assert np.mean(e1) < 3e-15 + np.mean(ulp), e1


@pytest.mark.parametrize("n", [16384, 1 << 20])
def test_a_single_step_returns_finished(vc, n):
    """initialize and iterate leave nothing running on the filter's stream,
    also after a resample (1.1: at every step), so its pointers can be read
    from any stream."""
    import ctypes

    import torch
    d = dev(np.array([[0.3, -0.2]] * 6))
    pf = vc.ParticleFilter(n, 64, vc.MULTINOMIAL, 1.1, seed=1, max_steps=6)
    st = ctypes.c_void_p()
    vc.call("vsmc_cuda_pf_stream", pf.handle, ctypes.byref(st))
    stream = torch.cuda.ExternalStream(st.value)
    vc.call("vsmc_cuda_pf_initialize", pf.handle, d[0].data_ptr())
    assert stream.query()
    for t in range(1, 6):
        vc.call("vsmc_cuda_pf_iterate", pf.handle, d[t].data_ptr())
        assert stream.query()
    state, weight = (v.cpu().numpy() for v in _views(pf, n))
    h = pf.history(6)
    assert (h["resampled"] == 1).all()
    assert (weight == weight[0]).all()
    np.testing.assert_allclose(state[0].mean(), h["mean"][5][0], rtol=1e-10)
    pf.close()
