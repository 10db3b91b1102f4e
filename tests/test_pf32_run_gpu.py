"""A precision-32 run by one cooperative kernel against the same run by
launches: histories, particles and log-weights bit for bit, at the edges of
its tiles (1024 particles per block) and of the sizes it takes, and the steps
after it."""
import ctypes

import numpy as np
import pytest

from conftest import dev

pytestmark = pytest.mark.gpu


def _obs(T, seed=3):
    rng = np.random.default_rng(seed)
    p, v = rng.normal(0, 2, 2), rng.normal(0, 1, 2)
    out = np.empty((T, 2))
    for t in range(T):
        p, v = p + 0.1 * v, v + 0.1 * rng.normal(0, 1, 2)
        out[t] = p + 0.5 * rng.standard_t(10, 2)
    return out


def _cells(vc, pf, n):
    import torch

    class View:
        def __init__(self, ptr, count):
            self.owner = pf
            self.__cuda_array_interface__ = {
                "data": (ptr, False), "shape": (count,), "strides": None,
                "typestr": "<i4", "version": 3}

    s, w = pf.state_ptrs()
    ld = (n + 255) // 256 * 256
    state = torch.as_tensor(View(s, 4 * ld), device="cuda").cpu().numpy()
    lw = torch.as_tensor(View(w, n), device="cuda").cpu().numpy()
    return state.reshape(4, ld)[:, :n], lw


def _run(vc, n, T, scheme, graph, threshold, more=0):
    pf = vc.ParticleFilter(n, 32, scheme, threshold, seed=11,
                           max_steps=T + more)
    pf.use_graph(graph)
    obs = _obs(T + more)
    out = pf.run(obs[:T])
    for t in range(T, T + more):
        vc.call("vsmc_cuda_pf_iterate", pf.handle, dev(obs[t]).data_ptr())
    if more:
        out = pf.history(T + more)
    state, lw = _cells(vc, pf, n)
    pf.close()
    return out, state, lw


def _check(a, b):
    for k in ("mean", "ess", "resampled", "logz"):
        assert np.array_equal(a[0][k], b[0][k]), k
    assert np.array_equal(a[1], b[1])
    # after a resample the stored log-weights are stale, in both the same way
    assert np.array_equal(a[2], b[2])


@pytest.mark.parametrize("scheme", ["stratified", "systematic"])
@pytest.mark.parametrize("n", [2, 31, 1000, 1024, 1025, 2049, 8192, 100003,
                               600000, 622593, 700001])
def test_run_equals_launches(vc, scheme, n):
    s = vc.SCHEMES[scheme]
    a = _run(vc, n, 30, s, True, 0.5)
    b = _run(vc, n, 30, s, False, 0.5)
    assert a[0]["resampled"].sum() > 0 or n < 32
    _check(a, b)


@pytest.mark.parametrize("T,threshold,more", [(1, 0.5, 0), (1, 1.1, 2),
                                              (7, 0.0, 3), (1030, 0.5, 2)])
def test_lengths_and_steps_after(vc, T, threshold, more):
    """One step, no resampling at all, a resample at every step, a run longer
    than one launch, and iterations that follow a run."""
    n = 3000
    a = _run(vc, n, T, vc.SYSTEMATIC, True, threshold, more)
    b = _run(vc, n, T, vc.SYSTEMATIC, False, threshold, more)
    _check(a, b)


def test_invalid_weights_reported(vc):
    """An observation that is not a number leaves no weight: the run reports
    it and the filter can run again."""
    n, T = 5000, 6
    pf = vc.ParticleFilter(n, 32, vc.STRATIFIED, 0.5, seed=2, max_steps=T)
    obs = _obs(T)
    good = pf.run(obs)
    bad = obs.copy()
    bad[3] = np.nan
    with pytest.raises(vc.VsmcCudaError) as e:
        pf.run(bad)
    assert e.value.status == vc.ERR_NONFINITE
    again = pf.run(obs)
    assert np.array_equal(good["ess"], again["ess"])
    pf.close()
