"""The six schemes at the edges of the counting pass's tiles (2048 elements,
16384 in one cluster) against the oracle, with an engine whose block is partly
used, and what the pass assumes of the stratified uniforms."""
import ctypes

import numpy as np
import pytest

from conftest import P, dev, host


@pytest.mark.gpu
@pytest.mark.parametrize("scheme", range(6))
@pytest.mark.parametrize("m,n", [
    (2, 2), (3, 5), (255, 255), (2047, 2047), (2048, 2048), (2049, 2049),
    (4097, 4097), (16384, 16384), (16385, 16385), (16385, 40000),
    (40001, 16384)])
def test_schemes_at_tile_edges(vc, port, scheme, m, n):
    import torch
    rng = np.random.default_rng(10 * m + scheme)
    w = np.exp(rng.normal(0, 2, m))
    w[rng.random(m) < 0.2] = 0.0  # runs of equal CDF values
    w[0] = 1.0
    w /= w.sum()
    key = np.array([21, 5], np.uint32)
    ctr = np.array([7, 0, 0, 0], np.uint32)
    rep_ref = np.zeros(m, np.int32)
    next_ref = np.zeros(4, np.uint32)
    port.vo_resample_words(scheme, m, n, P(key), P(ctr), P(w), P(rep_ref),
                           P(next_ref))
    r = vc.rng(vc.PHILOX4X32, key=[21, 5], ctr=[7, 0, 0, 0])
    rep = torch.zeros(m, dtype=torch.int32, device="cuda")
    vc.call("vsmc_cuda_resample", m, n, ctypes.byref(r), dev(w).data_ptr(),
            rep.data_ptr(), scheme, None)
    nxt = torch.zeros(4, dtype=torch.int32, device="cuda")
    vc.call("vsmc_cuda_rng_rand", ctypes.byref(r), 4, nxt.data_ptr(), None)
    got = host(rep)
    assert got.sum() == n
    # multinomial and residual take a log and an exp: a uniform may differ
    # in its last bit, which at these sizes moves no count
    assert np.array_equal(got, rep_ref)
    assert np.array_equal(host(nxt).view(np.uint32), next_ref)


@pytest.mark.gpu
@pytest.mark.parametrize("used", [1, 2, 3])
@pytest.mark.parametrize("n", [1000, 4096, 30001])
def test_partly_used_engine_block(vc, used, n):
    """Counts and engine advance when the stream starts inside a block equal
    those from uniforms made of the same words."""
    import torch
    rng = np.random.default_rng(n + used)
    w = rng.random(n)
    w /= w.sum()
    a = vc.rng(vc.PHILOX4X32, 77)
    skip = torch.zeros(used, dtype=torch.int32, device="cuda")
    vc.call("vsmc_cuda_rng_rand", ctypes.byref(a), used, skip.data_ptr(),
            None)
    b = vc.Rng.from_buffer_copy(a)
    rep = torch.zeros(n, dtype=torch.int32, device="cuda")
    vc.call("vsmc_cuda_resample_stratified", n, n, ctypes.byref(a),
            dev(w).data_ptr(), rep.data_ptr(), None)
    words = torch.zeros(n, dtype=torch.int32, device="cuda")
    vc.call("vsmc_cuda_rng_rand", ctypes.byref(b), n, words.data_ptr(), None)
    delta = 1.0 / n
    u = host(words).view(np.uint32) * 2.0 ** -32 * delta + np.arange(n) * delta
    F = np.searchsorted(np.maximum.accumulate(u), np.cumsum(w[:-1]),
                        side="right")
    want = np.diff(np.concatenate([[0], F, [n]]))
    assert np.array_equal(host(rep), want)
    used_words = min(n, n - int(want[-1]) + 1)
    total = used + used_words
    assert (int(a.ctr[0]), int(a.index)) == (
        (total - 1) // 4 + 1, (total - 1) % 4 + 1)


@pytest.mark.parametrize("n", [3, 1000, 999983, (1 << 24) + 1, (1 << 31) - 1])
def test_stratified_uniforms_step_back_only_at_small_words(n):
    """u_j of the stratified sequence is below u_{j-1} only where word j is
    below 2^13, and never below u_{j-2}: the extreme words around random and
    last positions."""
    rng = np.random.default_rng(n % 1000)
    j = np.unique(np.concatenate([
        rng.integers(2, max(n, 4), 20000), [2, n - 1]]))
    j = j[(j >= 2) & (j < n)].astype(np.float64)
    delta = 1.0 / n
    top = (2.0 ** 32 - 1) * 2.0 ** -32 * delta

    def u(word, j):
        return word * 2.0 ** -32 * delta + j * delta

    assert (u(2.0 ** 13, j) >= top + (j - 1) * delta).all()
    assert (u(0.0, j) >= top + (j - 2) * delta).all()
