"""The sequential sum at the edges of its tiles (2048 elements, 256 per
warp) and on inputs whose sums need breakpoints: binade crossings, ties,
leading zeros, tiny values, an infinite term."""
import numpy as np
import pytest

from conftest import dev, host

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 31, 255, 256, 257, 2047, 2048, 2049, 4096, 6143, 20481, 131073,
         600001]


def _values(kind, n):
    rng = np.random.default_rng(n)
    if kind == "lognormal":
        return np.exp(rng.normal(0, 3, n))
    if kind == "equal":
        return np.full(n, 1.0 / n)
    if kind == "zeros":  # whole tiles of zeros, then values among zeros
        x = np.where(rng.random(n) < 0.3, rng.random(n), 0.0)
        x[: n * 2 // 3] = 0.0
        x[0] = -0.0
        return x
    if kind == "ties":  # odd multiples of half the ulp of sums in [1, 2)
        x = (2.0 * rng.integers(0, 8, n) + 1) * 2.0 ** -53
        x[0] = 1.0
        return x
    if kind == "growing":  # every sum crosses a binade, then small terms
        x = rng.random(n) * 1e-3
        m = min(n, 900)
        x[:m] = 2.0 ** (np.arange(m) - 500.0)
        return x
    x = rng.random(n) * 5e-324 * 2.0 ** 40  # denormal terms and sums
    x[n // 2:] *= 2.0 ** 30
    return x


@pytest.mark.parametrize("kind", ["lognormal", "equal", "zeros", "ties",
                                  "growing", "denormal"])
@pytest.mark.parametrize("n", SIZES)
def test_prefix_and_total_bit_exact(vc, kind, n):
    import torch
    x = _values(kind, n)
    out = torch.zeros(n, dtype=torch.float64, device="cuda")
    tot = torch.zeros(2, dtype=torch.float64, device="cuda")
    d = dev(x)
    vc.call("vsmc_cuda_sequential_sum", n, d.data_ptr(), out.data_ptr(),
            tot.data_ptr(), None)
    vc.call("vsmc_cuda_sequential_sum", n, d.data_ptr(), None,
            tot.data_ptr() + 8, None)
    want = np.cumsum(np.concatenate([[0.0], x]))[1:]
    assert np.array_equal(host(out).view(np.uint64), want.view(np.uint64))
    assert (host(tot) == want[-1]).all()


@pytest.mark.parametrize("at", [0, 5, 2047, 2048, 30000])
def test_infinite_term(vc, at):
    """u01_sorted sums -log(u) / (n - j): a zero uniform's term is infinite
    and every sum from there on is too (the sorted value is 1)."""
    import torch
    n = 40001
    u = np.random.default_rng(at).random(n) * 0.9 + 0.05
    u[at] = 0.0
    out = torch.zeros(n, dtype=torch.float64, device="cuda")
    vc.call("vsmc_cuda_u01_sorted", n, dev(u).data_ptr(), out.data_ptr(),
            None)
    g = host(out)
    assert (g[at:] == 1.0).all()
    want = 1 - np.exp(-np.cumsum(-np.log(u[:at]) / (n - np.arange(at))))
    assert np.abs(g[:at] - want).max(initial=0) < 1e-13
