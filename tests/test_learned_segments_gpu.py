"""The learned-proposal step over segments that end inside a tile, inside a
segment and in a later one, against the oracle's FP32 filter.

The output weights are zero (the output biases are not), so the network's
BF16 rounding drops out and only the split of the particles over warps, tiles
and segments is tested; the bearing noise is 0.5 rad and nothing is
resampled.  The FP32 errors of a log-weight (normals 1e-6, bearing 1e-5 rad
over a variance of 0.25) stay below 1e-4, so the effective sample size agrees
to 1e-4 n + 0.01, less than what one particle left out or taken twice would
change, log-evidence to 1e-3 and the mean (spread 1 to 2) to 2e-3."""
import ctypes

import numpy as np
import pytest

from conftest import P

pytestmark = pytest.mark.gpu

NPAR = 64 * 6 + 64 + 64 * 64 + 64 + 8 * 64 + 8
SIZES = [2, 31, 127, 128, 129, 511, 512, 513, 1000, 1023, 1024, 1025, 1153,
         2047, 2500]


def test_ragged_segments_match_oracle(vc, port):
    import torch
    from oracle.binding import bearings_model
    T = 4
    om, m = bearings_model(), vc.bearings_model()
    om.sigma_z = m.sigma_z = 0.5
    tr, obs = np.zeros(4 * T), np.zeros(T)
    port.vo_bearings_simulate(0, T, ctypes.byref(om), P(tr), P(obs))
    rng = np.random.default_rng(4)
    p = rng.normal(0, 0.1, NPAR).astype(np.float32)
    p[4544:4544 + 8 * 64] = 0
    prop = vc.Proposal()
    prop.params.copy_(torch.from_numpy(p).cuda())
    prop.pack()
    seeds = list(range(2, 2 + len(SIZES)))
    b = vc.FilterBatch(SIZES, [T] * len(SIZES), seeds,
                       models=[m] * len(SIZES), threshold=0.0, bearings=True,
                       packed=prop.packed.data_ptr())
    got = b.run(np.tile(obs, len(SIZES)))
    b.close()
    for n, seed, g in zip(SIZES, seeds, got):
        mean, ess, logz = np.zeros(2 * T), np.zeros(T), np.zeros(T)
        res = np.zeros(T, np.int32)
        port.vo_bearings_pf_run(32, n, T, seed, 1, 0.0, ctypes.byref(om),
                                P(obs), P(p), 0, P(mean), P(ess), P(res),
                                P(logz))
        np.testing.assert_allclose(g["ess"], ess, rtol=0,
                                   atol=1e-4 * n + 0.01, err_msg=str(n))
        np.testing.assert_allclose(g["logz"], logz, rtol=0, atol=1e-3)
        np.testing.assert_allclose(g["mean"], mean.reshape(T, 2), rtol=0,
                                   atol=2e-3)
