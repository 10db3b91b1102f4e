"""Learned filters whose step runs in blocks of 128 threads (more segments than
two an SM) against the same filters run alone (256 threads): the sums' order is
the same, so every history has the same bits.  A filter of several segments is
cut at multiples of 1024 particles of the whole batch, so of those only the
first is cut as it is alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 129, 1000, 1025, 2500])
def test_many_segments_match_one_filter(vc, n):
    import torch
    T = 12
    torch.manual_seed(3)
    prop = vc.Proposal()
    prop.params.normal_(0, 0.05)
    prop.pack()
    packed = prop.packed.data_ptr()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    per = (n + 1023) // 1024
    nf = (2 * sms) // per + 7  # more than two segments an SM
    rng = np.random.default_rng(n)
    obs = 0.78 + 0.01 * rng.normal(size=T)
    many = vc.FilterBatch([n] * nf, [T] * nf, list(range(nf)), bearings=True,
                          packed=packed)
    got = many.run(np.tile(obs, nf))
    many.close()
    for k in (0, 1, nf // 2, nf - 1) if n <= 1024 else (0,):
        one = vc.FilterBatch([n], [T], [k], bearings=True, packed=packed)
        want = one.run(obs)[0]
        one.close()
        for key in ("mean", "ess", "logz", "resampled"):
            assert np.array_equal(got[k][key], want[key]), (k, key)
