"""The engine's Student-t variates where the scalar draws for rejected slots
matter: degrees of freedom of each gamma algorithm with many rejections, chunk
sizes around a warp and a chunk, every position of the engine's buffer.  Each
must agree with the oracle to the FP64 functions' last bits and leave the
engine where the oracle's is (a draw taken from a wrong word moves both)."""
import ctypes

import numpy as np
import pytest

from conftest import P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("df", [0.1, 1.2, 1.9, 2.1, 3.0, 4.0])
@pytest.mark.parametrize("eng", [0, 1])
def test_draws_match_oracle(vc, port, eng, df):
    import torch
    kind = vc.PHILOX4X32 if eng == 0 else vc.THREEFRY4X64
    key = (15, 27) if eng == 0 else (15, 27, 31, 43)
    for n in (2, 33, 64, 1000, 1024, 4097):
        for skip in (0, 1, 2, 3):
            r = vc.rng(kind, key=list(key), ctr=[8, 2, 0, 0])
            if skip:
                buf = torch.zeros(8, dtype=torch.int64, device="cuda")
                vc.call("vsmc_cuda_rng_rand", ctypes.byref(r), skip,
                        buf.data_ptr(), None)
            out = torch.zeros(n, dtype=torch.float64, device="cuda")
            vc.call("vsmc_cuda_rng_student_t", ctypes.byref(r), n,
                    out.data_ptr(), ctypes.c_double(df), None)
            k = np.array(list(key) + [0] * (4 - len(key)), np.uint64)
            c = np.array([8, 2, 0, 0], np.uint64)
            want, co = np.zeros(n), np.zeros(4, np.uint64)
            idx = np.zeros(1, np.uint32)
            port.vo_student_t_batch_f64(eng, P(k), P(c), skip, n, df, P(want),
                                        P(co), P(idx))
            np.testing.assert_allclose(out.cpu().numpy(), want, rtol=1e-12,
                                       atol=1e-300, err_msg=f"{n} {skip}")
            assert [int(x) for x in r.ctr] == [int(x) for x in co]
            assert r.index == int(idx[0])
