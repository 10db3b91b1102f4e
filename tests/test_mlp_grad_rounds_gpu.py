"""Loss and gradient of the proposal network at batch sizes where the rounds
of 64 samples fall unevenly on the blocks and their two groups of warps: one
whole round, one sample more, one round for every block and one more, rounds
for both groups of a single block, and enough rounds that the loss terms are
added in several parts.

Tolerances: a sample left out or counted twice moves the loss by about 1 / B;
FP32 sums and the activations that round to another BF16 value move it by less
than 1e-5, the gradient by less than 2e-3 of its norm (the bounds of the other
sizes' test)."""
import ctypes

import numpy as np
import pytest

from conftest import P, dev, host

pytestmark = pytest.mark.gpu

NPAR = 64 * 6 + 64 + 64 * 64 + 64 + 8 * 64 + 8


@pytest.mark.parametrize("B", [64, 65, 9729, 19457, 200001])
def test_loss_grad_rounds_match_oracle(vc, port, B):
    import torch
    rng = np.random.default_rng(B)
    p = rng.normal(0, 0.3, NPAR).astype(np.float32)
    prop = vc.Proposal()
    prop.params.copy_(torch.from_numpy(p).cuda())
    prop.pack()
    feat = rng.normal(0, 1, (B, 6)).astype(np.float32)
    nu = rng.normal(0, 1, (B, 4)).astype(np.float32)
    loss = torch.zeros(1, dtype=torch.float64, device="cuda")
    grad = torch.zeros(NPAR, dtype=torch.float32, device="cuda")
    vc.call("vsmc_cuda_mlp_loss_grad", prop.packed.data_ptr(), B,
            dev(feat).data_ptr(), dev(nu).data_ptr(), loss.data_ptr(),
            grad.data_ptr(), None)
    rl = ctypes.c_double()
    rg = np.zeros(NPAR)
    port.vo_mlp_loss_grad(P(p), B, P(feat), P(nu), ctypes.byref(rl), P(rg))
    assert abs(host(loss)[0] - rl.value) <= 1e-5 * abs(rl.value)
    g = host(grad).astype(np.float64)
    assert np.linalg.norm(g - rg) < 2e-3 * np.linalg.norm(rg)
