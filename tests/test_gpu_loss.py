"""The network's loss (k_mse): the exact sum of its float32 terms rounded once, the same bits every
time, added to what the loss held, and the gradient beside it (needs a B200).  Tolerance: float64 sums of n
terms of one sign are within n 2^-53 of exact, so the float32 result is within half a unit and that."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("start", (0.0, 0.75))
@pytest.mark.parametrize("V,Cp,nout", ((1, 8, 4), (31, 8, 4), (1024, 4, 4), (8191, 8, 3), (8193, 8, 4), (12288, 8, 4),
                                       (120001, 8, 4), (500, 5, 1)))
def test_loss_is_the_rounded_sum_of_its_terms(V, Cp, nout, start):
    import torch
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for -m gpu tests")
    from water_flow_simulation_b200 import _native as nat
    lib, rng = nat.load(), np.random.default_rng(V)
    pred = rng.standard_normal((V, Cp)).astype(np.float32)
    target = rng.standard_normal((V, nout)).astype(np.float32)
    mask = (rng.random(V) > 0.25).astype(np.float32)
    inv_n = np.float32(1.0 / max(mask.sum(), 1.0))
    p, t, m = (torch.as_tensor(a).cuda() for a in (pred, target, mask))
    losses = []
    for _ in range(2):
        dpred, loss = torch.full((V, Cp), 7.0, device="cuda"), torch.full((1,), start, device="cuda")
        nat.check(lib.lbm_nn_mse(p.data_ptr(), Cp, t.data_ptr(), nout, m.data_ptr(), V, float(inv_n), dpred.data_ptr(),
                                 loss.data_ptr(), torch.cuda.current_stream().cuda_stream), "lbm_nn_mse")
        losses.append(loss.cpu().numpy()[0])
    d = pred[:, :nout] - target
    exact = math.fsum([start, *(mask[:, None] * d * d * inv_n).ravel().tolist()])
    assert losses[0] == losses[1]
    assert abs(float(losses[0]) - exact) <= 0.5 * float(np.spacing(losses[0])) + V * nout * 2.0 ** -53 * exact
    grad = np.zeros((V, Cp), np.float32)
    grad[:, :nout] = np.float32(2.0) * mask[:, None] * d * inv_n
    assert np.array_equal(dpred.cpu().numpy(), grad)
    loss.fill_(start)                                      # in place: the gradient over the prediction
    nat.check(lib.lbm_nn_mse(p.data_ptr(), Cp, t.data_ptr(), nout, m.data_ptr(), V, float(inv_n), p.data_ptr(),
                             loss.data_ptr(), torch.cuda.current_stream().cuda_stream), "lbm_nn_mse")
    assert loss.cpu().numpy()[0] == losses[0] and np.array_equal(p.cpu().numpy(), grad)
