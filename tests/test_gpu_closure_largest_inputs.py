"""Inference with two inputs of opposite sign at the top of FP32's range under one
unit: weights of 1/4 and 1/8 either way keep the first layer's sums finite and away
from zero (0.125 or 0.375 of the value), so that the units saturate as in FP64 and
nothing becomes NaN.  Values from 3.397e38 on round to infinity in BF16.  Tolerance
2e-5 of the largest output, that of the other tests of the kernel's edges."""
import numpy as np
import pytest

from oracle import closure_oracle as clo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [1e38, 3.39e38, 3.397e38, float(np.finfo(np.float32).max)])
def test_inputs_of_opposite_sign(value):
    import torch
    from coral_b200.closure import Closure
    net = Closure(seed=4)
    p = net.params().astype(np.float64)
    W0 = p[:clo.HID * clo.NIN].reshape(clo.HID, clo.NIN)
    W0[:] = 0.0
    unit, centre = np.arange(clo.HID), 13
    W0[:, 2 * clo.TAPS + centre] = 0.25 * np.where(unit & 1, 1, -1)
    W0[:, centre] = 0.125 * np.where(unit & 2, 1, -1)
    net.set_params(p.astype(np.float32))
    grid = (5, 6, 7)
    f = np.random.default_rng(2).standard_normal((4,) + grid)
    f[2, 1, 2, 3], f[0, 1, 2, 3] = value, -value
    tau = torch.empty((9,) + grid, dtype=torch.float64, device="cuda")
    net.infer(torch.from_numpy(f).cuda(), tau)
    torch.cuda.synchronize()
    ref = clo.forward(p, clo.gather(f, np.arange(5 * 6 * 7), [1.0] * 4))[-1]
    got = tau.cpu().numpy().reshape(9, -1).T
    assert np.isfinite(got).all() and np.abs(got - ref).max() <= 2e-5 * np.abs(ref).max()
    net.close()
