"""Relative accuracy of the closure's inference from inputs of order one down to
nearly quiescent ones: zero biases and no weight on the wall coordinate, so that the
pre-activations are as small as the fields, against the FP64 restatement.
Tolerance: 1e-6 of the largest output.  Every operation rounds within 2^-24 = 6e-8
of its value at any scale; random signs over the 11 sums a layer adds up (9 steps,
bias and activation at most) and 4 layers give sqrt(44) x 6e-8 = 4e-7.  A lost BF16
plane of the activations is 2^-17 = 8e-6, and an activation function that is good
to an absolute 1e-7 only is 1e-4 of an output at inputs of 0.001."""
import numpy as np
import pytest

from oracle import closure_oracle as clo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1.0, 0.1, 1e-2, 1e-3, 1e-5, 1e-8])
def test_inference_keeps_relative_accuracy(scale):
    import torch
    from coral_b200.closure import Closure
    net = Closure(seed=7)
    p = net.params().astype(np.float64)  # as created: zero biases
    p[:clo.HID * clo.NIN].reshape(clo.HID, clo.NIN)[:, 4 * clo.TAPS:] = 0.0
    net.set_params(p.astype(np.float32))
    grid = (6, 9, 36)
    f = scale * np.random.default_rng(1).standard_normal((4,) + grid)
    tau = torch.empty((9,) + grid, dtype=torch.float64, device="cuda")
    net.infer(torch.from_numpy(f).cuda(), tau)
    torch.cuda.synchronize()
    n = int(np.prod(grid))
    ref = clo.forward(p, clo.gather(f, np.arange(n), [1.0] * 4))[-1]
    assert np.abs(tau.cpu().numpy().reshape(9, -1).T - ref).max() <= 1e-6 * np.abs(ref).max()
    net.close()
