"""The training loss of a large batch: 2^22 times the same point must give the loss of
64 times that point, the mean of equal terms.  Both counts are powers of two, so the
mean's factor is exact, a point's nine squares are summed in the same FP32 order on
both sides, and the sums over points are in FP64: equal to 2^22 x 2^-53 = 5e-10.  (In
FP32 each thread's chain of some 400 tiles rounds within 1e-6.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("point", [0, 77, 269])
def test_loss_does_not_drift_with_the_batch(point):
    import torch
    from coral_b200.closure import Closure
    net = Closure(seed=11)
    rng = np.random.default_rng(point)
    grid = (6, 5, 9)
    x = torch.from_numpy(rng.standard_normal((1, 4) + grid).astype(np.float32)).cuda()
    y = torch.from_numpy(rng.standard_normal((1, 9) + grid).astype(np.float32)).cuda()
    losses = [net.train(x, y, torch.full((n,), point, dtype=torch.int64, device="cuda"), apply=False)
              for n in (64, 1 << 22)]
    net.close()
    assert abs(losses[1] - losses[0]) <= 5e-10 * losses[0]
