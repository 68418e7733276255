"""The closure kernels at the edges of their tiles: point counts around the 16
points of an inference tile and the 64 of a training tile, one-cell-wide
grids (the stencil wraps onto itself), and infinite inputs, against the FP64
restatement.  Tolerance: a product of 135 FP32 terms rounds within
135 x 2^-24 = 8e-6 of its terms' magnitudes; 2e-5 of the largest value leaves
room for the four layers."""
import numpy as np
import pytest

from oracle import closure_oracle as clo

pytestmark = pytest.mark.gpu

INS, OUTS = [0.5, 0.7, 0.9, 1.3], [1.0, 2.0, 0.5, 1.5, 1.0, 0.8, 1.2, 0.9, 1.1]
TOL = 2e-5


def _net(seed):
    from coral_b200.closure import Closure
    net = Closure(seed=seed)
    p = net.params()
    rng = np.random.default_rng(seed)
    k = 0
    for o, i in clo.SIZES:  # biases too
        k += o * i
        p[k:k + o] = 0.1 * rng.standard_normal(o)
        k += o
    net.set_params(p)
    net.set_scales(INS, OUTS)
    return net, p.astype(np.float64)


# 1, 15, 16, 17, 31, 33, 65 points; one column, one row, one z level
@pytest.mark.parametrize("grid", [(1, 1, 1), (1, 3, 5), (4, 4, 1), (1, 17, 1), (31, 1, 1), (1, 1, 33), (13, 1, 5),
                                  (6, 9, 36)])
def test_inference_tiles(grid):
    import torch
    net, p = _net(3)
    rng = np.random.default_rng(1)
    f = rng.standard_normal((4,) + grid)
    tau = torch.full((9,) + grid, float("nan"), dtype=torch.float64, device="cuda")
    net.infer(torch.from_numpy(f).cuda(), tau)
    torch.cuda.synchronize()
    n = int(np.prod(grid))
    ref = clo.forward(p, clo.gather(f, np.arange(n), INS))[-1] * np.array(OUTS)
    assert np.abs(tau.cpu().numpy().reshape(9, -1).T - ref).max() <= TOL * np.abs(ref).max()
    net.close()


@pytest.mark.parametrize("value", [np.inf, -np.inf, 3.4e38, 1e300, np.nan])
def test_inference_of_overflowing_inputs(value):
    """An input beyond BF16's (or FP32's) range saturates the units it reaches,
    as in FP64; NaN stays NaN in its stencil and nowhere else."""
    import torch
    net, p = _net(4)
    rng = np.random.default_rng(2)
    grid = (5, 6, 7)
    f = rng.standard_normal((4,) + grid)
    f[2, 1, 2, 3] = value
    tau = torch.empty((9,) + grid, dtype=torch.float64, device="cuda")
    net.infer(torch.from_numpy(f).cuda(), tau)
    torch.cuda.synchronize()
    with np.errstate(invalid="ignore", over="ignore"):
        ref = clo.forward(p, clo.gather(f, np.arange(5 * 6 * 7), INS))[-1] * np.array(OUTS)
    got = tau.cpu().numpy().reshape(9, -1).T
    assert np.array_equal(np.isnan(got), np.isnan(ref))
    ok = ~np.isnan(ref)
    assert np.abs(got[ok] - ref[ok]).max() <= TOL * np.abs(ref[ok]).max()
    net.close()


# around one training tile, several tiles, more tiles than CTAs
@pytest.mark.parametrize("npts", [1, 15, 63, 64, 65, 300, 148 * 64 + 5])
def test_gradient_tiles(npts):
    import torch
    net, p = _net(5)
    rng = np.random.default_rng(npts)
    grid, nsnap = (6, 5, 9), 3
    n = int(np.prod(grid))
    x = rng.standard_normal((nsnap, 4) + grid).astype(np.float32)
    y = rng.standard_normal((nsnap, 9) + grid).astype(np.float32)
    pts = rng.integers(0, nsnap * n, npts)
    dev = [torch.from_numpy(a).cuda() for a in (x, y, pts)]
    net.zero_gradient()
    loss = net.train(*dev, apply=False)
    g = net.gradient()
    X, T = np.empty((npts, 135)), np.empty((npts, 9))
    for s in range(nsnap):
        at = pts // n == s
        X[at] = clo.gather(x[s].astype(np.float64), pts[at] % n, INS)
        T[at] = y[s].reshape(9, -1)[:, pts[at] % n].T / np.array(OUTS)
    l_ref, g_ref = clo.loss_and_grad(p, X, T)
    assert abs(loss - l_ref) <= TOL * l_ref
    assert np.abs(g - g_ref).max() <= TOL * np.abs(g_ref).max()
    # accumulation over calls, and reading twice
    net.train(*dev, apply=False)
    assert np.abs(net.gradient() - 2 * g_ref).max() <= 2 * TOL * np.abs(g_ref).max()
    assert np.array_equal(net.gradient(), net.gradient())
    net.zero_gradient()
    assert not net.gradient().any()
    net.close()
