"""The separate forward z pass with nine variables (a step with a closure attached) at
the lengths whose passes it groups in its own way: with all parameters of the
closure zero its output is zero, and the step is that of the fused z pass.  Same
transforms, so the tolerance is that of two roundings of the transforms carried
through a step: 1e-11 relative L2, as against the oracle."""
import numpy as np
import pytest

from tests.problems import equations, params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz", [36, 72, 108, 144, 216, 288, 324])
def test_step_with_a_zero_closure(nz):
    from coral_b200.closure import Closure
    from coral_b200.solver import PlaneLayer
    eq, par = equations(), params(12, 16, nz, dt=1e-5)
    net = Closure(seed=1)
    net.set_params(np.zeros_like(net.params()))
    out = []
    for attached in (False, True):
        pl = PlaneLayer(eq, par)
        rng = np.random.default_rng(nz)
        f = rng.standard_normal((2, pl.NXH, pl.NYAA, pl.T[0])) * np.exp(-np.arange(pl.T[0]) / 20.0)
        pl.set_field(0, 1e-2 * (f[0] + 1j * f[1]))
        if attached:
            net.attach(pl)
        pl.march_forward(1e-5, 2)
        pl.synchronize()
        out.append(pl.get_field(0))
        pl.close()
    net.close()
    assert np.isfinite(out[0]).all() and np.linalg.norm(out[1] - out[0]) <= 1e-11 * np.linalg.norm(out[0])
