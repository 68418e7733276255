"""The fused z pass where its lines meet the shared memory of an SM: a recipe with 7
full variables at NZ 384 (padded lines of 599 elements: batches of 9 lines do not
fit, batches of 6 do) and at NZ 192 (one CTA an SM with 9, two with 6), one step
against the oracle, with the 9-line and the 6-line setting, on the smallest
horizontal grid.  Tolerance 1e-11 relative L2, that of the other steps against the
oracle: changing this state by 1e-16 of each entry changes the oracle's step by
2e-13 at most, so it is 50 times what one rounding of every input does."""
import numpy as np
import pytest

from oracle import coral_oracle as co
from tests.problems import ROOT, params

pytestmark = pytest.mark.gpu


def _close(a, b):
    return np.linalg.norm(a - b) <= 1e-11 * np.linalg.norm(b)


@pytest.mark.parametrize("lines", [9, 6])
@pytest.mark.parametrize("nz", [192, 384])
def test_seven_full_variables_match_oracle(nz, lines):
    from coral_b200.solver import PlaneLayer
    with open(ROOT + "/tests/golden/examples/coral.equations.convective_dynamo") as f:
        eq = f.read()
    par = params(4, 4, nz, dt=1e-6)
    pl, ref = PlaneLayer(eq, par), co.Solver(eq, par)
    assert pl.query(8) == 7
    pl.set_variant("z_pass", 0 if lines == 6 else 1)
    rng = np.random.default_rng(3)
    for s, lay in enumerate(ref.lay):
        f = rng.standard_normal((2, pl.NXH, pl.NYAA, lay.T)) * np.exp(-np.arange(lay.T) / 20.0)
        ref.field[s] = 1e-3 * (f[0] + 1j * f[1])
        pl.set_field(s, ref.field[s])
    for s, lay in enumerate(ref.zlay):
        ref.zfield[s] = 1e-3 * rng.standard_normal(lay.T) * np.exp(-np.arange(lay.T) / 20.0)
        pl.set_mean_field(s, ref.zfield[s])
    ref.step(1e-6)
    pl.march_forward(1e-6, 1)
    pl.synchronize()
    for s, lay in enumerate(ref.lay):
        got = pl.get_field(s)
        for idx in lay.var_pos:
            assert _close(got[..., idx], ref.field[s][..., idx])
    for s in range(len(ref.zlay)):
        assert _close(pl.get_mean_field(s), ref.zfield[s])
    pl.close()
