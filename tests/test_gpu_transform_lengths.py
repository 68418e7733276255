"""Transforms and a step at every transform length with merged FFT passes (3 N / 2 =
54 .. 486 for N = 36 .. 324, none a power-of-two multiple of 24), along each axis
against the oracle.  Tolerance: that of the other transform tests, 1e-13 of the
largest value (a length-486 FFT rounds within a few 1e-16 of it)."""
import numpy as np
import pytest

from oracle import coral_oracle as co
from tests.problems import equations, params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [36, 72, 108, 144, 216, 288, 324])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_transform_length(n, axis):
    from coral_b200.solver import PlaneLayer
    grid = [12, 16, 12]
    grid[axis] = n
    pl = PlaneLayer(equations(), params(*grid))
    g = co.Solver(equations(), params(*grid)).g
    rng = np.random.default_rng(n + axis)
    spec = rng.standard_normal((pl.NXH, pl.NYAA, pl.NZ)) + 1j * rng.standard_normal((pl.NXH, pl.NYAA, pl.NZ))
    ref = co.spec_to_phys(spec, g)
    assert np.abs(pl.spec_to_phys(spec) - ref).max() <= 1e-13 * np.abs(ref).max()
    phys = rng.standard_normal((pl.NYAA, pl.NXAA, pl.NZAA))
    ref = co.phys_to_spec(phys, g)
    assert np.abs(pl.phys_to_spec(phys) - ref).max() <= 1e-13 * np.abs(ref).max()
    pl.close()


@pytest.mark.parametrize("grid", [(36, 16, 72), (16, 108, 36), (72, 36, 12)])
def test_step_at_merged_lengths(grid):
    """The fused z pass at 54 and 108 points, the single-term y build at 54 and 162."""
    from coral_b200.solver import PlaneLayer
    eq, par = equations(), params(*grid, dt=1e-5)
    pl, ref = PlaneLayer(eq, par), co.Solver(eq, par)
    rng = np.random.default_rng(7)
    f = 1e-2 * (rng.standard_normal(ref.field[0].shape) + 1j * rng.standard_normal(ref.field[0].shape))
    pl.set_field(0, f)
    ref.field[0] = f.copy()
    for _ in range(2):
        ref.step(1e-5)
    pl.march_forward(1e-5, 2)
    pl.synchronize()
    assert np.linalg.norm(pl.get_field(0) - ref.field[0]) <= 1e-11 * np.linalg.norm(ref.field[0])
    pl.close()
