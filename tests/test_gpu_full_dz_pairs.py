"""Steps of a recipe with dense operators and z derivatives in its full variables
(toroidal-poloidal) against the oracle, at the edges of the kernels
that take several systems or columns a CTA: grids below and above the size from
which the right-hand side and K_std take two systems a CTA (0.75 N^2 systems, from
1184 on), and z lengths of 12 to 108 (column strides in shared memory; even and odd
chains of 6 to 54 divides).  Tolerance 1e-11 relative L2 per variable, that of the
other steps against the oracle."""
import pytest

from tests.problems import params
from tests.test_gpu_parity_sizes import _steps_match
from tests.test_gpu_shared_factors import _recipe

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid", [(4, 4, 12), (8, 12, 108), (36, 36, 16), (48, 36, 24)])
def test_toroidal_poloidal_steps_match_oracle(grid):
    _steps_match(_recipe("toroidal_poloidal"), params(*grid, dt=1e-6), dt=1e-6, nsteps=2, seed=31, amp=1e-3)
