"""The band factorisation's shared-memory window against the in-place kernel, bit
for bit, where the window's edges meet the matrix's: the window instances for
bands within (9, 23) and within (15, 31), matrices of fewer rows than the band,
row counts that no chunk of 8 assembled rows divides, partial groups of systems,
and a second factorisation over the first one's storage (dt changed)."""
import numpy as np
import pytest

from tests.problems import params
from tests.test_gpu_shared_factors import _recipe

pytestmark = pytest.mark.gpu


def _run(eq, par, in_place):
    from coral_b200.solver import PlaneLayer
    pl = PlaneLayer(eq, par)
    if in_place:
        pl.set_variant("band_factor", 1)
    rng = np.random.default_rng(5)
    for s in range(pl.n_kxky):
        f = rng.standard_normal((2, pl.NXH, pl.NYAA, pl.T[s])) * np.exp(-np.arange(pl.T[s]) / 20.0)
        pl.set_field(s, 1e-3 * (f[0] + 1j * f[1]))
    out = []
    for dt in (1e-5, 2e-5):
        pl.march_forward(dt, 1)
        out += [pl.get_field(s) for s in range(pl.n_kxky)]
    pl.close()
    return out


@pytest.mark.parametrize("grid", [(4, 4, 8), (12, 16, 12), (24, 12, 16), (8, 8, 36), (8, 12, 108)])
@pytest.mark.parametrize("name", ["rbc_noslip_ra1e5", "rrbc_stressfree_ek1e-4_ra5e7", "toroidal_poloidal"])
def test_window_and_in_place_factors_agree(name, grid):
    eq, par = _recipe(name), params(*grid, dt=1e-5)
    for a, b in zip(_run(eq, par, False), _run(eq, par, True)):
        assert np.isfinite(a).all() and np.array_equal(a, b)


# a workspace of 1 or 3 groups at a time: chunks of one, a last one that is partial
@pytest.mark.parametrize("chunk", [1, 3])
@pytest.mark.parametrize("name", ["rbc_noslip_ra1e5", "rrbc_stressfree_ek1e-4_ra5e7"])
def test_chunked_factorisation_agrees(name, chunk, monkeypatch):
    eq, par = _recipe(name), params(24, 24, 16, dt=1e-5)
    whole = _run(eq, par, False)
    monkeypatch.setenv("CORAL_FACTOR_CHUNK", str(chunk))
    for a, b in zip(whole, _run(eq, par, False)):
        assert np.array_equal(a, b)
