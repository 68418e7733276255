"""The band substitution with one LU factorisation per (kx, ky), (kx, -ky) pair:
recipes whose operators have that mirror symmetry share factors, others do not,
and either way the step is that of one factorisation per system bit for bit
(signs commute with rounding and with the pivot search)."""
import numpy as np
import pytest

from tests.problems import ROOT, equations, params

pytestmark = pytest.mark.gpu


def _recipe(name):
    if name == "toroidal_poloidal":  # operators in kx^2 + ky^2 only; band within (15, 31)
        with open(ROOT + "/tests/golden/benchmark02/coral.equations.toroidalPoloidal") as f:
            return f.read()
    return equations(name)


def _run(eq, par, seed, variants=()):
    from coral_b200.solver import PlaneLayer
    pl = PlaneLayer(eq, par)
    for knob, value in variants:
        pl.set_variant(knob, value)
    rng = np.random.default_rng(seed)
    for s in range(pl.n_kxky):
        f = rng.standard_normal((2, pl.NXH, pl.NYAA, pl.T[s])) * np.exp(-np.arange(pl.T[s]) / 20.0)
        pl.set_field(s, 1e-3 * (f[0] + 1j * f[1]))
    pl.march_forward(1e-5, 3)
    pl.synchronize()
    out = [pl.get_field(s) for s in range(pl.n_kxky)]
    units, nact = pl.query(1300), sum(1 for _ in _active(pl))
    pl.close()
    return out, units, nact


def _active(pl):
    NY = 2 * pl.NYAA // 3
    for ix in range(pl.NXH):
        for iy in range(pl.NYAA):
            ky = iy if iy <= pl.NYAA // 2 else iy - pl.NYAA
            if 2 * abs(ky) < NY and (ix, iy) != (0, 0):
                yield ix, ky


# 4 x 4: 1 active ky either side and 5 units, fewer than a group; 12 x 16 and
# 24 x 12: groups with a partial last one; NZ 8 and 12: fewer columns than the
# copies run ahead
@pytest.mark.parametrize("grid", [(4, 4, 8), (12, 16, 12), (24, 12, 16), (16, 24, 48)])
@pytest.mark.parametrize("name,mirror", [("rbc_noslip_ra1e5", True), ("rrbc_stressfree_ek1e-4_ra5e7", False),
                                         ("toroidal_poloidal", True)])
def test_shared_factors_are_bitwise_neutral(name, mirror, grid, monkeypatch):
    eq, par = _recipe(name), params(*grid, dt=1e-5)
    monkeypatch.delenv("CORAL_NO_KY_MIRROR", raising=False)
    got, units, nact = _run(eq, par, 1)
    monkeypatch.setenv("CORAL_NO_KY_MIRROR", "1")
    ref, all_units, _ = _run(eq, par, 1)
    assert all_units == nact
    # systems with ky < 0 share their partner's unit
    pairs = sum(1 for ix, ky in _iter(grid) if ky < 0)
    assert units == (nact - pairs if mirror else nact)
    for a, b in zip(got, ref):
        assert np.isfinite(a).all() and np.array_equal(a, b)


def _iter(grid):
    NX, NY, _ = grid
    for ix in range(NX // 2):
        for ky in range(-(NY // 2) + 1, NY // 2):
            if (ix, ky) != (0, 0):
                yield ix, ky


@pytest.mark.parametrize("name", ["rbc_noslip_ra1e5", "rrbc_stressfree_ek1e-4_ra5e7"])
def test_wider_band_instance_is_bitwise_neutral(name):
    """Band (9, 23) recipes through the instance for bands within (15, 31)."""
    eq, par = _recipe(name), params(16, 12, 24, dt=1e-5)
    a, _, _ = _run(eq, par, 2)
    b, _, _ = _run(eq, par, 2, variants=[("band_substitution", 1)])
    assert all(np.array_equal(x, y) for x, y in zip(a, b))


def test_ensemble_of_shared_and_unshared_factors():
    """One batched substitution over members with and without the symmetry."""
    from coral_b200.ensemble import Ensemble
    from coral_b200.solver import PlaneLayer
    eqs = [_recipe("rbc_noslip_ra1e5"), _recipe("rrbc_stressfree_ek1e-4_ra5e7"), _recipe("rbc_noslip_ra1e5")]
    pars = [params(12, 16, 16, dt=1e-5), params(16, 12, 24, dt=1e-5), params(24, 12, 12, dt=1e-5)]
    ens = Ensemble(eqs, pars)
    rng = np.random.default_rng(3)
    singles = []
    for m, eq, par in zip(ens.members, eqs, pars):
        f = 1e-3 * rng.standard_normal((m.NXH, m.NYAA, m.T[0])) * (1 + 0.5j)
        m.set_field(0, f)
        pl = PlaneLayer(eq, par)
        pl.set_field(0, f)
        pl.march_forward(1e-5, 3)
        pl.synchronize()
        singles.append(pl.get_field(0))
        pl.close()
    ens.march_forward(1e-5, 3)
    ens.synchronize()
    assert ens.batched
    for m, s in zip(ens.members, singles):
        assert np.array_equal(m.get_field(0), s)
    ens.close()
