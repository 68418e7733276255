"""The memory of the band factors, and their packing in place.  A recipe without the ky
mirror symmetry holds its factors once, as one with it does (its units half as many,
packed form beside them); staged a few groups at a time, a partial last chunk
included, the packed factors give the same steps bit for bit."""
import numpy as np
import pytest

from tests.problems import params
from tests.test_gpu_shared_factors import _recipe, _run

pytestmark = pytest.mark.gpu

MIRROR, ROTATING = "rbc_noslip_ra1e5", "rrbc_stressfree_ek1e-4_ra5e7"


def test_factors_are_held_once():
    from coral_b200.solver import PlaneLayer
    held = []
    for name in (MIRROR, ROTATING):
        pl = PlaneLayer(_recipe(name), params(96, 96, 96))
        held.append(pl.query(11))
        pl.close()
    # 48 x 95 - 1 systems of two blocks of at least 280 columns, 34 doubles each
    factors = (48 * 95 - 1) * 2 * 280 * 34 * 8
    assert abs(held[1] - held[0]) <= factors / 4, (held, factors)


# 275 units in groups of 32, 143 in groups of 16: 9 groups either way
@pytest.mark.parametrize("chunk", [2, 4, 5, 8])
@pytest.mark.parametrize("name,upw", [(MIRROR, 16), (ROTATING, 32)])
def test_partial_last_chunk_agrees(name, upw, chunk, monkeypatch):
    eq, par = _recipe(name), params(24, 24, 16, dt=1e-5)
    monkeypatch.delenv("CORAL_FACTOR_CHUNK", raising=False)
    whole, units, _ = _run(eq, par, 4)
    groups = -(-units // upw)
    assert groups % chunk != 0 and groups > chunk
    monkeypatch.setenv("CORAL_FACTOR_CHUNK", str(chunk))
    for a, b in zip(whole, _run(eq, par, 4)[0]):
        assert np.isfinite(a).all() and np.array_equal(a, b)
