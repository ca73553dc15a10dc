"""Interpolation of a density off periodic cells, rescaled from the coarse
grid, against the oracle: values that are not finite leave the same points as
they were and spoil the same ones."""
import numpy as np
import pytest

from oracle import gpaw_layer as L
from tests.helpers import to_dev, to_np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('value', [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize('n', [1, 2, 3, 4])
def test_values_that_are_not_finite(n, value, cuda):
    from gpaw_b200 import GridDescriptor
    from gpaw_b200.pot_calc import FDDensityTransfers
    N, pbc = (20, 24, 22), (0, 1, 0)
    gdp, gdo = GridDescriptor(N, 5.0, pbc), L.GridDescriptor(N, 5.0, pbc)
    nt = np.random.default_rng(n).random((3,) + tuple(gdo.n_c))
    nt[1, 7, 9, 11] = value
    with np.errstate(invalid='ignore'):
        ref = L.interpolate_density(gdo, gdo.refine(), nt, n)
    got = to_np(FDDensityTransfers(gdp, gdp.refine(), n)
                .interpolate_density(to_dev(nt)))
    ok = np.isfinite(ref)
    assert ok[[0, 2]].all()
    assert np.array_equal(np.isfinite(got), ok)
    # sums in another order: n eps of 10^4 points at most
    assert np.abs(got[ok] / ref[ok] - 1).max() < 1e-11
