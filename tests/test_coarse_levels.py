"""Which levels of the dielectric solver's V-cycle go into one launch (a fake
library; no GPU needed)."""
from types import SimpleNamespace as NS

import pytest

from gpaw_b200 import _lib
from gpaw_b200.solvation import _CoarseLevels

SIDES = (127, 63, 31, 15, 7)


class FakeLib:
    """Takes levels whose first one has at most `limit` points."""

    def __init__(self, limit):
        self.limit = limit

    def gb_wcoarse_new(self, n, *args):
        if SIDES[len(SIDES) - n]**3 <= self.limit:
            args[-1]._obj.value = 1
        return 0

    def gb_wcoarse_free(self, h):
        pass


def _solver():
    n = len(SIDES)
    array = NS(is_cuda=True, data_ptr=lambda: 8)
    transformer = NS(transformer=NS(_h=None))
    return NS(relax_method=2, levels=n - 1, phis=[array] * n,
              rhos=[array] * n, presmooths=[1] * n, postsmooths=[1] * n,
              weights=[0.5] * n, restrictors=[transformer] * n,
              interpolators=[transformer] * n,
              operators=[NS(gd=NS(n_c=(s, s, s)), operator=NS(_h=None))
                         for s in SIDES])


# clusters of 16 CTAs, of 8, and none
@pytest.mark.parametrize('limit,first', [(32768, 2), (16384, 3), (0, None)])
def test_longest_run_that_the_library_takes(limit, first, monkeypatch):
    monkeypatch.setattr(_lib, 'load', lambda: FakeLib(limit))
    levels = _CoarseLevels.build(_solver())
    assert (levels and levels.first) == first
