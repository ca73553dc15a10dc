"""Order-2 transfers of real grids against the oracle, bit for bit, on small
batches (short chunks) and on large ones (many CTAs, long chunks), whose
results on many copies of the same grids must equal the oracle's on each."""
import numpy as np
import pytest

from oracle import gpaw_layer as L
from tests.helpers import to_dev, to_np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('N,pbc', [((34, 38, 70), (0, 0, 0)),
                                   ((32, 36, 66), (1, 1, 1)),
                                   ((10, 130, 64), (0, 1, 0)),
                                   ((6, 8, 6), (1, 0, 1))])
@pytest.mark.parametrize('large', [False, True])
def test_order2_transfers(N, pbc, large, cuda):
    import torch
    from gpaw_b200 import GridDescriptor, Transformer
    gdp, gdo = GridDescriptor(N, 5.0, pbc), L.GridDescriptor(N, 5.0, pbc)
    rng = np.random.default_rng(5)
    a = rng.standard_normal((3,) + tuple(gdo.n_c))
    ref = L.Transformer(gdo, gdo.coarsen(), 1).apply(a)
    back = L.Transformer(gdo.coarsen(), gdo, 1).apply(ref)
    copies = 1
    if large:
        copies = int(148 * 16 * 32 * 16 / ref.size) + 1
    x = to_dev(a).repeat(copies, 1, 1, 1)
    r = Transformer(gdp, gdp.coarsen(), 1).apply(x)
    b = Transformer(gdp.coarsen(), gdp, 1).apply(r)
    for got, want in ((r, ref), (b, back)):
        assert np.array_equal(to_np(got[:3]), want)
        assert torch.equal(got, got[:3].repeat(copies, 1, 1, 1))
