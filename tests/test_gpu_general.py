"""The tiled kernel for general stencils against the oracle, bit for bit (the
same operations in the same order), at planes that its tiles divide evenly
or not, every range it takes and one it does not."""
import numpy as np
import pytest

from oracle import gpaw_layer as L
from tests.helpers import to_dev, to_np

pytestmark = pytest.mark.gpu

SKEW = np.array([[1.0, 0, 0], [-0.5, np.sqrt(0.75), 0], [0, 0, 1.1]])
FCC = np.array([[0, 1.0, 1.0], [1.0, 0, 1.0], [1.0, 1.0, 0]])


def _pair(N, cell, pbc, coefs, offsets, dtype):
    from gpaw_b200 import FDOperator, GridDescriptor
    c = cell * 0.4 * np.array(N)[:, None]
    gdp, gdo = GridDescriptor(N, c, pbc), L.GridDescriptor(N, c, pbc)
    return (gdp, FDOperator(coefs, offsets, gdp, dtype),
            gdo, L.FDOperator(coefs, offsets, gdo, dtype))


def _data(rng, shape, dtype):
    x = rng.standard_normal(shape)
    return x + 1j * rng.standard_normal(shape) if dtype is complex else x


@pytest.mark.parametrize('dtype', [float, complex])
@pytest.mark.parametrize('N,pbc', [((7, 17, 33), (1, 1, 1)),
                                   ((9, 16, 32), (0, 0, 0)),
                                   ((20, 31, 65), (1, 0, 1)),
                                   ((8, 8, 8), (0, 1, 1))])
@pytest.mark.parametrize('r', [1, 2, 3, 4, 6, 7])
def test_general_stencil(N, pbc, r, dtype, cuda):
    rng = np.random.default_rng(r)
    if (np.array(N) - (1 - np.array(pbc)) < r).any():
        pytest.skip('stencil longer than the grid')
    offsets = [(0, 0, 0), (r, -r, r), (-r, 0, 1), (0, r, -1), (0, 0, -r),
               (1, 1, 0), (-1, -1, -1), (0, -r, r), (r, 0, 0)]
    coefs = rng.standard_normal(len(offsets))
    gdp, op, gdo, oo = _pair(N, SKEW, pbc, coefs, offsets, dtype)
    ph = gdo.phase_factor_cd((0.2, -0.35, 0.1)) if dtype is complex else None
    a = _data(rng, (2,) + tuple(gdo.n_c), dtype)
    rho = _data(rng, a.shape, dtype)
    ref = np.zeros_like(a)
    oo.apply(a, ref, ph)
    x, out = to_dev(a), to_dev(np.zeros_like(a))
    op.apply(x, out, ph)
    assert np.array_equal(to_np(out), ref)
    res = x.new_zeros(x.shape)
    op.residual(x, to_dev(rho), res, ph)
    assert np.array_equal(to_np(res), ref - rho)
    v = rng.standard_normal(tuple(gdo.n_c))
    op.apply_potential(x, out, to_dev(v), ph)
    assert np.array_equal(to_np(out), ref + a * v)
    if dtype is float:
        b, c = a[0].copy(), to_dev(a[0].copy())
        oo.relax(2, b, rho[0], 3, 0.7)
        op.relax(2, c, to_dev(rho[0]), 3, 0.7)
        assert np.array_equal(to_np(c), b)


@pytest.mark.parametrize('cell', ['hex', 'fcc'])
@pytest.mark.parametrize('nn', [1, 3, 5])
def test_general_laplacian(cell, nn, cuda):
    from gpaw_b200 import GridDescriptor, Laplace
    N = (34, 34, 18) if cell == 'hex' else (18, 18, 18)
    c = (SKEW if cell == 'hex' else FCC) * 0.4 * np.array(N)[:, None]
    gdp, gdo = GridDescriptor(N, c, 1), L.GridDescriptor(N, c, 1)
    ph = gdo.phase_factor_cd((0.25, 0.0, 0.1))
    a = _data(np.random.default_rng(1), (3,) + N, complex)
    ref = np.zeros_like(a)
    L.Laplace(gdo, -0.5, nn, complex).apply(a, ref, ph)
    out = to_dev(np.zeros_like(a))
    Laplace(gdp, -0.5, nn, complex).apply(to_dev(a), out, ph)
    assert np.array_equal(to_np(out), ref)


@pytest.mark.parametrize('dtype', [float, complex])
@pytest.mark.parametrize('nn', [1, 3])
def test_axis_aligned_in_another_order(nn, dtype, cuda):
    """Centre, then the axes in the order 0, 1, 2: laid out as a Laplacian is,
    but not summed in its order.  The residual's norm has one partial sum for
    each block of the kernel that runs (few or many planes, one grid or
    more).  Tolerance: the sums' order, n eps."""
    import torch
    rng = np.random.default_rng(nn)
    offsets = [(0, 0, 0)]
    for axis in range(3):
        for sign in (1, -1):
            for d in range(1, nn + 1):
                o = [0, 0, 0]
                o[axis] = sign * d
                offsets.append(tuple(o))
    coefs = rng.standard_normal(len(offsets))
    for N, nin in (((64, 64, 64), 1), ((10, 33, 70), 5), ((90, 12, 8), 2)):
        gdp, op, gdo, oo = _pair(N, np.eye(3), (1, 0, 1), coefs, offsets,
                                 dtype)
        a = _data(rng, (nin,) + tuple(gdo.n_c), dtype)
        rho = _data(rng, a.shape, dtype)
        ref = np.zeros_like(a)
        ph = gdo.phase_factor_cd((0.2, 0, 0.1)) if dtype is complex else None
        oo.apply(a, ref, ph)
        x, res = to_dev(a), to_dev(np.zeros_like(a))
        norm = torch.zeros(nin, dtype=torch.float64, device='cuda')
        op.operator.residual(x, to_dev(rho), res, ph, 0.5, norm)
        assert np.array_equal(to_np(res), ref - rho)
        want = 0.5 * (np.abs(ref - rho)**2).reshape(nin, -1).sum(1)
        assert np.abs(to_np(norm) / want - 1).max() < 1e-13 * a[0].size**0.5
