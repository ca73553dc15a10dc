"""Which kernels an operator's stencil takes (no GPU needed)."""
import numpy as np
import pytest

from gpaw_b200 import _lib, cgpaw

TILED, GENERAL, GENERIC = 2, 1, 0
N = (12, 14, 16)


def _path(offsets, cfd=None, size=N):
    offsets = np.array(offsets)
    r = int(np.abs(offsets).max())
    if cfd is None:
        cfd = bool((np.count_nonzero(offsets, axis=1) <= 1).all())
    M = np.array(size) + 2 * r
    flat = offsets @ np.array([M[1] * M[2], M[2], 1])
    op = cgpaw.Operator(np.ones(len(flat)), flat, size, r, [[0, 0]] * 3,
                        True, None, cfd)
    return _lib.load().gb_operator_path(op._h)


def _axes(order, nn):
    out = [(0, 0, 0)]
    for axis in order:
        for sign in (1, -1):
            for d in range(1, nn + 1):
                o = [0, 0, 0]
                o[axis] = sign * d
                out.append(tuple(o))
    return out


@pytest.mark.parametrize('nn', [1, 3, 6])
def test_axis_order(nn):
    """Only the order of the Laplacians, axis 2 first, takes the kernels that
    are written for it."""
    assert _path(_axes((2, 1, 0), nn)) == TILED
    for order in [(0, 1, 2), (2, 0, 1), (1, 2, 0)]:
        assert _path(_axes(order, nn)) == GENERAL


def test_generic_path_on_request(monkeypatch):
    """GPAW_B200_FD_PATH=generic: one thread a point for every stencil, so
    that the other kernels can be compared with it."""
    skew = [(0, 0, 0), (1, -1, 0), (-1, 1, 0), (0, 2, 1)]
    assert _path(skew) == GENERAL
    monkeypatch.setenv('GPAW_B200_FD_PATH', 'generic')
    assert _path(skew) == GENERIC
    assert _path(_axes((2, 1, 0), 3)) == GENERIC


def test_stencils_left_to_the_generic_path():
    """Ranges above 6, and diagonal taps declared axis-aligned (their corner
    values read zero)."""
    assert _path([(0, 0, 0), (7, -1, 0)]) == GENERIC
    assert _path([(0, 0, 0), (1, 1, 0)], cfd=True) == GENERIC
    assert _path([(0, 0, 0), (1, 1, 0)], cfd=False) == GENERAL
