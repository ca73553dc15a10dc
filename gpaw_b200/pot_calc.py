"""Grid transfers of the finite-difference potential calculator
(drop-in for the transfer part of gpaw/new/fd/pot_calc.py).

``FDPotentialCalculator`` moves densities from the wave-function grid to the
fine grid (twice as many points per axis) with a tri-linear .. tri-heptic
interpolation and potentials back with the matching restriction
(gpaw/new/fd/pot_calc.py:37-41, 57-61).  On grids that are not periodic in
every direction the interpolated density is rescaled so that its integral
equals the coarse one (:72-80).  Both transfers are the sm_100a
``Transformer`` kernels; the fine integral is a weighted sum over the coarse
grid (the interpolation's column sums), so both integrals come from one read
of it and the interpolation writes rescaled values.
"""
from __future__ import annotations

import ctypes as C
import functools

import numpy as np
import torch

from ._lib import check
from .cgpaw import _stream
from .transformers import Transformer


@functools.lru_cache(maxsize=256)
def interpolation_column_sums(nc, nf, periodic, plo, skip, nn):
    """Sum over the nf fine points of the order-2nn interpolation weights of
    each of nc coarse points (one axis; plo: input padding below, skip: first
    fine point omitted, as transformer_geometry gives them)."""
    x = np.arange(2 * nn) - nn + 0.5
    u = np.arange(nf) + skip
    m = nn - 1 + u // 2 - plo           # coarse point at or below u
    even = u % 2 == 0
    index, weight = [m[even]], [np.ones(int(even.sum()))]
    for j in range(nn):
        others = np.delete(x, nn + j)
        w = np.prod(-others / (x[nn + j] - others))
        for k in (m[~even] - j, m[~even] + 1 + j):
            index.append(k)
            weight.append(np.full(len(k), w))
    index, weight = np.concatenate(index), np.concatenate(weight)
    if periodic:
        index = index % nc
    else:
        ok = (index >= 0) & (index < nc)
        index, weight = index[ok], weight[ok]
    out = np.bincount(index, weight, nc)
    out.setflags(write=False)
    return out


_NAMES = ['linear', 'cubic', 'quintic', 'heptic']


class FDDensityTransfers:
    """interpolate / restrict / interpolate_density of FDPotentialCalculator
    for a wave-function grid ``gd`` and its refinement ``finegd``."""

    def __init__(self, gd, finegd, interpolation_stencil_range=3,
                 dtype=float):
        self.grid = gd
        self.fine_grid = finegd
        n = int(interpolation_stencil_range)
        self.interpolation_stencil_range = n
        self._interpolate = Transformer(gd, finegd, n, dtype)
        self._restrict = Transformer(finegd, gd, n, dtype)
        # the column sums go to the device now, so that a first call may be
        # under a stream capture (a synchronous copy; with their computation
        # 0.13 ms for axis lengths that were not met before, 0.03 ms for
        # others; a rescaled interpolation takes 0.06 to 0.09 ms less for
        # them)
        self._weights = None
        if getattr(self._interpolate, 'dtype', None) is float and \
                not bool(gd.pbc_c.all()) and torch.cuda.is_available():
            self._upload_column_sums()

    def _upload_column_sums(self):
        t = self._interpolate
        w = [interpolation_column_sums(
            t.ngpin[c], t.ngpout[c], bool(self.grid.pbc_c[c]),
            int(t.pad_cd[c, 0]), int(t.skip_cd[c, 0]), t.nn)
            for c in range(3)]
        self._weights = torch.from_numpy(np.concatenate(w)).to(
            self.grid.device)

    def _column_sums(self):
        """Device addresses of the three axes' column sums."""
        if self._weights is None:
            self._upload_column_sums()
        p = self._weights.data_ptr()
        n = self._interpolate.ngpin
        return (C.c_void_p * 3)(p, p + 8 * n[0], p + 8 * (n[0] + n[1]))

    def __str__(self):
        degree = self.interpolation_stencil_range * 2 - 1
        name = _NAMES[degree // 2]
        return (f'interpolation: tri-{name}' +
                f' # {degree}. degree polynomial\n')

    def interpolate(self, a_xR, a_xr=None):
        """gpaw/new/fd/pot_calc.py:57-58."""
        return self._interpolate.apply(a_xR, a_xr)

    def restrict(self, a_xr, a_xR=None):
        """gpaw/new/fd/pot_calc.py:60-61."""
        return self._restrict.apply(a_xr, a_xR)

    def interpolate_density(self, nt_sR, nt_sr=None):
        """_interpolate_density (gpaw/new/fd/pot_calc.py:72-80): the
        interpolated density, each spin rescaled to the coarse integral
        when the grid is not periodic in all directions (skipped where the
        fine integral is 1e-14 or less).  Returns nt_sr."""
        t = self._interpolate
        if not bool(self.grid.pbc_c.all()) and \
                getattr(t, 'dtype', None) is float and nt_sR.is_cuda and \
                nt_sR.dtype == torch.float64 and nt_sR.dim() in (3, 4) and \
                nt_sR.numel() > 0:
            if nt_sr is None:
                nt_sr = self.fine_grid.empty(tuple(nt_sR.shape[:-3]))
            t.transformer.check_arrays(nt_sR, nt_sr)
            nin = nt_sR.numel() // (t.ngpin[0] * t.ngpin[1] * t.ngpin[2])
            lib = t.transformer._lib
            ndoubles = lib.gb_density_work(nin)
            if ndoubles:
                work = nt_sR.new_empty(ndoubles)
                check(lib.gb_density_interpolate(
                    t.transformer._h, C.c_void_p(nt_sR.data_ptr()),
                    C.c_void_p(nt_sr.data_ptr()), nin, self._column_sums(),
                    float(self.grid.dv), float(self.fine_grid.dv),
                    C.c_void_p(work.data_ptr()), _stream()))
                return nt_sr
        nt_sr = self.interpolate(nt_sR, nt_sr)
        if not bool(self.grid.pbc_c.all()):
            shape = nt_sR.shape[:-3]
            one = len(shape) == 0
            c = nt_sR.reshape((1,) + tuple(nt_sR.shape[-3:])) if one \
                else nt_sR.reshape((-1,) + tuple(nt_sR.shape[-3:]))
            f = nt_sr.reshape((1,) + tuple(nt_sr.shape[-3:])) if one \
                else nt_sr.reshape((-1,) + tuple(nt_sr.shape[-3:]))
            Nt1 = c.reshape(c.shape[0], -1).sum(dim=1) * self.grid.dv
            Nt2 = f.reshape(f.shape[0], -1).sum(dim=1) * self.fine_grid.dv
            scale = torch.where(Nt2 > 1e-14, Nt1 / Nt2,
                                torch.ones_like(Nt2))
            f.mul_(scale.view(-1, 1, 1, 1))
        return nt_sr
