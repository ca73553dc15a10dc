"""Eigenvectors of the one-dimensional parts of an axis-aligned stencil.

On an orthorhombic grid the operator is T0 + T1 + T2 with one symmetric
n x n matrix an axis, so three small eigenproblems diagonalise it (fast
diagonalisation: Lynch, Rice and Thomas, Numer. Math. 6, 185 (1964)).  Each
matrix commutes with a reflection of its points, j <-> n - 1 - j for a zero
boundary and j <-> (n - j) mod n for a periodic one, so its eigenvectors
split into even and odd ones, given here as two half-size blocks.
"""
from __future__ import annotations

import functools

import numpy as np

# The direct correction takes at most this many modes of one parity an axis
# (one warp for twelve of them, sixteen warps a block).
MAX_HALF = 192


def half_sizes(n, periodic):
    """Even and odd modes of an axis of n points."""
    he = n // 2 + 1 if periodic else (n + 1) // 2
    return he, n - he


@functools.lru_cache(maxsize=128)
def axis_modes(n, periodic, taps):
    """Even block, odd block ([point][mode]; the columns have unit norm over
    the n points) and the eigenvalues (even first) of
    (T x)_j = sum_d taps[d - 1] (x_{j + d} - 2 x_j + x_{j - d}).

    The smooth modes' eigenvalues are small beside |T| (by (pi / n)^2), and
    an eigensolver gives them to rounding of |T|; they are recomputed to
    their own rounding (closed form, or the Rayleigh quotient, whose error is
    quadratic in the vector's, in extended precision)."""
    he, ho = half_sizes(n, periodic)
    if periodic:
        j, k = np.arange(he), np.arange(he)
        even = np.sqrt(2.0 / n) * np.cos(2 * np.pi / n * np.outer(j, k))
        even[:, 0] = np.sqrt(1.0 / n)
        if n % 2 == 0:
            even[:, -1] = np.sqrt(1.0 / n) * (-1.0)**j
        m = np.arange(1, ho + 1)
        odd = np.sqrt(2.0 / n) * np.sin(2 * np.pi / n * np.outer(m, m))

        def lam(q):
            return sum(-4.0 * t * np.sin(np.pi / n * (d + 1) * q)**2
                       for d, t in enumerate(taps))
        values = np.concatenate([lam(k), lam(m)])
    else:
        T = np.zeros((n, n))
        for d, t in enumerate(taps, 1):
            if d < n:
                T += t * (np.eye(n, k=d) + np.eye(n, k=-d))
        mirror = T[:ho, ::-1][:, :ho]
        Te = np.zeros((he, he))
        Te[:ho, :ho] = T[:ho, :ho] + mirror
        if he > ho:
            Te[:ho, ho] = Te[ho, :ho] = np.sqrt(2.0) * T[:ho, ho]
            Te[ho, ho] = T[ho, ho]
        even = np.linalg.eigh(Te)[1]
        even[:ho] *= np.sqrt(0.5)
        odd = np.zeros((0, 0))
        if ho:
            odd = np.linalg.eigh(T[:ho, :ho] - mirror)[1] * np.sqrt(0.5)
        full = np.zeros((n, n), np.longdouble)
        full[:he, :he] = even
        full[:ho, he:] = odd
        full[n - ho:, :he] = even[:ho][::-1]
        full[n - ho:, he:] = -odd[::-1]
        Tv = np.zeros_like(full)
        for d, t in enumerate(taps, 1):
            Tv -= 2 * np.longdouble(t) * full
            if d < n:
                Tv[d:] += np.longdouble(t) * full[:-d]
                Tv[:-d] += np.longdouble(t) * full[d:]
        values = ((full * Tv).sum(0) / (full * full).sum(0)).astype(float)
    out = tuple(np.ascontiguousarray(a) for a in (even, odd, values))
    for a in out:
        a.setflags(write=False)
    return out


def separable_modes(op, gd):
    """Per axis (even block, odd block, eigenvalues) of an FDOperator whose
    stencil is a symmetric sum of axis stencils (the centre coefficient is
    with axis 0), or None."""
    nn = op.mp
    taps = np.zeros((3, 2, nn))
    centre = 0.0
    for c, o in zip(op.coef_p, op.offset_pc):
        axes = np.flatnonzero(o)
        if len(axes) == 0:
            centre += c
        elif len(axes) == 1:
            d = o[axes[0]]
            taps[axes[0], int(d < 0), abs(d) - 1] += c
        else:
            return None
    if (taps[:, 0] != taps[:, 1]).any():
        return None
    out = []
    for a in range(3):
        n, per = int(gd.n_c[a]), bool(gd.pbc_c[a])
        if half_sizes(n, per)[0] > MAX_HALF:
            return None
        t = taps[a, 0]
        scale = t[np.abs(t).argmax()]
        if scale == 0.0:
            return None
        # the eigenvectors depend on the taps' ratios only: one entry serves
        # every spacing
        even, odd, lam = axis_modes(n, per, tuple(float(np.round(x, 14))
                                                  for x in t / scale))
        lam = scale * lam
        # what the axes' second differences leave of the centre coefficient
        # (zero for a Laplacian, up to rounding)
        centre += 2.0 * t.sum()
        out.append((even, odd, np.ascontiguousarray(lam)))
    if abs(centre) > 1e-12 * abs(op.coef_p[0]):
        out[0] = out[0][:2] + (out[0][2] + centre,)
    return out
