"""The calls that users of gpaw_b200 make, as cases that can be timed and
checked.

``listed()`` holds twelve calls over the range that real-space DFT work
meets, from one small grid to 256 wave functions; ``draw(rng)`` gives more of
the same ranges.  ``prepare`` builds what a program keeps between calls
(inputs, operators, solvers), ``run`` makes one call through the public
classes, ``exact`` restates the call in plain 64-bit torch.

Kinds of call:

apply        FDOperator.apply: the kinetic operator -1/2 Laplacian on bands
hamiltonian  FDHamiltonian.apply_local_potential: kin(psi) + v psi in one call
transfers    Transformer: restriction of bands and interpolation back
density      FDDensityTransfers: spin densities to the fine grid (rescaled off
             periodic cells) and a potential back
precond      Preconditioner: the multigrid preconditioner on band residuals
poisson      FDPoissonSolver.solve at its default tolerance
mixed        MixedPoissonSolver.solve at its default tolerance
batch        PoissonBatch.solve: many grids of uneven sizes at once
dielectric   WeightedFDPoissonSolver.solve: the solvation model's potential
"""
import math

import numpy as np
import torch

from gpaw_b200 import (FDHamiltonian, FDPoissonSolver, GridDescriptor,
                       Laplace, MixedPoissonSolver, Preconditioner,
                       Transformer)
from gpaw_b200.batch import PoissonBatch
from gpaw_b200.pot_calc import FDDensityTransfers
from gpaw_b200.solvation import WeightedFDPoissonSolver

BOHR = 0.5291772105638411
KPT = (0.25, 0.0, 0.1)


def listed():
    return [
        # one small real grid: the smallest call of a serving loop, where the
        # host path and the launch are all there is
        dict(name='apply_small_f64', kind='apply', cell='box', N='24x24x24',
             pbc='111', nn=3, bands=1, complex=False),
        # kinetic energy of all bands at a k-point (the headline workload)
        dict(name='apply_bands_c128', kind='apply', cell='box',
             N='96x96x96', pbc='111', nn=3, bands=256, complex=True),
        # H psi of a molecule: real bands, zero boundaries, odd extents
        dict(name='hamiltonian_f64', kind='hamiltonian', cell='box',
             N='112x120x96', pbc='000', nn=3, bands=32, complex=False),
        # kinetic energy in a hexagonal cell (surfaces, 2-D materials): the
        # stencil has an in-plane diagonal direction
        dict(name='apply_hex_c128', kind='apply', cell='hex',
             N='72x72x100', pbc='111', nn=3, bands=24, complex=True),
        # bands to the coarse grid and back, sextic order
        dict(name='transfers_c128', kind='transfers', N='96x96x96',
             pbc='111', nn=3, bands=64, complex=True),
        # a molecule's spin densities to the fine grid, a potential back
        dict(name='density_f64', kind='density', N='80x96x88',
             pbc='000', nn=3, spins=2),
        # residuals of a block of real bands (the 112^3 configuration)
        dict(name='precond_f64', kind='precond', N='112x112x112',
             pbc='000', bands=128, complex=False),
        # residuals of a smaller block of Bloch bands, uneven sides
        dict(name='precond_c128', kind='precond', N='80x96x72',
             pbc='111', bands=16, complex=True),
        # the Hartree potential of a small molecule (64^3, 0.2 Angstrom)
        dict(name='poisson_64', kind='poisson', N='64x64x64',
             pbc='000', gaussians=8),
        # the Hartree potential on a large fine grid, 1e-10
        dict(name='mixed_192', kind='mixed', N='192x192x192',
             pbc='000', gaussians=64, levels=4),
        # a batch of solves on uneven grids, one call
        dict(name='batch_48', kind='batch', count=48, seed=0, low=32,
             high=128, pbc='000'),
        # a solute in a dielectric continuum on the 64^3 grid
        dict(name='dielectric_64', kind='dielectric', N='64x64x64',
             pbc='000', gaussians=8),
    ]


def _log_int(rng, lo, hi, multiple=1):
    x = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return int(min(hi, max(lo, multiple * round(x / multiple))))


def _sides(rng, lo, hi, multiple):
    return [_log_int(rng, lo, hi, multiple) for _ in range(3)]


def _bands(rng, N, es, most, cap_bytes):
    one = N[0] * N[1] * N[2] * es
    return max(1, min(_log_int(rng, 1, most), cap_bytes // one))


def _text(N):
    return 'x'.join(str(n) for n in N)


def _read(case):
    """The case with its sizes and boundary flags as lists of numbers."""
    case = dict(case, pbc=[int(p) for p in case['pbc']])
    if 'N' in case:
        case['N'] = [int(n) for n in case['N'].split('x')]
    return case


def draw(rng):
    kind = rng.choice(['apply', 'apply', 'hamiltonian', 'apply_skew',
                       'transfers', 'density', 'precond', 'poisson', 'mixed',
                       'batch', 'dielectric'])
    pbc = rng.choice(['111', '000', '110', '000', '111'])
    cx = rng.random() < 0.5
    es = 16 if cx else 8
    if kind in ('apply', 'hamiltonian'):
        N = _sides(rng, 16, 160, 1 if rng.random() < 0.5 else 4)
        return dict(kind=kind, cell='box', N=_text(N), pbc=pbc,
                    nn=rng.choice([1, 2, 3, 3, 3, 4, 5, 6]), complex=cx,
                    bands=_bands(rng, N, es, 256, 2 << 30))
    if kind == 'apply_skew':
        cell = rng.choice(['hex', 'fcc'])
        n = _log_int(rng, 18, 96)
        N = [n, n, _log_int(rng, 20, 128) if cell == 'hex' else n]
        return dict(kind='apply', cell=cell, N=_text(N), pbc='111',
                    nn=rng.choice([1, 2, 3, 3, 4]), complex=cx,
                    bands=_bands(rng, N, es, 32, 1 << 28))
    if kind == 'transfers':
        N = _sides(rng, 24, 160, 2)
        return dict(kind=kind, N=_text(N), pbc=pbc, nn=rng.choice([1, 2, 3, 4]),
                    complex=cx, bands=_bands(rng, N, es, 128, 1 << 30))
    if kind == 'density':
        return dict(kind=kind, N=_text(_sides(rng, 16, 128, 2)), pbc=pbc,
                    nn=rng.choice([1, 2, 3, 4]), spins=rng.choice([1, 2]))
    if kind == 'precond':
        N = _sides(rng, 24, 144, 4)
        return dict(kind=kind, N=_text(N), pbc=pbc, complex=cx,
                    bands=_bands(rng, N, es, 128, 1 << 30))
    if kind == 'poisson':
        return dict(kind=kind, N=_text(_sides(rng, 24, 128, 8)), pbc=pbc,
                    gaussians=rng.randint(4, 16))
    if kind == 'mixed':
        return dict(kind=kind, N=_text(_sides(rng, 32, 192, 16)), pbc=pbc,
                    gaussians=rng.randint(4, 64), levels=rng.choice([4, 6]))
    if kind == 'batch':
        return dict(kind=kind, count=rng.randint(8, 40),
                    seed=rng.randint(1, 1 << 20), low=32, high=128,
                    pbc=rng.choice(['000', '111']))
    return dict(kind='dielectric', N=_text(_sides(rng, 32, 96, 8)), pbc='000',
                gaussians=rng.randint(4, 12))


# ------------------------------------------------------------------ inputs
def _cell(case):
    """Cell vectors (Bohr) at a spacing of 0.2 Angstrom along each axis."""
    h = 0.2 / BOHR
    N = case['N']
    if case.get('cell') == 'hex':
        a, c = h * N[0], h * N[2]
        return [[a, 0, 0], [-a / 2, a * math.sqrt(3) / 2, 0], [0, 0, c]]
    if case.get('cell') == 'fcc':
        a = h * N[0] / math.sqrt(2)
        return [[0, a, a], [a, 0, a], [a, a, 0]]
    return [h * n for n in N]


def _grid(case, device):
    return GridDescriptor(tuple(case['N']), _cell(case),
                          tuple(bool(p) for p in case['pbc']), device=device)


def _phases(case, gd):
    if not case['complex']:
        return None
    return gd.phase_factor_cd(tuple(k if p else 0.0 for k, p in
                                    zip(KPT, case['pbc'])))


def _generator(device, seed):
    g = torch.Generator(device=device)
    g.manual_seed(int(seed))
    return g


def _normal(shape, cx, device, seed):
    g = _generator(device, seed)
    return torch.randn(shape, generator=g, device=device,
                       dtype=torch.complex128 if cx else torch.float64)


def _points(N, pbc):
    return [n if p else n - 1 for n, p in zip(N, pbc)]


def _coords(N, pbc, device):
    """Point coordinates along each axis (Bohr), shaped for broadcasting."""
    h = 0.2 / BOHR
    out = []
    for c in range(3):
        x = h * (torch.arange(N[c], device=device, dtype=torch.float64)
                 if pbc[c] else
                 torch.arange(1, N[c], device=device, dtype=torch.float64))
        out.append(x.view([-1 if d == c else 1 for d in range(3)]))
    return out


def _density(N, pbc, count, device, seed):
    """A neutral sum of Gaussians: widths 0.5-1.2 Angstrom, charges 0.5-2 of
    either sign, centres in the middle 0.2-0.8 of the box."""
    rng = np.random.default_rng(int(seed))
    h = 0.2 / BOHR
    L = h * np.array(N)
    x, y, z = _coords(N, pbc, device)
    rho = torch.zeros(_points(N, pbc), dtype=torch.float64, device=device)
    for _ in range(count):
        c = rng.uniform(0.2, 0.8, 3) * L
        w = rng.uniform(0.5, 1.2) / BOHR
        q = rng.uniform(0.5, 2.0) * rng.choice([-1.0, 1.0])
        gx, gy, gz = (torch.exp(-(t - ct)**2 / w**2)
                      for t, ct in zip((x, y, z), c))
        rho += (q * (math.pi * w * w)**-1.5 * gx) * gy * gz
    return rho - rho.mean()


class Dielectric:
    """eps(r) and its gradient for a spherical cavity with a smooth wall:
    1 inside, 80 outside."""

    def __init__(self, N, pbc, device):
        L = 0.2 / BOHR * np.array(N)
        x, y, z = _coords(N, pbc, device)
        dx, dy, dz = (t - l / 2 for t, l in zip((x, y, z), L))
        r = torch.sqrt(dx * dx + dy * dy + dz * dz).clamp_min(1e-12)
        r0, w = 0.28 * L.min(), 1.0
        t = torch.tanh((r - r0) / w)
        slope = 79.0 * 0.5 * (1.0 - t * t) / (w * r)
        self.eps_gradeps = [(1.0 + 79.0 * 0.5 * (1.0 + t)).contiguous()] + \
            [(slope * d).contiguous() for d in (dx, dy, dz)]


def _batch_sides(case):
    rng = np.random.default_rng(case['seed'])
    sides = np.arange(case['low'], case['high'] + 1, 8)
    return [[int(x) for x in rng.choice(sides, 3)]
            for _ in range(case['count'])]


def _batch_density(case, i, N, device, seed):
    return _density(N, case['pbc'], 4 + (7 * i) % 13, device,
                    1000 * int(seed) + i)


def _inputs(case, seed, device):
    """The arrays of the call, from the seed alone."""
    kind = case['kind']
    if kind == 'batch':
        return [_batch_density(case, i, N, device, seed)
                for i, N in enumerate(_batch_sides(case))]
    N, pbc = case['N'], case['pbc']
    n = _points(N, pbc)
    if kind in ('apply', 'hamiltonian', 'transfers', 'precond'):
        x = _normal([case['bands']] + n, case['complex'], device, seed)
        if kind != 'hamiltonian':
            return x
        return x, _normal(n, False, device, seed + 1)
    if kind == 'density':
        g = _generator(device, seed)
        nt = torch.rand([case['spins']] + n, generator=g, device=device,
                        dtype=torch.float64) + 0.01
        fine = _points([2 * k for k in N], pbc)
        return nt, _normal([case['spins']] + fine, False, device, seed + 1)
    return _density(N, pbc, case['gaussians'], device, seed)


# --------------------------------------------------------------- the calls
def prepare(case, seed):
    case = _read(case)
    device = torch.device('cuda', torch.cuda.current_device())
    kind = case['kind']
    s = dict(kind=kind)
    if kind == 'batch':
        gds = [GridDescriptor(tuple(N), _cell(dict(N=N)),
                              tuple(bool(p) for p in case['pbc']),
                              device=device) for N in _batch_sides(case)]
        s.update(gds=gds, rhos=_inputs(case, seed, device),
                 solver=PoissonBatch(gds))
        return s
    gd = s['gd'] = _grid(case, device)
    if kind == 'apply':
        x = _inputs(case, seed, device)
        s.update(x=x, out=torch.empty_like(x), phases=_phases(case, gd),
                 op=Laplace(gd, -0.5, case['nn'],
                            complex if case['complex'] else float))
    elif kind == 'hamiltonian':
        x, v = _inputs(case, seed, device)
        s.update(x=x, v=v, out=torch.empty_like(x), phases=_phases(case, gd),
                 op=FDHamiltonian(gd, kin_stencil=case['nn'],
                                  dtype=complex if case['complex'] else float))
    elif kind == 'transfers':
        x = _inputs(case, seed, device)
        dtype = complex if case['complex'] else float
        gd2 = gd.coarsen()
        s.update(x=x, phases=_phases(case, gd),
                 down=Transformer(gd, gd2, case['nn'], dtype),
                 up=Transformer(gd2, gd, case['nn'], dtype),
                 coarse=gd2.empty(case['bands'], dtype),
                 fine=torch.empty_like(x))
    elif kind == 'density':
        nt, v = _inputs(case, seed, device)
        s.update(nt=nt, v=v,
                 op=FDDensityTransfers(gd, gd.refine(), case['nn']))
    elif kind == 'precond':
        x = _inputs(case, seed, device)
        dtype = complex if case['complex'] else float
        s.update(x=x, out=torch.empty_like(x), phases=_phases(case, gd),
                 op=Preconditioner(gd, Laplace(gd, -0.5, 3, dtype), dtype,
                                   block=case['bands']))
    else:
        if kind == 'poisson':
            solver = FDPoissonSolver()
        elif kind == 'mixed':
            solver = MixedPoissonSolver(levels=case['levels'])
        else:
            solver = WeightedFDPoissonSolver()
            solver.set_dielectric(Dielectric(case['N'], case['pbc'], device))
        solver.set_grid_descriptor(gd)
        s.update(rho=_inputs(case, seed, device), solver=solver)
    return s


def run(s):
    kind = s['kind']
    if kind == 'apply':
        s['op'].apply(s['x'], s['out'], s['phases'])
        return s['out']
    if kind == 'hamiltonian':
        s['op'].apply_local_potential(s['v'], s['x'], s['out'], s['phases'])
        return s['out']
    if kind == 'transfers':
        s['down'].apply(s['x'], s['coarse'], s['phases'])
        s['up'].apply(s['coarse'], s['fine'], s['phases'])
        return [s['coarse'], s['fine']]
    if kind == 'density':
        return [s['op'].interpolate_density(s['nt']),
                s['op'].restrict(s['v'])]
    if kind == 'precond':
        return s['op'](s['x'], s['phases'], out=s['out'])
    if kind == 'batch':
        phis = [gd.zeros() for gd in s['gds']]
        s['solver'].solve(phis, s['rhos'])
        return phis
    phi = s['gd'].zeros()
    s['solver'].solve(phi, s['rho'])
    return phi


def work(case):
    """Bytes: every input read once, every output written once.  Operations:
    of the stencils as they are defined (a product and a sum a coefficient);
    for the solvers of the V-cycles that their schedules take (about 10, 14
    and 11) at some 6 passes of the fine grid, and the coarse grids 1/7."""
    case = _read(case)
    kind = case['kind']
    if kind == 'batch':
        pts = sum(np.prod(_points(N, case['pbc'])) for N in
                  _batch_sides(case))
        return dict(bytes=24.0 * pts, flops=14 * 6 * 38 * 8 / 7 * float(pts))
    pts = float(np.prod(_points(case['N'], case['pbc'])))
    if kind in ('poisson', 'mixed', 'dielectric'):
        cycles, per = {'poisson': (10, 38), 'mixed': (14, 38),
                       'dielectric': (11, 80)}[kind]
        arrays = 7 if kind == 'dielectric' else 3
        return dict(bytes=8.0 * arrays * pts,
                    flops=cycles * 6 * per * 8 / 7 * pts)
    if kind == 'density':
        fine = float(np.prod(_points([2 * n for n in case['N']],
                                     case['pbc'])))
        return dict(bytes=8.0 * case['spins'] * 2 * (pts + fine),
                    flops=case['spins'] * fine * 4 * 4 * case['nn'])
    es = 16 if case['complex'] else 8
    pts *= case['bands']
    re = 2 if case['complex'] else 1
    if kind == 'transfers':
        return dict(bytes=es * pts * (1 + 1 / 8) * 2,
                    flops=re * pts * 2 * 4 * case['nn'])
    if kind == 'precond':
        return dict(bytes=es * pts * 2, flops=re * pts * (38 + 12 + 12))
    dirs = {'box': 3, 'hex': 4, 'fcc': 6}[case['cell']]
    flops = re * pts * 2 * (1 + 2 * dirs * case['nn'])
    nbytes = es * pts * 2
    if kind == 'hamiltonian':
        nbytes += 8 * pts / case['bands']
        flops += re * pts * 2
    return dict(bytes=nbytes, flops=flops)


def tolerance(case):
    """Linear maps of 64-bit data: sums in another order, measured against
    `exact`, differ by 1e-16 to 7e-16; the FP64 solvers' V-cycles carry that
    to 1e-14 .. 1e-13.  The mixed solvers stop at a relative residual of 1e-10
    and differ from the exact solution by some 1e-11 of its norm."""
    kind = case['kind']
    if kind in ('mixed', 'batch'):
        return dict(rel=1e-10)
    if kind in ('poisson', 'dielectric'):
        return dict(rel=1e-12)
    return dict(rel=3e-15)


# ------------------------------------------- the same in plain 64-bit torch
_SECOND = {1: [-2, 1], 2: [-5 / 2, 4 / 3, -1 / 12],
           3: [-49 / 18, 3 / 2, -3 / 20, 1 / 90],
           4: [-205 / 72, 8 / 5, -1 / 5, 8 / 315, -1 / 560],
           5: [-5269 / 1800, 5 / 3, -5 / 21, 5 / 126, -5 / 1008, 1 / 3150],
           6: [-5369 / 1800, 12 / 7, -15 / 56, 10 / 189, -1 / 112, 2 / 1925,
               -1 / 16632]}
_FIRST = {1: [1 / 2], 3: [3 / 4, -3 / 20, 1 / 60]}


def _line(n, periodic, entries, phase, dtype, device):
    """n x n matrix of sum over (offset, coefficient) along one axis."""
    A = np.zeros((n, n), complex)
    for i in range(n):
        for o, c in entries:
            j, f = i + o, 1.0
            if not 0 <= j < n:
                if not periodic:
                    continue
                f = phase if j >= n else np.conj(phase)
                j %= n
            A[i, j] += c * f
    if not dtype.is_complex:
        A = A.real
    return torch.from_numpy(np.ascontiguousarray(A)).to(device, dtype)


def _along(M, x, axis):
    """Matrix M along axis 0, 1 or 2 of the last three of x."""
    d = x.dim() - 3 + axis
    return torch.movedim(torch.tensordot(x, M, dims=([d], [1])), -1, d)


def _phase_of(case, c):
    k = KPT[c] if case.get('complex') and case['pbc'][c] else 0.0
    return np.exp(2j * np.pi * k)


def _laplacian(case, N, nn, scale, dtype, device):
    """A function of x: scale times the box Laplacian; its diagonal; the
    three axis matrices."""
    h = 0.2 / BOHR * case['N'][0] / N[0]
    c = _SECOND[nn]
    entries = [(0, c[0])] + [(s * d, c[d]) for d in range(1, nn + 1)
                             for s in (1, -1)]
    n = _points(N, case['pbc'])
    M = [_line(n[a], case['pbc'][a], [(o, scale * v / h**2)
                                      for o, v in entries],
               _phase_of(case, a), dtype, device) for a in range(3)]

    def f(x):
        return _along(M[0], x, 0) + _along(M[1], x, 1) + _along(M[2], x, 2)
    return f, 3 * scale * c[0] / h**2, M


def _gradient(case, N, nn, scale, v, device):
    h = 0.2 / BOHR * case['N'][0] / N[0]
    entries = [(s * d, s * scale / h * _FIRST[nn][d - 1])
               for d in range(1, nn + 1) for s in (1, -1)]
    n = _points(N, case['pbc'])
    M = _line(n[v], case['pbc'][v], entries, 1.0, torch.float64, device)
    return lambda x: _along(M, x, v)


def _mid_weights(nn):
    """Lagrange weights at the mid-point of 2 nn equidistant points, for the
    pairs at distance 1/2, 3/2, ..."""
    xs = [m + 0.5 for m in range(-nn, nn)]
    return [math.prod(-xm / (x - xm) for xm in xs if xm != x)
            for x in xs[nn:]]


def _restrict(case, N, nn, dtype, device):
    """Restriction from N to N / 2 points."""
    w = _mid_weights(nn)
    entries = [(0, 0.5)] + [(s * (2 * m + 1), 0.5 * w[m])
                            for m in range(nn) for s in (1, -1)]
    n = _points(N, case['pbc'])
    M = []
    for a in range(3):
        A = _line(n[a], case['pbc'][a], entries, _phase_of(case, a), dtype,
                  device)
        M.append(A[(0 if case['pbc'][a] else 1)::2])

    def f(x):
        for a in (2, 1, 0):
            x = _along(M[a], x, a)
        return x
    return f


def _interpolate(case, N, nn, dtype, device):
    """Interpolation from N / 2 to N points."""
    w = _mid_weights(nn)
    M = []
    for a in range(3):
        p = case['pbc'][a]
        nc = N[a] // 2 if p else N[a] // 2 - 1
        nf = N[a] if p else N[a] - 1
        A = np.zeros((nf, nc), complex)
        ph = _phase_of(case, a)
        for i in range(nf):
            f = i if p else i + 1             # fine point number
            if f % 2 == 0:
                terms = [(f // 2, 1.0)]
            else:
                terms = [(f // 2 - m, w[m]) for m in range(nn)] + \
                    [(f // 2 + 1 + m, w[m]) for m in range(nn)]
            for j, c in terms:
                j = j if p else j - 1
                g = 1.0
                if not 0 <= j < nc:
                    if not p:
                        continue
                    g = ph if j >= nc else np.conj(ph)
                    j %= nc
                A[i, j] += c * g
        if not dtype.is_complex:
            A = A.real
        M.append(torch.from_numpy(np.ascontiguousarray(A)).to(device, dtype))

    def f(x):
        for a in (2, 1, 0):
            x = _along(M[a], x, a)
        return x
    return f


def _skew(case, x):
    """-1/2 Laplacian of a periodic hexagonal or fcc cell: second differences
    along the lattice's shortest directions."""
    h, nn = 0.2 / BOHR, case['nn']
    if case['cell'] == 'hex':
        dirs = [((1, 0, 0), 2 / 3), ((0, 1, 0), 2 / 3), ((1, 1, 0), 2 / 3),
                ((0, 0, 1), 1.0)]
    else:
        dirs = [(d, 0.5) for d in ((1, 0, 0), (0, 1, 0), (0, 0, 1),
                                   (1, -1, 0), (1, 0, -1), (0, 1, -1))]
    p = x
    for c in range(3):
        d = x.dim() - 3 + c
        n = x.shape[d]
        ph = complex(_phase_of(case, c))
        lo, hi = p.narrow(d, n - nn, nn), p.narrow(d, 0, nn)
        if x.is_complex():
            lo, hi = lo * ph.conjugate(), hi * ph
        p = torch.cat([lo, p, hi], d)
    n = x.shape[-3:]
    out = torch.zeros_like(x)
    for d, a in dirs:
        a *= -0.5 / h**2
        out += a * _SECOND[nn][0] * x
        for k in range(1, nn + 1):
            for s in (k, -k):
                b = [nn + s * v for v in d]
                out += a * _SECOND[nn][k] * p[..., b[0]:b[0] + n[0],
                                              b[1]:b[1] + n[1],
                                              b[2]:b[2] + n[2]]
    return out


def _chunks(f, x, most=1 << 27):
    """f over the bands of x, a few at a time."""
    k = max(1, most // x[0].numel() // x.element_size())
    return torch.cat([f(x[i:i + k]) for i in range(0, len(x), k)])


def _levels(case):
    grids = [list(case['N'])]
    while len(grids) < 9 and all(n % 2 == 0 for n in grids[-1]):
        N = [n // 2 for n in grids[-1]]
        if any(m < 1 for m in _points(N, case['pbc'])):
            break
        grids.append(N)
    return grids


def _multigrid(case, rho, weights=None):
    """The V-cycles of the FP64 solvers until sum(r^2) dv <= 2e-10: weighted
    Jacobi 2/1 sweeps (weight 2/3) on the finest grid, 4/4 below (weight 1),
    8 + 8 on the coarsest (where only the second 8 run)."""
    dev, dt = rho.device, torch.float64
    grids = _levels(case)
    last = len(grids) - 1
    ops, down, up = [], [], []
    w = weights
    scale = -0.25 / math.pi
    for l, N in enumerate(grids):
        lap, diag, _ = _laplacian(case, N, 3 if l == 0 else 1, scale, dt, dev)
        if w is None:
            ops.append((lap, diag))
        else:
            grads = [_gradient(case, N, 3 if l == 0 else 1, scale, v, dev)
                     for v in range(3)]
            ops.append((lambda x, w=w, lap=lap, grads=grads:
                        w[0] * lap(x) + w[1] * grads[0](x) +
                        w[2] * grads[1](x) + w[3] * grads[2](x),
                        diag * w[0]))
        if l < last:
            down.append(_restrict(case, N, 1, dt, dev))
            up.append(_interpolate(case, N, 1, dt, dev))
            if w is not None:
                w = [down[-1](t) for t in w]

    def relax(l, phi, r, sweeps):
        A, diag = ops[l]
        om = 2 / 3 if l == 0 else 1.0
        for _ in range(sweeps):
            phi = phi + om * (r - A(phi)) / diag
        return phi

    def cycle(l, phi, r):
        if l < last:
            phi = relax(l, phi, r, 2 if l == 0 else 4)
            rc = down[l](ops[l][0](phi) - r)
            phi = phi - up[l](cycle(l + 1, torch.zeros_like(rc), rc))
        return relax(l, phi, r, 8 if l == last else 1 if l == 0 else 4)

    dv = (0.2 / BOHR)**3
    phi = torch.zeros_like(rho)
    for _ in range(1000):
        phi = cycle(0, phi, rho)
        if float(((ops[0][0](phi) - rho)**2).sum()) * dv <= 2e-10:
            break
    return phi - phi.mean() if all(case['pbc']) else phi


def _direct(case, rho):
    """The exact solution, in the eigenvectors of each axis's matrix."""
    _, _, M = _laplacian(case, case['N'], 3, -0.25 / math.pi, torch.float64,
                         rho.device)
    e, V = zip(*(torch.linalg.eigh(m) for m in M))
    x = rho
    for a in range(3):
        x = _along(V[a].T.contiguous(), x, a)
    lam = e[0][:, None, None] + e[1][None, :, None] + e[2][None, None, :]
    if all(case['pbc']):                       # the constant is free: zero
        k = int(lam.abs().argmin())
        x.view(-1)[k] = 0.0
        lam.view(-1)[k] = 1.0
    x = x / lam
    for a in range(3):
        x = _along(V[a].contiguous(), x, a)
    return x - x.mean() if all(case['pbc']) else x


def _precondition(case, R):
    dt, dev, N0 = R.dtype, R.device, case['N']
    N1, N2 = [n // 2 for n in N0], [n // 4 for n in N0]
    K0, diag, _ = _laplacian(case, N0, 3, -0.5, dt, dev)
    K1 = _laplacian(case, N1, 1, -0.5, dt, dev)[0]
    K2 = _laplacian(case, N2, 1, -0.5, dt, dev)[0]
    down0, down1 = (_restrict(case, N, 1, dt, dev) for N in (N0, N1))
    up1, up2 = (_interpolate(case, N, 1, dt, dev) for N in (N0, N1))
    s = 0.66666666 / diag

    def f(r):
        r1 = down0(-r)
        d1 = 4 * s * r1
        r2 = down1(K1(d1) - r1)
        d2 = 16 * s * r2
        d1 = d1 - up2(d2 - 16 * s * (K2(d2) - r2))
        d1 = d1 - 4 * s * (K1(d1) - r1)
        q = -up1(d1)
        return -(q - s * (K0(q) - r))
    return _chunks(f, R)


def exact(case, seed):
    case = _read(case)
    device = torch.device('cuda', torch.cuda.current_device())
    kind = case['kind']
    got = _inputs(case, seed, device)
    if kind == 'batch':
        return [_direct(dict(N=N, pbc=case['pbc']), r)
                for N, r in zip(_batch_sides(case), got)]
    if kind in ('apply', 'hamiltonian'):
        x, v = got if kind == 'hamiltonian' else (got, None)
        if case['cell'] != 'box':
            return _chunks(lambda t: _skew(case, t), x)
        lap, _, _ = _laplacian(case, case['N'], case['nn'], -0.5, x.dtype,
                               device)
        return _chunks(lap if v is None else lambda t: lap(t) + t * v, x)
    if kind == 'transfers':
        x = got
        down = _restrict(case, case['N'], case['nn'], x.dtype, device)
        up = _interpolate(case, case['N'], case['nn'], x.dtype, device)
        coarse = _chunks(down, x)
        return [coarse, _chunks(up, coarse)]
    if kind == 'density':
        nt, v = got
        N = [2 * n for n in case['N']]
        f = _interpolate(case, N, case['nn'], nt.dtype, device)(nt)
        if not all(case['pbc']):
            f = f * (8 * nt.sum((1, 2, 3)) / f.sum((1, 2, 3))).view(-1, 1, 1,
                                                                    1)
        return [f, _restrict(case, N, case['nn'], v.dtype, device)(v)]
    if kind == 'precond':
        return _precondition(case, got)
    if kind == 'mixed':
        return _direct(case, got)
    if kind == 'poisson':
        return _multigrid(case, got)
    return _multigrid(case, got,
                      Dielectric(case['N'], case['pbc'], device).eps_gradeps)
