"""The coarse levels of the FP64 V-cycles in one cluster launch against the
per-level kernels, bit for bit (the same operations in the same order): plain
and dielectric operator, levels on either side of the 1024 points that one
CTA takes alone and up to the 32768 of the first fused level, every
boundary."""
import numpy as np
import pytest

from tests.helpers import to_np

pytestmark = pytest.mark.gpu
GRIDS = [((64, 64, 64), 0), ((64, 64, 64), 1), ((32, 48, 80), (1, 0, 1)),
         ((16, 24, 8), 0), ((8, 8, 12), 1), ((40, 80, 48), (0, 1, 0)),
         ((12, 20, 28), 0)]


def _rho(gd, seed):
    import torch
    g = torch.Generator(device='cuda')
    g.manual_seed(seed)
    rho = torch.randn(tuple(gd.n_c), generator=g, dtype=torch.float64,
                      device='cuda')
    return rho - rho.mean()


@pytest.mark.parametrize('N,pbc', GRIDS)
def test_plain_levels(N, pbc, cuda, monkeypatch):
    from gpaw_b200 import FDPoissonSolver, GridDescriptor
    gd = GridDescriptor(N, tuple(0.37 * n for n in N), pbc)
    rho = _rho(gd, 1)
    got = []
    for tail in '10':
        monkeypatch.setenv('GPAW_B200_POISSON_TAIL', tail)
        ps = FDPoissonSolver()
        ps.set_grid_descriptor(gd)
        phi = gd.zeros()
        errs = [ps.iterate2(0.0, phi=phi, rho=rho) for _ in range(4)]
        assert (ps._exec.lib.gb_poisson_fused_levels(ps._exec.h) > 0) == \
            (tail == '1')
        got.append((to_np(phi), errs))
    assert np.array_equal(got[0][0], got[1][0]) and got[0][1] == got[1][1]


class _Dielectric:
    def __init__(self, gd):
        import torch
        i = [torch.arange(int(n), dtype=torch.float64, device='cuda').view(
            [-1 if c == d else 1 for d in range(3)])
            for c, n in enumerate(gd.n_c)]
        w = torch.cos(0.3 * i[0]) * torch.sin(0.2 * i[1] + 0.1 * i[2])
        self.eps_gradeps = [2.0 + w] + [0.2 * torch.roll(w, k, k).contiguous()
                                        for k in range(3)]


@pytest.mark.parametrize('N,pbc', GRIDS)
def test_dielectric_levels(N, pbc, cuda, monkeypatch):
    from gpaw_b200 import GridDescriptor, PoissonConvergenceError
    from gpaw_b200.solvation import WeightedFDPoissonSolver
    gd = GridDescriptor(N, tuple(0.37 * n for n in N), pbc)
    rho = _rho(gd, 2)
    got = []
    for graph in '10':
        monkeypatch.setenv('GPAW_B200_WGRAPH', graph)
        # six V-cycles (these weights are no gradient of a dielectric, so
        # convergence is not the point)
        ps = WeightedFDPoissonSolver(eps=0.0, maxiter=6)
        ps.set_dielectric(_Dielectric(gd))
        ps.set_grid_descriptor(gd)
        phi = gd.zeros()
        with pytest.raises(PoissonConvergenceError):
            ps.solve(phi, rho, charge=0.0)
        if graph == '1':
            assert ps._coarse is not None
        got.append(to_np(phi))
    assert np.isfinite(got[0]).all() and got[0].any()
    assert np.array_equal(got[0], got[1])
