"""The mixed solver's direct correction (fast diagonalisation) against dense
linear algebra and the oracle's operator.

Tolerance: the correction is six products with orthogonal matrices and one
division, so its backward error is a few n eps |L| |phi|; with
|L| |phi| / |rho| at most the condition number (below 1e4 on these grids)
the relative residual stays below 1e4 * 1e-14 = 1e-10, and the solution's
relative error below the same bound."""
import numpy as np
import pytest

from oracle import gpaw_layer as L
from tests.helpers import to_dev, to_np

pytestmark = pytest.mark.gpu
SCALE = -0.25 / np.pi


def _solver(N, pbc, nn=3, **kw):
    from gpaw_b200 import GridDescriptor, MixedPoissonSolver
    cell = tuple(0.35 * n * s for n, s in zip(N, (1.0, 1.1, 0.9)))
    gd = GridDescriptor(N, cell, pbc)
    ps = MixedPoissonSolver(nn=nn, tol=1e-10, **kw)
    ps.set_grid_descriptor(gd)
    return gd, ps, L.GridDescriptor(N, cell, pbc)


def _residual(gdo, nn, phi, rho):
    out = np.zeros_like(rho)
    L.Laplace(gdo, SCALE, nn).apply(np.ascontiguousarray(phi), out)
    return np.linalg.norm(rho - out) / np.linalg.norm(rho)


# sides at the edges of the 12-mode tiles, the 8-column stages and the
# 64-line blocks; every boundary; the widest axis the path takes and the
# first it does not
@pytest.mark.parametrize('N,pbc,nn', [
    ((4, 6, 8), 0, 1), ((4, 6, 8), 1, 3), ((24, 26, 50), 0, 3),
    ((22, 24, 46), 1, 2), ((24, 48, 18), (1, 0, 1), 3),
    ((18, 130, 34), (0, 1, 0), 3), ((96, 64, 34), 0, 3),
    ((8, 16, 384), 0, 3), ((8, 382, 16), 1, 3), ((8, 16, 386), 0, 3)])
def test_direct_solves_to_rounding(N, pbc, nn, cuda):
    gd, ps, gdo = _solver(N, pbc, nn, maxiter=400)
    rng = np.random.default_rng(1)
    rho = rng.standard_normal(tuple(gdo.n_c))
    rho -= rho.mean()
    phi = to_dev(rng.standard_normal(rho.shape))      # any initial guess
    n = ps.solve_neutral(phi, to_dev(rho))
    assert _residual(gdo, nn, to_np(phi), rho) <= 1.01e-10
    assert ps.rel_residual <= 1e-10
    if max(N) <= 384:
        assert n <= 2


@pytest.mark.parametrize('pbc', [0, 1])
def test_direct_against_dense_solution(pbc, cuda):
    N = (8, 10, 12)
    gd, ps, gdo = _solver(N, pbc)
    n = tuple(int(x) for x in gdo.n_c)
    op = L.Laplace(gdo, SCALE, 3)
    A = np.zeros((np.prod(n),) * 2)
    for i in range(len(A)):
        x, y = np.zeros(len(A)), np.zeros(n)
        x[i] = 1.0
        op.apply(x.reshape(n), y)
        A[:, i] = y.ravel()
    rho = np.random.default_rng(2).standard_normal(n)
    rho -= rho.mean()
    ref = np.linalg.lstsq(A, rho.ravel(), rcond=1e-12)[0].reshape(n)
    phi = gd.zeros()
    ps.solve_neutral(phi, to_dev(rho))
    assert np.linalg.norm(to_np(phi) - ref) <= 1e-10 * np.linalg.norm(ref)


def test_eager_correction_equals_the_solve(cuda):
    """The form for profilers, kernel by kernel."""
    import ctypes as C
    import torch
    gd, ps, gdo = _solver((24, 32, 100), 0)
    rho = to_dev(np.random.default_rng(7).standard_normal(tuple(gdo.n_c)))
    phi, got = gd.zeros(), gd.zeros()
    assert ps.solve_neutral(phi, rho) == 1
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert ps._h.lib.gb_mixed_direct_eager(
        ps._h.h, C.c_void_p(got.data_ptr()), C.c_void_p(rho.data_ptr()),
        st) == 0
    assert torch.equal(got, phi)


def test_the_caller_chooses_the_correction(cuda):
    """Direct under a low limit, V-cycles under a high one; a grid without a
    direct correction is refused."""
    N = (48, 40, 56)
    for correction, maxiter in (('direct', 2), ('vcycle', 200)):
        gd, ps, gdo = _solver(N, 0, maxiter=maxiter, correction=correction)
        rho = np.random.default_rng(3).standard_normal(tuple(gdo.n_c))
        phi = gd.zeros()
        n = ps.solve_neutral(phi, to_dev(rho))
        assert (n > 5) == (correction == 'vcycle')
        assert _residual(gdo, 3, to_np(phi), rho) <= 1.01e-10
    for N, nn in (((8, 16, 386), 3), ((16, 16, 16), 4)):
        with pytest.raises(ValueError, match='direct'):
            _solver(N, 0, nn, correction='direct')


def test_few_vcycles_allowed_keeps_the_vcycles(cuda):
    """maxiter below 50 is a limit on V-cycles: that path, same solution."""
    N = (48, 40, 56)
    rho = None
    out = []
    for maxiter in (49, 50):
        gd, ps, gdo = _solver(N, 0, maxiter=maxiter)
        if rho is None:
            rho = np.random.default_rng(3).standard_normal(tuple(gdo.n_c))
        phi = gd.zeros()
        n = ps.solve_neutral(phi, to_dev(rho))
        assert (n > 5) == (maxiter == 49)
        out.append(to_np(phi))
    assert np.abs(out[0] - out[1]).max() <= 1e-7 * np.abs(out[1]).max()


def test_direct_phi_may_be_rho(cuda):
    """phi and rho in one array: rho is read as it was at the call, alone
    and in a batch."""
    import torch
    from gpaw_b200.batch import PoissonBatch
    gd, ps, gdo = _solver((24, 32, 40), 0)
    rho = to_dev(np.random.default_rng(4).standard_normal(tuple(gdo.n_c)))
    a = rho.clone()
    ps.solve_neutral(a, rho)
    b = rho.clone()
    ps.solve_neutral(b, b)
    assert torch.equal(a, b)
    batch = PoissonBatch([gd, gd])
    c, d = rho.clone(), gd.zeros()
    batch.solve([c, d], [c, c])
    assert torch.equal(c, a)
    assert _residual(gdo, 3, to_np(d), to_np(rho)) <= 1.01e-10


def test_batch_and_solvers_freed_in_any_order(cuda):
    """A solver keeps its outcome when the batch is gone, and the batch may
    be the last to go."""
    import gc
    import torch
    from gpaw_b200 import GridDescriptor
    from gpaw_b200.batch import PoissonBatch
    gds = [GridDescriptor(N, 4.0, 0) for N in ((16, 24, 32), (24, 16, 16))]
    rng = np.random.default_rng(5)
    rhos = [to_dev(rng.standard_normal(tuple(gd.n_c))) for gd in gds]

    def solved():
        batch = PoissonBatch(gds)
        batch.enqueue([gd.zeros() for gd in gds], rhos)
        torch.cuda.synchronize()
        return batch

    batch = solved()
    want = batch.results()
    solvers = batch.solvers
    del batch
    gc.collect()
    assert [ps.result() for ps in solvers] == want
    assert all(0 < ps.rel_residual <= 1e-10 for ps in solvers)
    batch = solved()
    for ps in batch.solvers:
        ps._h = None                  # frees the solver
    gc.collect()
    del batch
    gc.collect()


@pytest.mark.parametrize('N,pbc', [((192, 16, 24), 0), ((16, 190, 24), 1),
                                   ((16, 24, 100), 0)])
def test_direct_is_deterministic_for_any_data(N, pbc, cuda):
    """Sums that overflow or are not finite: the same outcome every time (a
    half of an axis reads no row that another warp writes)."""
    gd, ps, gdo = _solver(N, pbc)
    rng = np.random.default_rng(6)
    for bad in (1e308, np.inf, np.nan):
        rho = rng.standard_normal(tuple(gdo.n_c))
        rho[tuple(n // 3 for n in rho.shape)] = bad
        seen = []
        for _ in range(4):
            phi = gd.zeros()
            try:
                ps.solve_neutral(phi, to_dev(rho))
            except RuntimeError:
                pass
            seen.append((ps.niter, to_np(phi)))
        for n, phi in seen[1:]:
            assert n == seen[0][0]
            assert np.array_equal(phi, seen[0][1], equal_nan=True)
