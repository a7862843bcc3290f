"""Multigrid CG on odd periodic axes, whose coarsening puts the odd node at the
seam: both forms of it (2m + 1 nodes, m odd and m even), repeated (2^k - 1 and
2^k + 1 nodes), next to tile edges, on either axis and both.  phi within 1e-7 of
max|phi| of the oracle's LU after a solve to relative residual 1e-10 (as the other
multigrid tests), in at most twice the iterations of the even axis one node longer."""
import numpy as np
import pytest

from test_gpu_multigrid_shapes import _setup
from test_gpu_parity import EPS0, make_ctx

pytestmark = pytest.mark.gpu


def _solve(nx, ny, periodic, rho):
    ctx = make_ctx(nx, ny, 1e-3, 1e-3)
    ctx.poisson_create(EPS0)
    _setup(ctx, nx, ny, periodic)
    assert ctx.set_method(2) == 2
    phi, it, rr = ctx.solve_host(-rho, rtol=1e-10, maxit=500)
    ctx.close()
    assert rr <= 1e-10
    return phi, it


@pytest.mark.parametrize("nx,ny,periodic", [(64, 63, (2,)), (64, 65, (2,)), (66, 33, (2,)), (257, 130, (1,)),
                                            (31, 255, (2,)), (129, 67, (1, 2)), (95, 190, (1,)), (100, 7, (2,)),
                                            (40, 161, (1, 2))])
def test_odd_periodic_axes(orc, lib, nx, ny, periodic):
    rho = np.random.default_rng(nx * 37 + ny).normal(0, 1e-6, (nx + 1, ny + 1))
    phi, it = _solve(nx, ny, periodic, rho[:nx, :ny].copy())
    ps = orc.PoissonOracle(nx, ny, 1e-3, 1e-3, EPS0)
    _setup(ps, nx, ny, periodic)
    ref = ps.solve(-rho[:nx, :ny])
    assert np.max(np.abs(phi - ref)) <= 1e-7 * np.max(np.abs(ref))
    ex, ey = nx + (1 in periodic and nx % 2), ny + (2 in periodic and ny % 2)
    assert it <= 2 * _solve(ex, ey, periodic, rho[:ex, :ey].copy())[1]
