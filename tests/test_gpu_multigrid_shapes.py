"""Multigrid CG on grids at the edges of its levels and tiles: one level, two
levels, an axis that is never coarsened, tiles wider than the grid, odd and
periodic axes -- against the oracle's LU, phi within 1e-7 of max|phi| after a
solve to relative residual 1e-10 (the tolerances of the multigrid tests)."""
import numpy as np
import pytest

from test_gpu_parity import EPS0, make_ctx

pytestmark = pytest.mark.gpu


def _setup(t, nx, ny, periodic):
    for axis in periodic:
        t.apply_periodic(axis)
    blob = np.zeros((nx, ny), bool)
    blob[nx // 3:nx // 3 + 2, ny // 2:ny // 2 + 2] = True
    t.apply_dirichlet(blob, 12.0)
    if 2 not in periodic:
        side = np.zeros((nx, ny), bool)
        side[0, : (ny + 1) // 2] = True
        t.apply_dirichlet(side, -3.0)


@pytest.mark.parametrize("nx,ny,periodic", [(3, 3, ()), (20, 20, ()), (21, 20, ()), (40, 11, ()), (900, 2, (1,)),
                                            (3, 700, ()), (33, 65, (1,)), (66, 34, (1, 2)), (17, 51, (1, 2)),
                                            (129, 127, ()), (301, 97, (1,)), (96, 640, (2,))])
def test_shapes_match_the_oracle(orc, lib, nx, ny, periodic):
    dx = 1e-3
    rho = np.random.default_rng(nx * 31 + ny).normal(0, 1e-6, (nx, ny))
    ctx = make_ctx(nx, ny, dx, dx)
    ctx.poisson_create(EPS0)
    _setup(ctx, nx, ny, periodic)
    assert ctx.set_method(2) == 2
    ps = orc.PoissonOracle(nx, ny, dx, dx, EPS0)
    _setup(ps, nx, ny, periodic)
    for scale in (1.0, -0.4):  # the second solve starts from the first one's potential
        phi, it, rr = ctx.solve_host(-scale * rho, rtol=1e-10, maxit=500)
        assert rr <= 1e-10
        ref = ps.solve(-scale * rho)
        assert np.max(np.abs(phi - ref)) <= 1e-7 * np.max(np.abs(ref))
    ctx.close()
