"""The largest odd factor of ny that is solved directly (1024; any for singular
operators, whose CG has no multigrid): which solver a separable operator takes on
either side, and that both sides solve to 1e-9 -- phi within 1e-7 of max|phi| of the other
solver's."""
import numpy as np
import pytest

from test_gpu_parity import EPS0, _setup_bc, make_ctx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,ny,solver", [("slab", 1023, 0), ("slab", 2046, 0), ("slab", 3072, 0),
                                            ("slab", 1025, 2), ("slab", 2039, 2), ("slab", 3075, 2),
                                            ("slab", 4095, 2), ("periodic", 1025, 0)])
def test_solver_by_odd_factor(lib, kind, ny, solver):
    nx = 12
    rho = np.random.default_rng(ny).normal(0, 1e-6, (nx, ny))
    rho -= rho.mean()
    out = []
    for method in (0, 1 if kind == "periodic" else 2):
        ctx = make_ctx(nx, ny, 1e-3, 1e-3)
        ctx.poisson_create(EPS0)
        _setup_bc(ctx, kind, nx, ny)
        assert ctx.set_method(method) == (solver if method == 0 else method)
        phi, it, rr = ctx.solve_host(-rho, rtol=1e-9, maxit=20000)
        assert rr <= 1e-9
        out.append(phi)
        ctx.close()
    assert np.max(np.abs(out[0] - out[1])) <= 1e-7 * np.max(np.abs(out[1]))
