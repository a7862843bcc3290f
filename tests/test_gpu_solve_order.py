"""Repeated host solves on a small grid (right-hand sides below the 64 KB that
cudaMemcpy may hand back before the device has them): every solve takes its
own right-hand side -- the residual of the returned potential, evaluated on
the host, meets the tolerance (FP64 of the same operator: 1e-9 solved, at most
2e-9 measured)."""
import numpy as np
import pytest

from test_gpu_parity import EPS0, _setup_bc, make_ctx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", [0, 1, 2])
def test_each_host_solve_uses_its_own_right_hand_side(lib, method):
    nx, ny = 40, 32
    rho = np.random.default_rng(1).normal(0, 1e-6, (nx, ny))
    ctx = make_ctx(nx, ny, 1e-3, 1e-3)
    ctx.poisson_create(EPS0)
    _setup_bc(ctx, "slab", nx, ny)
    ctx.set_method(method)
    for k in range(200):
        f = -(0.3 + (k % 7)) * rho
        phi, _, _ = ctx.solve_host(f, rtol=1e-9, maxit=5000)
        assert ctx.poisson_residual(f, phi) <= 2e-9, k
    ctx.close()
