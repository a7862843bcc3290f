"""The field part of a step as one block (small grids) against the same stages
called one by one (density, solve, field), from the same particles: sizes at
the edges of its limits, ny = 2, other powers of two and odd ny, double-float
and FP64 states, driven, floating (circuit) and periodic operators.  rho of
the same positions is the same sums (1e-12 of its maximum); both potentials meet
the step's tolerance, 1e-9 (1e-10 in FP64), so they agree within 1e-7 of
max|phi|, and E within 1e-6 of max|E|."""
import numpy as np
import pytest

from test_gpu_parity import EPS0, ME, QE, _setup_bc, make_ctx, rand_particles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,nx,ny,rtol", [("slab", 257, 2, 1e-9), ("slab", 2048, 2, 1e-9), ("slab", 2049, 2, 1e-9),
                                             ("slab", 3, 2, 1e-9), ("slab", 48, 32, 1e-9), ("slab", 49, 32, 1e-9),
                                             ("slab", 33, 7, 1e-9), ("slab", 64, 24, 1e-9), ("slab", 257, 2, 1e-10),
                                             ("slab", 40, 16, 1e-10), ("periodic", 128, 2, 1e-9),
                                             ("periodic", 32, 32, 1e-10), ("periodic", 21, 9, 1e-9),
                                             ("neumann_gauss", 201, 2, 1e-9), ("driven", 129, 2, 1e-9),
                                             ("open_box", 10, 10, 1e-9), ("open_box", 20, 20, 1e-10),
                                             ("open_box", 21, 20, 1e-9), ("open_box", 34, 34, 1e-10),
                                             ("open_box", 300, 3, 1e-9)])
def test_step_field_matches_the_single_stages(lib, kind, nx, ny, rtol):
    dx, n = 1e-4, 4000
    rng = np.random.default_rng(nx + 7 * ny)
    per = kind == "periodic"

    def make():
        ctx = make_ctx(nx, ny, dx, dx, (int(per),) * 4)
        s = ctx.species_create(-QE, ME, 2e5, n)
        ctx.set_boundary(s, lib.BND_WRAP, lib.BND_WRAP)
        ctx.poisson_create(EPS0)
        if kind == "driven":
            _setup_bc(ctx, "slab", nx, ny)
            left = np.zeros((nx, ny), bool)
            left[0, :] = True
            ctx.drive_dirichlet(left, 30.0, 13.56e6, 0.4, 5.0)
        else:
            _setup_bc(ctx, kind, nx, ny)
        return ctx, s

    ctx, s = make()
    ctx.upload(s, *rand_particles(rng, n, nx, ny, dx, dx, 2e5))
    for k in range(3):
        ctx.step(1e-11, 1, seed=1, rtol=rtol)
        ctx.sync()
    it, rr = ctx.solve_info()
    assert rr <= rtol
    x, v, ids = ctx.download(s)
    rho, phi, E = ctx.field(lib.FIELD_RHO), ctx.field(lib.FIELD_PHI), ctx.field(lib.FIELD_E)
    sigma = ctx.get_sigma(1) if kind == "neumann_gauss" else None
    ctx.close()
    ref, s = make()
    ref.upload(s, x, v, ids=ids)
    if sigma is not None:
        ref.set_sigma(1, sigma)
    if kind == "driven":  # the third solve uses V(dt)
        left = np.zeros((nx, ny), bool)
        left[0, :] = True
        ref.apply_dirichlet(left, 30.0 * np.sin(2 * np.pi * 13.56e6 * 1e-11 + 0.4) + 5.0)
    rho_r = ref.charge_density()
    assert np.max(np.abs(rho - rho_r)) <= 1e-12 * np.max(np.abs(rho_r))
    ref.solve(rtol=rtol, maxit=200)
    phi_r, E_r = ref.field(lib.FIELD_PHI), ref.field(lib.FIELD_E)
    assert np.max(np.abs(phi - phi_r)) <= 1e-7 * np.max(np.abs(phi_r))
    assert np.max(np.abs(E - E_r)) <= 1e-6 * np.max(np.abs(E_r))
    ref.close()
