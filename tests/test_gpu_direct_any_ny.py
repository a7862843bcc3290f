"""Direct solves of separable operators whose ny is not a power of two (dense
DFTs of the odd factor): primes, small and large odd factors, x-periodic,
singular and floating-electrode operators, against the oracle's LU -- phi
within 1e-7 of max|phi| after a solve to relative residual 1e-9 -- and the
cases that keep CG."""
import numpy as np
import pytest

from test_gpu_parity import EPS0, ME, QE, _setup_bc, make_ctx, rand_particles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,nx,ny", [("slab", 33, 3), ("slab", 64, 6), ("slab", 130, 97), ("slab", 41, 100),
                                        ("slab", 31, 255), ("slab", 9, 1023), ("slab", 700, 15), ("slab", 1300, 12),
                                        ("periodic", 30, 12), ("periodic", 21, 9), ("neumann", 33, 7),
                                        ("neumann_gauss", 64, 24)])
def test_direct_solve_matches_oracle(orc, lib, kind, nx, ny):
    dx = 1e-3
    rho = np.random.default_rng(nx + ny).normal(0, 1e-6, (nx, ny))
    if kind == "periodic":
        rho -= rho.mean()
    ctx = make_ctx(nx, ny, dx, dx)
    ctx.poisson_create(EPS0)
    _setup_bc(ctx, kind, nx, ny)
    assert ctx.set_method(0) == 0
    phi, it, rr = ctx.solve_host(-rho, rtol=1e-9, maxit=100)
    assert rr <= 1e-9 and it <= 6, (it, rr)
    ps = orc.PoissonOracle(nx, ny, dx, dx, EPS0)
    _setup_bc(ps, kind, nx, ny)
    ref = ps.solve(-rho)
    if kind == "periodic":
        ref = ref - ref.mean()
    assert np.max(np.abs(phi - ref)) <= 1e-7 * np.max(np.abs(ref))
    ctx.close()


@pytest.mark.parametrize("nx,ny", [(65, 24), (50, 33)])
def test_steps_agree_with_multigrid_cg(lib, nx, ny):
    """Whole steps (captured) through the direct solve and through forced
    multigrid CG: both meet 1e-9, so phi agrees within 1e-7 of max|phi|."""
    out = []
    for method in (0, 2):
        rng = np.random.default_rng(4)
        ctx = make_ctx(nx, ny, 1e-4, 1e-4)
        se = ctx.species_create(-QE, ME, 2e4, 30000)
        ctx.set_boundary(se, lib.BND_DISCARD, lib.BND_WRAP)
        ctx.upload(se, *rand_particles(rng, 30000, nx, ny, 1e-4, 1e-4, 3e5))
        ctx.poisson_create(EPS0)
        _setup_bc(ctx, "slab", nx, ny)
        assert ctx.set_method(method) == method
        ctx.step(1e-11, 4, seed=1, rtol=1e-9)
        ctx.sync()
        out.append(ctx.field(lib.FIELD_PHI))
        ctx.close()
    assert np.max(np.abs(out[0] - out[1])) <= 1e-7 * np.max(np.abs(out[1]))


def test_tight_tolerances_and_the_network_keep_cg(lib):
    """A tolerance below 1e-9 and an attached warm-start network take CG, mid-run
    too, and the direct solve returns afterwards; an ensemble still refuses the
    operator."""
    from iskra_gb300.device import Ensemble
    from iskra_gb300._lib import IskraError
    nx, ny = 40, 24
    rho = np.random.default_rng(1).normal(0, 1e-6, (nx, ny))
    ctx = make_ctx(nx, ny, 1e-3, 1e-3)
    ctx.poisson_create(EPS0)
    _setup_bc(ctx, "slab", nx, ny)
    tight, it, rr = ctx.solve_host(-rho, rtol=1e-12, maxit=500)
    assert rr <= 1e-12 and it > 3
    loose, it, rr = ctx.solve_host(-0.5 * rho, rtol=1e-9, maxit=500)
    assert rr <= 1e-9 and it <= 3
    again, _, rr = ctx.solve_host(-rho, rtol=1e-9, maxit=500)
    assert rr <= 1e-9 and np.max(np.abs(again - tight)) <= 1e-7 * np.max(np.abs(tight))
    ctx.lws_create(4, seed=1)
    assert ctx.set_method(0) == 2
    _, it, rr = ctx.solve_host(-0.3 * rho, rtol=1e-9, maxit=500)
    assert rr <= 1e-9 and it > 3
    ctx.lws_destroy()
    assert ctx.set_method(0) == 0
    ctx.close()
    ctx = make_ctx(20, 12, 1e-3, 1e-3)
    ctx.species_create(-QE, ME, 1e4, 100)
    ctx.poisson_create(EPS0)
    _setup_bc(ctx, "slab", 20, 12)
    with pytest.raises(IskraError):
        ens = Ensemble(ctx, 2, 100)
        ens.step(1e-11, 1)
        ens.sync()
    ctx.close()
