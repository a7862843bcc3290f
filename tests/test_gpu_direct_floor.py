"""Operators of ny with an odd factor on wide grids, uniform rho: the recomputed residual
of a direct solve has a rounding floor that grows with nx^2, and tolerances below it
are met by CG as before these operators were solved directly.  The potential between
the columns of 0 and 100 V is 100 s + rho/(2 eps0) x (L - x), s = x / L, exactly in the
discrete operator too: within 1e-7 of its maximum (CG's own recomputed residual
is up to 3e-8 at 12000 columns)."""
import numpy as np
import pytest

from test_gpu_parity import EPS0, ME, QE, _setup_bc, make_ctx, rand_particles

pytestmark = pytest.mark.gpu
RHO = 1e-6


def _ctx(nx, ny):
    ctx = make_ctx(nx, ny, 1e-3, 1e-3)
    ctx.poisson_create(EPS0)
    _setup_bc(ctx, "slab", nx, ny)
    return ctx


def _exact(nx, ny):
    x = np.arange(nx) * 1e-3
    phi = 100.0 * x / x[-1] + RHO / (2 * EPS0) * x * (x[-1] - x)
    return np.repeat(phi[:, None], ny, axis=1)


@pytest.mark.parametrize("rtol", [1e-8, 1e-9])
@pytest.mark.parametrize("nx,ny", [(1500, 12), (4096, 3), (4096, 12), (6000, 97), (12000, 12)])
def test_wide_grids_meet_the_tolerance(lib, nx, ny, rtol):
    ctx = _ctx(nx, ny)
    phi, it, rr = ctx.solve_host(np.full((nx, ny), -RHO), rtol=rtol)
    assert rr <= rtol
    ref = _exact(nx, ny)
    assert np.max(np.abs(phi - ref)) <= 1e-7 * np.max(ref)
    ctx.close()


@pytest.mark.parametrize("nx,ny,rtol", [(97, 3, 1e-9), (300, 3, 1e-9), (2000, 12, 1e-9), (4096, 12, 1e-8),
                                        (12000, 12, 1e-9), (700, 255, 1e-9), (64, 1023, 1e-9)])
def test_steps_from_a_cold_start(lib, nx, ny, rtol):
    """Captured steps: as many corrections as a solve takes, CG where they stall."""
    ctx = _ctx(nx, ny)
    s = ctx.species_create(-QE, ME, 1e-3, 100)  # (no weight to speak of)
    ctx.set_boundary(s, lib.BND_WRAP, lib.BND_WRAP)
    ctx.upload(s, *rand_particles(np.random.default_rng(nx), 100, nx, ny, 1e-3, 1e-3, 1e3))
    ctx.set_background(np.full((nx, ny), RHO))
    ref = _exact(nx, ny)
    for steps in (1, 5):
        ctx.step(1e-12, steps, seed=1, rtol=rtol)
        it, rr = ctx.solve_info()
        assert rr <= rtol
        assert np.max(np.abs(ctx.field(lib.FIELD_PHI) - ref)) <= 1e-7 * np.max(ref)
    ctx.close()


def test_looser_tolerances_stay_direct(lib):
    nx, ny = 12000, 12
    ctx = _ctx(nx, ny)
    f = np.full((nx, ny), -RHO)
    _, it, rr = ctx.solve_host(f, rtol=1e-9)
    assert rr <= 1e-9
    _, it, rr = ctx.solve_host(0.5 * f, rtol=1e-7)
    assert rr <= 1e-7 and it <= 4
    ctx.close()


def test_errors_end_the_call(lib):
    """A direct step of such an operator reports a flag at its step, and a solve that
    meets no number reports ISKRA_ENOTCONV."""
    from iskra_gb300._lib import IskraError
    for nx, ny in ((33, 7), (301, 97)):
        ctx = _ctx(nx, ny)
        s = ctx.species_create(-QE, ME, 1e-3, 100)
        ctx.set_boundary(s, lib.BND_WRAP, lib.BND_WRAP)
        ctx.upload(s, *rand_particles(np.random.default_rng(nx), 100, nx, ny, 1e-3, 1e-3, 1e3))
        ctx.set_sort_every(0)
        ctx.step(1e-12, 2, seed=1, rtol=1e-8)
        per_step = ctx.kernel_launches() // 2
        assert per_step > 0
        bg = np.zeros((nx, ny))
        bg[nx // 2, ny // 2] = np.nan
        ctx.set_background(bg)
        with pytest.raises(IskraError) as e:
            ctx.step(1e-12, 20, seed=1, rtol=1e-8)
        assert e.value.code == 9  # ISKRA_ENOTCONV
        assert ctx.kernel_launches() == 3 * per_step
        ctx.close()


@pytest.mark.parametrize("every", [0, 2])
def test_going_over_to_cg_inside_a_call(lib, every):
    """A call whose first solve stalls does the rest of its steps through CG: the same
    bits as one call per step."""
    nx, ny, rtol = 12000, 12, 1e-9
    out = []
    for calls in ([4], [1, 1, 1, 1]):
        ctx = _ctx(nx, ny)
        s = ctx.species_create(-QE, ME, 1e-3, 100)
        ctx.set_boundary(s, lib.BND_WRAP, lib.BND_WRAP)
        ctx.upload(s, *rand_particles(np.random.default_rng(nx), 100, nx, ny, 1e-3, 1e-3, 1e3))
        ctx.set_background(np.full((nx, ny), RHO))
        ctx.set_sort_every(every)
        for n in calls:
            ctx.step(1e-12, n, seed=1, rtol=rtol)
        it, rr = ctx.solve_info()
        assert rr <= rtol
        x, v, ids = ctx.download(s)
        o = np.argsort(ids)
        out.append((ctx.field(lib.FIELD_PHI), x[o], v[o]))
        ctx.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
