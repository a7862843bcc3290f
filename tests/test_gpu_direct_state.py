"""The state of direct solves whose ny is no power of two is FP64, as in CG solves of
the same operators: rho of the same positions has the same bits through both solvers,
and the E that pushes particles is the stored FP64 field rounded once."""
import numpy as np
import pytest

from test_gpu_parity import EPS0, ME, QE, _setup_bc, make_ctx, rand_particles

pytestmark = pytest.mark.gpu


def _ctx(lib, nx, ny, n, method):
    rng = np.random.default_rng(nx + ny)
    ctx = make_ctx(nx, ny, 1e-4, 1e-4)
    s = ctx.species_create(-QE, ME, 2e4, n)
    ctx.set_boundary(s, lib.BND_DISCARD, lib.BND_WRAP)
    ctx.upload(s, *rand_particles(rng, n, nx, ny, 1e-4, 1e-4, 3e5))
    ctx.set_background(rng.normal(QE * 2e12, QE * 1e11, (nx, ny)))
    ctx.poisson_create(EPS0)
    _setup_bc(ctx, "slab", nx, ny)
    assert ctx.set_method(method) == method
    return ctx, s


@pytest.mark.parametrize("nx,ny", [(33, 7), (65, 24), (50, 33), (301, 97)])
def test_charge_density_keeps_its_bits(lib, nx, ny):
    out = []
    for method in (0, 2):
        ctx, s = _ctx(lib, nx, ny, 30000, method)
        ctx.step(1e-11, 1, seed=1, rtol=1e-8)
        ctx.sync()
        out.append(ctx.field(lib.FIELD_RHO))
        ctx.close()
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("nx,ny", [(33, 7), (65, 24), (50, 33), (301, 97)])
def test_pushed_field_is_the_stored_field(lib, nx, ny):
    """A second context takes E from the host (FP64, rounded once by the upload) and
    pushes the same particles: bit for bit what the step's own E does to them."""
    ctx, s = _ctx(lib, nx, ny, 30000, 0)
    ctx.step(1e-11, 2, seed=1, rtol=1e-8)
    ctx.sync()
    E = ctx.field(lib.FIELD_E)
    x, v, ids = ctx.download(s)
    out = []
    for own in (True, False):
        if own:
            c, sid = ctx, s
        else:
            c, sid = _ctx(lib, nx, ny, 30000, 0)
            c.upload_E(E)
        c.upload(sid, x, v, ids=ids)
        c.advance(sid, 1e-10)
        xx, vv, ii = c.download(sid)
        o = np.argsort(ii)
        out.append((xx[o], vv[o]))
        if not own:
            c.close()
    ctx.close()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
