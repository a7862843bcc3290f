"""Asking for the solver in effect changes nothing: steps with the question between them
leave the potential with the same bits as steps without, at tolerances where an
operator of odd ny takes CG and where it is solved directly."""
import numpy as np
import pytest

from test_gpu_parity import EPS0, ME, QE, _setup_bc, make_ctx, rand_particles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,nx,ny,rtol,solver", [("slab", 33, 7, 1e-10, 0), ("slab", 130, 97, 1e-10, 0),
                                                    ("slab", 33, 7, 1e-8, 0), ("slab", 64, 32, 1e-10, 0),
                                                    ("open_box", 20, 20, 1e-9, 2)])
def test_query_between_steps(lib, kind, nx, ny, rtol, solver):
    out = []
    for ask in (False, True):
        ctx = make_ctx(nx, ny, 1e-4, 1e-4)
        s = ctx.species_create(-QE, ME, 2e4, 20000)
        ctx.set_boundary(s, lib.BND_WRAP, lib.BND_WRAP)
        ctx.upload(s, *rand_particles(np.random.default_rng(nx), 20000, nx, ny, 1e-4, 1e-4, 3e5))
        ctx.poisson_create(EPS0)
        _setup_bc(ctx, kind, nx, ny)
        for k in range(4):
            ctx.step(1e-11, 1, seed=1, rtol=rtol)
            if ask:
                assert ctx.set_method(0) == solver
        out.append(ctx.field(lib.FIELD_PHI))
        ctx.close()
    assert np.array_equal(out[0], out[1])
