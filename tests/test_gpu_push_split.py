"""The push on grids of few tiles, whose particles are split over several
blocks per tile (at least 384 particles each): the smallest and largest
slices, remainders of a warp and of a slice.  Positions, velocities and the
deposit against the oracle from the device's own state: positions within 1e-6
of max(|x|, dx), velocities within 1e-6, density within 1e-9 of its maximum
(the tolerances of the push parity tests)."""
import numpy as np
import pytest

from test_gpu_parity import ME, QE, by_id, check_push, make_ctx, rand_particles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,n", [(10, 10, 1), (10, 10, 33), (10, 10, 384), (10, 10, 385), (10, 10, 40 * 384 + 1),
                                     (257, 2, 9000), (257, 2, 105001), (3, 40, 5000)])
def test_split_tiles_match_the_oracle(orc, lib, nx, ny, n):
    dx, w, dt = 1e-4, 1e3, 1e-10
    rng = np.random.default_rng(n + nx)
    ctx = make_ctx(nx, ny, dx, dx)
    sid = ctx.species_create(-QE, ME, w, n)
    ctx.set_boundary(sid, lib.BND_WRAP, lib.BND_WRAP)
    ctx.upload(sid, *rand_particles(rng, n, nx, ny, dx, dx, 3e5))
    E = np.asfortranarray(rng.normal(0, 2e3, (nx, ny, 3)))
    E[:, :, 2] = 0.0
    ctx.upload_E(E)
    x0, v0, i0 = by_id(*ctx.download(sid))
    ctx.advance(sid, dt)
    dens = ctx.density(sid)
    x1, v1, i1 = by_id(*ctx.download(sid))
    assert np.array_equal(i0, i1)
    xr, vr = x0.copy(order="F"), v0.copy(order="F")
    pu = orc.grid_to_particle(E.astype(np.float32).astype(np.float64), dx, dx, xr)
    orc.push_cartesian(xr, vr, pu, None, -QE / ME, dt)
    for d, (nn, h) in enumerate(((nx, dx), (ny, dx))):
        orc.wrap(xr, d, nn, h)
    # a particle within rounding of the wrap seam may land on either side of it
    for d, nn in enumerate((nx, ny)):
        L = (nn - 1) * dx
        off = np.abs(x1[:, d] - xr[:, d]) > 0.5 * L
        xr[off, d] += np.where(x1[off, d] > xr[off, d], L, -L)
    check_push(x1, v1, xr, vr, v0, dx)
    ref = orc.density(nx, ny, dx, dx, np.asfortranarray(x1), w, (0, 0, 0, 0))
    assert np.max(np.abs(dens - ref)) <= 1e-9 * np.max(np.abs(ref))
    ctx.close()
