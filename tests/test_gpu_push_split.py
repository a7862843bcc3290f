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


@pytest.mark.parametrize("n,cap", [(4095, 5000), (4096, 5000), (65536, 70000), (65536, 8 * 65536),
                                   (65536, 8 * 65536 + 1)])
def test_steps_after_a_source_fill_do_not_depend_on_its_sort(lib, n, cap):
    """A species filled by a source is sorted once before its first step when
    the fill is large (at least 4096 particles and an eighth of the
    capacity): same fields, bit for bit, as with an explicit sort or none."""
    out = []
    for how in ("auto", "sorted", "never"):
        ctx = make_ctx(65, 33, 1e-4, 1e-4)
        sid = ctx.species_create(-QE, ME, 1e3, cap)
        ctx.set_boundary(sid, lib.BND_DISCARD, lib.BND_WRAP)
        src = ctx.source_create(sid, (n + 0.5) / 1e-11, [64e-4, 32e-4], [6e5, 6e5, 6e5])
        ctx.source_sample(src, 1e-11, seed=5)
        ctx.poisson_create(8.8541878128e-12)
        col = np.zeros((65, 33), bool)
        col[0, :] = True
        ctx.apply_dirichlet(col, 0.0)
        if how == "sorted":
            ctx.sort(sid)
        if how == "never":
            ctx.set_sort_every(0)
        ctx.step(1e-11, 3, seed=1, rtol=1e-8)
        x, v, _ = by_id(*ctx.download(sid))
        out.append((x, v, ctx.field(lib.FIELD_RHO), ctx.field(lib.FIELD_PHI)))
        ctx.close()
    for o in out[1:]:
        for a, b in zip(out[0], o):
            assert np.array_equal(a, b)
