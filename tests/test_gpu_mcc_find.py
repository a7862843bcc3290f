"""The single-context collision search at the edges of its rounds (32 slots a
warp and step; rounds of 2 or 8, chosen by the species' capacity): the same
particles collide, with the same velocities bit for bit, whichever round size
the capacity picks, and the counts are the ones the particles show."""
import numpy as np
import pytest

from test_gpu_parity import ME, QE, by_id, make_ctx, rand_particles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("table", ["log", "uneven"])
@pytest.mark.parametrize("n", [1, 31, 33, 511, 513, 2047, 70001])
def test_rounds_find_the_same_collisions(lib, n, table):
    nx, ny, dx = 33, 17, 1e-4
    eps = np.logspace(-2, 3, 256) if table == "log" else np.r_[0.01, np.linspace(0.5, 30, 61), 80.0, 1000.0]
    el, ex = np.full(len(eps), 4e-19), np.where(eps > 11.5, 2e-19, 0.0)
    gas = np.full((nx, ny), 2e21)
    rng = np.random.default_rng(n)
    x, v = rand_particles(rng, n, nx, ny, dx, dx, 1.5e6)
    out = []
    for cap in (n + 1, 1_300_000):
        ctx = make_ctx(nx, ny, dx, dx)
        s = ctx.species_create(-QE, ME, 1.0, cap)
        ctx.upload(s, x, v)
        m, _ = ctx.mcc_create(s, [(lib.MCC_ELASTIC_ISOTROPIC, 0.0, eps, el), (lib.MCC_EXCITATION, 11.5, eps, ex)],
                              6.63e-26, 300.0, gas)
        counts = np.zeros(2, np.int64)
        for step in (1, 2):
            ctx.mcc_perform(m, 2e-11, 7, step)
            counts += ctx.mcc_counts(m, 2)
        out.append((*by_id(*ctx.download(s)), counts))
        ctx.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
    changed = np.any(out[0][1] != v.astype(np.float32), axis=1).sum()
    assert changed <= out[0][3].sum()
    if n > 5000:
        assert 0.01 * n < changed
