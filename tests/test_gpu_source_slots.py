"""Several samples of one species in a step, each taking its slots where the one
before ended: counts (clamped by the capacity), unique identifiers and, as every step
has its own key, velocities that never repeat (the step counter is advanced by a
single species' push and by the last of three alike)."""
import numpy as np
import pytest

from test_gpu_parity import EPS0, ME, QE
from test_gpu_source import D, DX, L, N, WV, WX

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per,cap,species", [((1, 1), 1000, 1), ((255, 257), 100000, 1), ((4000, 300), 9000, 3)])
def test_samples_share_a_species(lib, per, cap, species):
    from iskra_gb300.device import Context
    ctx = Context(N, N, D, D, (0, 0, 0, 0))
    sids = [ctx.species_create(-QE, ME, 1e-3, cap) for _ in range(species)]
    for s in sids:
        ctx.set_boundary(s, lib.BND_WRAP, lib.BND_WRAP)
    ctx.poisson_create(EPS0)
    ctx.apply_periodic(1)
    wall = np.zeros((N, N), bool)
    wall[[0, -1], :] = True
    ctx.apply_dirichlet(wall, 0.0)
    dt, steps = 1e-12, 3
    for n in per:
        ctx.source_every_step(ctx.source_create(sids[0], (n + 0.5) / dt, WX, WV, DX, None), True)
    ctx.step(dt, steps, seed=9, rtol=1e-8)
    ctx.sync()
    want = min(cap, steps * sum(per))
    assert ctx.count(sids[0]) == want
    _, v, ids = ctx.download(sids[0])
    assert len(ids) == want and len(np.unique(ids)) == want
    assert len(np.unique(v[:, 2])) >= want - 2 - want // 1000  # (24-bit draws may coincide)
    ctx.close()
