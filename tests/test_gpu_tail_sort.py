"""Sorts for the sake of particles sampled between step calls: at most one per sort
period (a source at the species' capacity appends nothing, yet its samples count), none
for samples that a periodic sort has taken up.  Sorts are told from steps by their
kernels; particles by identifier do not depend on them."""
import numpy as np
import pytest

from test_gpu_parity import EPS0, ME, QE
from test_gpu_source import D, DX, L, N, WV, WX

pytestmark = pytest.mark.gpu
DT = 1e-12


def _ctx(lib, cap, every):
    from iskra_gb300.device import Context
    ctx = Context(N, N, D, D, (0, 0, 0, 0))
    s = ctx.species_create(-QE, ME, 1e-3, cap)
    ctx.set_boundary(s, lib.BND_WRAP, lib.BND_WRAP)
    ctx.poisson_create(EPS0)
    ctx.apply_periodic(1)
    wall = np.zeros((N, N), bool)
    wall[[0, -1], :] = True
    ctx.apply_dirichlet(wall, 0.0)
    ctx.set_sort_every(every)
    return ctx, s


def _kernels(lib, every, steps):
    ctx, s = _ctx(lib, 8192, every)
    ctx.step(DT, steps, seed=1, rtol=1e-8)
    n = ctx.kernel_launches()
    ctx.close()
    return n


@pytest.mark.parametrize("cap,sample,every,tail_sorts", [(8192, 8192, 16, 3), (8192, 2048, 16, 3), (32768, 1000, 4, 0),
                                                         (32768, 4095, 1000, 1), (4095, 4095, 16, 0)])
def test_sorts_per_period(lib, cap, sample, every, tail_sorts):
    step = _kernels(lib, 0, 1)
    sort = _kernels(lib, 1, 1) - step
    assert step > 0 and sort > 0
    ctx, s = _ctx(lib, cap, every)
    src = ctx.source_create(s, (sample + 0.5) / DT, WX, WV, DX, None)
    steps = 40
    for k in range(steps):
        ctx.source_sample(src, DT, seed=k)
        ctx.step(DT, 1, seed=1, rtol=1e-8)
    periodic = steps // every
    assert ctx.kernel_launches() == steps * step + (periodic + tail_sorts) * sort
    assert ctx.count(s) == min(cap, steps * sample)
    ctx.close()
