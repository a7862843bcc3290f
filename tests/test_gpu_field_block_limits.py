"""Both sides of each limit of the one-block field part of a step: the same comparison
with the single stages as at the other sizes, and which path ran.  A captured step of one
species is its push and, in one block, one field kernel; the launches of the larger
direct solves are at least seven, and CG solves run by the host are not captured (0)."""
import numpy as np
import pytest

import test_gpu_field_block as field_block
from test_gpu_parity import EPS0, ME, QE, _setup_bc, make_ctx, rand_particles

pytestmark = pytest.mark.gpu


def _kernels_per_step(lib, kind, nx, ny, rtol):
    ctx = make_ctx(nx, ny, 1e-4, 1e-4)
    s = ctx.species_create(-QE, ME, 2e4, 1000)
    ctx.set_boundary(s, lib.BND_WRAP, lib.BND_WRAP)
    ctx.upload(s, *rand_particles(np.random.default_rng(nx), 1000, nx, ny, 1e-4, 1e-4, 2e5))
    ctx.poisson_create(EPS0)
    _setup_bc(ctx, kind, nx, ny)
    ctx.set_sort_every(0)
    ctx.step(1e-11, 1, seed=1, rtol=rtol)
    n = ctx.kernel_launches()
    ctx.close()
    return n


@pytest.mark.parametrize("kind,nx,ny,rtol,path", [
    # multigrid CG: 40 bytes a node, the levels (56 bytes a node each) and the coarsest
    # inverse within 192 KB
    ("open_box", 36, 36, 1e-10, "block"), ("open_box", 37, 37, 1e-10, "host"),
    # direct: 1536 nodes, 4096 at ny = 2
    ("slab", 48, 32, 1e-9, "block"), ("slab", 49, 32, 1e-9, "launches"),
    ("slab", 2048, 2, 1e-9, "block"), ("slab", 2049, 2, 1e-9, "launches"),
    ("slab", 64, 24, 1e-9, "block"), ("slab", 65, 24, 1e-9, "launches")])
def test_either_side_of_the_limits(lib, kind, nx, ny, rtol, path):
    n = _kernels_per_step(lib, kind, nx, ny, rtol)
    assert {"block": 0 < n <= 2, "launches": n >= 7, "host": n == 0}[path], n
    field_block.test_step_field_matches_the_single_stages(lib, kind, nx, ny, rtol)
