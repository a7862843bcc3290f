"""Failing steps of the one-block multigrid CG: iskra_step returns the error of the
step that failed without running the ones after it (as where the host runs the
solve), and a residual that is no number ends the iteration at once."""
import numpy as np
import pytest

from test_gpu_parity import EPS0, ME, QE, _setup_bc, make_ctx, rand_particles

pytestmark = pytest.mark.gpu


def _box(lib, n, cap, np_):
    ctx = make_ctx(n, n, 1e-4, 1e-4)
    s = ctx.species_create(-QE, ME, 2e5, cap)
    ctx.set_boundary(s, lib.BND_WRAP, lib.BND_WRAP)
    ctx.upload(s, *rand_particles(np.random.default_rng(n), np_, n, n, 1e-4, 1e-4, 2e5))
    ctx.poisson_create(EPS0)
    _setup_bc(ctx, "open_box", n, n)
    ctx.set_sort_every(0)
    return ctx, s


@pytest.mark.parametrize("n", [10, 20, 30])
def test_call_ends_at_the_step_that_failed(lib, n):
    from iskra_gb300._lib import IskraError
    ctx, s = _box(lib, n, 1000, 1000)
    ctx.step(1e-11, 2, seed=1, rtol=1e-9)
    per_step = ctx.kernel_launches() // 2
    assert per_step > 0  # (captured steps are counted: the one-block path)
    bg = np.zeros((n, n))
    bg[1, n - 2] = np.nan
    ctx.set_background(bg)
    with pytest.raises(IskraError) as e:
        ctx.step(1e-11, 50, seed=1, rtol=1e-9)
    assert e.value.code == 9  # ISKRA_ENOTCONV
    assert ctx.kernel_launches() == 3 * per_step
    it, rr = ctx.solve_info()
    assert it <= 1 and not rr <= 1e-9
    ctx.close()


def test_other_errors_end_the_call_too(lib):
    """A full species dropping sampled particles: ISKRA_ECAPACITY is not raised by
    sources (they stop at the capacity), so an out-of-range particle on an axis
    without a boundary rule stands for the other flags."""
    from iskra_gb300._lib import IskraError
    ctx, s = _box(lib, 12, 1000, 1000)
    ctx.step(1e-11, 1, seed=1, rtol=1e-9)
    per_step = ctx.kernel_launches()
    ctx.set_boundary(s, lib.BND_NONE, lib.BND_NONE)
    with pytest.raises(IskraError) as e:
        ctx.step(1e-9, 20, seed=1, rtol=1e-9)  # 2e5 m/s x 1e-9 s: two cells a step
    assert e.value.code == 4  # ISKRA_EDOMAIN
    assert ctx.kernel_launches() <= 3 * per_step
    ctx.close()
