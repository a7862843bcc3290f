"""The tile sort with eight particles per lane (large stores) and one (small ones),
at counts around a warp's and a round's share, with discarded particles among them:
a sort moves whole records, so the particles by identifier are the same bits before
and after (tile size changed and changed back, each followed by another sort)."""
import numpy as np
import pytest

from test_gpu_parity import ME, QE, make_ctx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cap,n", [(3_000_000, 1), (3_000_000, 255), (3_000_000, 256), (3_000_000, 257),
                                   (3_000_000, 311297), (3_000_000, 2_990_001), (4000, 3999), (2_400_000, 2_400_000)])
def test_sort_keeps_every_record(lib, cap, n):
    rng = np.random.default_rng(n)
    nx, ny, dx = 90, 70, 1e-3
    ctx = make_ctx(nx, ny, dx, dx)
    s = ctx.species_create(-QE, ME, 1e5, cap)
    ctx.set_boundary(s, lib.BND_DISCARD, lib.BND_WRAP)
    x = np.asfortranarray(np.column_stack([rng.uniform(0, (nx - 1) * dx, n), rng.uniform(0, (ny - 1) * dx, n)]))
    v = np.asfortranarray(rng.normal(0, 1e6, (n, 3)))
    ctx.upload(s, x, v)
    ctx.advance(s, 5e-11)  # some leave in x and are dropped by the sort
    xa, va, ia = ctx.download(s)
    for size in (8, 16):
        ctx.set_tile(size)
        ctx.sort(s)
    xb, vb, ib = ctx.download(s)
    oa, ob = np.argsort(ia), np.argsort(ib)
    assert np.array_equal(ia[oa], ib[ob])
    assert np.array_equal(xa[oa], xb[ob]) and np.array_equal(va[oa], vb[ob])
    ctx.close()
