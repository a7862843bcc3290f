"""DSMC passes at the edges of their launch shapes: the one-block bucketing (at
most 8192 nodes and 32768 slots) against the three-launch one, and cells of one
to several rounds of pairs.  The same particles in species of a small and a
large capacity take the two bucketings: states, remainders and collision counts
are equal bit for bit."""
import numpy as np
import pytest

from test_gpu_parity import ME, QE, by_id, make_ctx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,npart,dt", [(3, 700, 1e-11), (12, 3000, 4e-9), (20, 5000, 1e-9), (91, 16000, 1e-7),
                                        (40, 1, 1e-9), (2, 33, 1e-9)])
@pytest.mark.parametrize("same", [False, True])
def test_bucketings_agree(lib, n, npart, dt, same):
    dh = 0.05
    rng = np.random.default_rng(n + npart)
    L = (n - 1) * dh
    sets = [(rng.uniform(0, L, (npart, 2)), rng.standard_normal((npart, 3)) * s) for s in (5e5, 800.0)]
    out = []
    for cap in (max(npart, 32000), 40000):
        ctx = make_ctx(n, n, dh, dh)
        sids = []
        for (x, v), (q, m) in zip(sets, ((-QE, ME), (0.0, 1.3e-26))):
            s = ctx.species_create(q, m, 1.0, cap)
            ctx.upload(s, x, v)
            sids.append(s)
        k = ctx.dsmc_create(sids[0], sids[0] if same else sids[1], [3e5, 6e5, 9e5, 12e5], [0.05, 0.5, 2.0, 0.05])
        for step in (1, 2, 3):
            ctx.dsmc_perform(k, dt, seed=3, step=step)
        rem, nu = ctx.dsmc_state(k)
        out.append([rem, nu] + [a for s in sids for a in by_id(*ctx.download(s))])
        ctx.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
    if npart >= 3000:
        assert out[0][1].sum() > 0
