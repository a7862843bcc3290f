"""Ensemble push on particle orders that take either way of its deposit (lane by
lane, or summed over runs of equal cells), with and without the next step's
collision selection: the density after a step equals a single-run context's bit for
bit (integer deposit).  Particles that cross several periods of a wrapped axis in a
step come back to where the modulo puts them (offsets are kept to 2^-24 of a cell:
tolerance 4 of those, after an FP32 step of up to 8 cells, 8 x 2^-24)."""
import numpy as np
import pytest

from test_gpu_ensemble import DT, DX, GAP, NX, configure, initial_state

pytestmark = pytest.mark.gpu


def _order(kind, x, v):
    n = len(x)
    if kind == "sorted":
        o = np.argsort(x[:, 0], kind="stable")
        return x[o], v[o]
    if kind == "one_cell":
        x = x.copy()
        x[:, 0] = (NX // 3 + x[:, 0] / GAP) * DX
        return x, v * 1e-3
    if kind == "pairs":  # seven neighbours of 32 in the same cell: just above the limit of six
        x, v = x.copy(), v.copy()
        for k in range(7):
            x[4 * k + 1::32] = x[4 * k::32][:len(x[4 * k + 1::32])]
            v[4 * k + 1::32] = v[4 * k::32][:len(v[4 * k + 1::32])]
        return x, v
    return x, v


@pytest.mark.parametrize("kind,n0,mcc", [("random", 4000, True), ("sorted", 4001, True), ("one_cell", 3000, True),
                                         ("pairs", 4000, False), ("sorted", 31, False), ("random", 1, True),
                                         ("random", 40000, False)])
def test_deposit_of_any_order(lib, kind, n0, mcc):
    from iskra_gb300.device import Ensemble
    w = 1e15 * GAP * DX / n0
    tmpl, se, si, _, _ = configure(lib, n0, 200.0, w, mcc)
    ens = Ensemble(tmpl, 2, 4 * n0 + 64)
    ens.set_seeds([5, 6])
    ens.set_drive_amplitude(0, np.array([200.0, 300.0]))
    states = []
    for r in range(2):
        st = [tuple(np.asfortranarray(a) for a in _order(kind, *s)) for s in initial_state(70 + r, n0)]
        states.append(st)
        for sid, (x, v) in zip((se, si), st):
            ens.upload(r, sid, x, v)
    ens.step(DT, 1)
    ens.sync()
    for r, amp in enumerate((200.0, 300.0)):
        ctx, ce, ci, _, _ = configure(lib, max(n0, 16), amp, w, mcc)
        for sid, (x, v) in zip((ce, ci), states[r]):
            ctx.upload(sid, x, v)
        ctx.step(DT, 1, seed=5 + r, rtol=1e-12)
        ctx.sync()
        assert np.array_equal(ctx.field(lib.FIELD_RHO), ens.field(r, lib.FIELD_RHO))
        ctx.close()
    ens.close()
    tmpl.close()


def test_several_periods(lib):
    from iskra_gb300.device import Ensemble
    n0 = 500
    w = 1e6 * GAP * DX / n0  # a field that moves nothing
    tmpl, se, si, _, _ = configure(lib, n0, 0.0, w, False)
    ens = Ensemble(tmpl, 1, 4 * n0)
    ens.set_seeds([1])
    ens.set_drive_amplitude(0, np.zeros(1))
    rng = np.random.default_rng(3)
    x = np.column_stack([rng.uniform(0.2 * GAP, 0.8 * GAP, n0), rng.uniform(0, DX, n0)])
    v = np.zeros((n0, 3))
    v[:, 1] = rng.uniform(-7.5, 7.5, n0) * DX / DT
    ids = np.arange(1, n0 + 1, dtype=np.uint32)
    ens.upload(0, si, np.asfortranarray(x), np.asfortranarray(v), ids)
    ens.step(DT, 1)
    ens.sync()
    xn, _, got = ens.download(0, si)
    assert len(got) == n0
    y = xn[np.argsort(got), 1] / DX
    ref = x[:, 1] / DX + v[:, 1].astype(np.float32).astype(float) * DT / DX
    d = y - ref
    d -= np.round(d)
    assert np.all((y >= 0) & (y <= 1)) and np.max(np.abs(d)) <= (4 + 8) * 2.0 ** -24
    ens.close()
    tmpl.close()
