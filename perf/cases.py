"""What users of the framework run, as measurable cases.

A case is one call pattern of a user's program on one size: a configured
context (grid, species, operator, collision sets: what the program keeps) and
one pass through the public entry points -- a few steps and the field record
that a program reads after them, one solve, one collision pass, one network
evaluation.  Field and particle records are kept in single precision, the
precision of the particle state; solves called by themselves return FP64.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from iskra_gb300 import _lib, chemistry, device
from iskra_gb300 import finite_difference_method as fdm
from iskra_gb300 import particle_in_cell as pic
from iskra_gb300.regular_grids import create_uniform_grid

QE = 1.602176634e-19
ME = 9.1093837015e-31
AMU = 1.66053906660e-27
KB = 1.380649e-23
EPS0 = 8.8541878128e-12
M_AR = 39.948 * AMU
F_RF, DT_RF = 13.56e6, 7.4e-11  # drive frequency and time step of the discharges


def listed():
    return [
        # the smallest whole step: 1D counter-streaming beams, periodic, read after every step
        {"name": "two_stream_step", "kind": "two_stream", "nx": 128, "np": 40000, "steps": 1},
        # the reference's boundary problem: beam source, floating and fixed electrodes, reflecting block
        {"name": "boundaries_10", "kind": "boundaries", "n": 10, "np": 20000, "steps": 10},
        # one plain run of the RF discharge (e- and Ar+ collisions), a record every 5 steps
        {"name": "discharge_1d", "kind": "discharge", "nx": 257, "np": 105000, "steps": 5, "circuit": False,
         "table": "log"},
        # the same discharge behind the series RLC circuit, with measured (unevenly spaced) cross sections
        {"name": "discharge_rlc", "kind": "discharge", "nx": 201, "np": 41000, "steps": 5, "circuit": True,
         "table": "uneven"},
        # the benchmark's plasma slab
        {"name": "slab_512", "kind": "slab", "nx": 512, "ny": 512, "np": 4000000, "steps": 20, "tracker": False},
        # a slab of odd sizes
        {"name": "slab_odd", "kind": "slab", "nx": 301, "ny": 97, "np": 400000, "steps": 5, "tracker": False},
        # a parameter scan of small discharges advanced together
        {"name": "ensemble_128", "kind": "ensemble", "nx": 257, "runs": 128, "np_lo": 10000, "np_hi": 200000,
         "steps": 10},
        # the large 2D discharge, iterative solver
        {"name": "discharge_2d_1024", "kind": "discharge_2d", "n": 1024, "np": 1 << 25, "steps": 3},
        # field solves by themselves: open box with an internal electrode, two charge distributions in turn,
        # host right-hand sides and potentials
        {"name": "poisson_box", "kind": "poisson", "nx": 321, "ny": 203, "open": True},
        # DSMC collisions of the reference's problem 05
        {"name": "dsmc_05", "kind": "dsmc", "n": 20, "np": 5000, "dt": 1e-9, "performs": 10},
        # host arrays in, a short run, host arrays out
        {"name": "round_trip", "kind": "round_trip", "nx": 128, "ny": 64, "np": 200000, "steps": 10},
        # the warm-start network: one evaluation and one gradient (forward and backward)
        {"name": "network_grad", "kind": "network", "nx": 256, "ny": 192},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["two_stream", "boundaries", "discharge", "slab", "slab", "ensemble", "discharge_2d", "poisson",
                       "dsmc", "round_trip", "network"])
    if kind == "two_stream":
        return {"kind": kind, "nx": _log_int(rng, 24, 600), "np": _log_int(rng, 2000, 200000),
                "steps": rng.randint(1, 4)}
    if kind == "boundaries":
        return {"kind": kind, "n": rng.randint(10, 40), "np": _log_int(rng, 4000, 60000), "steps": rng.randint(4, 12)}
    if kind == "discharge":
        return {"kind": kind, "nx": _log_int(rng, 65, 400), "np": _log_int(rng, 10000, 400000),
                "steps": rng.randint(2, 5), "circuit": rng.random() < 0.4, "table": rng.choice(["log", "uneven"])}
    if kind == "slab":
        ny = 1 << rng.randint(4, 9) if rng.random() < 0.5 else _log_int(rng, 17, 400)
        return {"kind": kind, "nx": _log_int(rng, 33, 700), "ny": ny, "np": _log_int(rng, 20000, 3000000),
                "steps": rng.randint(2, 10), "tracker": rng.random() < 0.3}
    if kind == "ensemble":
        lo = _log_int(rng, 2000, 20000)
        return {"kind": kind, "nx": _log_int(rng, 65, 380), "runs": _log_int(rng, 3, 100), "np_lo": lo,
                "np_hi": _log_int(rng, lo, 150000), "steps": rng.randint(3, 10)}
    if kind == "discharge_2d":
        return {"kind": kind, "n": _log_int(rng, 64, 700), "np": _log_int(rng, 1 << 17, 1 << 24),
                "steps": rng.randint(1, 3)}
    if kind == "poisson":
        return {"kind": kind, "nx": _log_int(rng, 31, 700), "ny": _log_int(rng, 23, 500), "open": rng.random() < 0.6}
    if kind == "dsmc":
        n = rng.randint(3, 40)
        return {"kind": kind, "n": n, "np": _log_int(rng, 2000, 30000), "dt": 1e-9 if n > 12 else 1e-11,
                "performs": rng.randint(2, 12)}
    if kind == "round_trip":
        return {"kind": kind, "nx": _log_int(rng, 32, 300), "ny": 1 << rng.randint(3, 7),
                "np": _log_int(rng, 5000, 500000), "steps": rng.randint(2, 12)}
    return {"kind": kind, "nx": 8 * _log_int(rng, 4, 64), "ny": 8 * _log_int(rng, 3, 64)}


# ---- inputs ------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _maxwell(g, n, lx, ly, vth):
    """n particles uniform over lx x ly, Maxwellian velocities: (2, n) and (3, n) FP64 on the GPU."""
    x = torch.rand((2, n), generator=g, device="cuda", dtype=torch.float64)
    x *= torch.tensor([[lx], [ly]], device="cuda", dtype=torch.float64)
    v = torch.randn((3, n), generator=g, device="cuda", dtype=torch.float64) * vth
    return x, v


def _host(t):
    """(D, n) GPU tensor -> (n, D) column-major host array."""
    return t.cpu().numpy().T


def _pinned(shape, dtype=torch.float64):
    t = torch.empty(int(np.prod(shape)), dtype=dtype, pin_memory=True)
    return t.numpy().reshape(shape, order="F")


def _record(nx, ny):
    """Pinned buffers of a field record and its single-precision copy."""
    return {_lib.FIELD_RHO: (_pinned((nx, ny)), np.empty((nx, ny), np.float32, order="F")),
            _lib.FIELD_PHI: (_pinned((nx, ny)), np.empty((nx, ny), np.float32, order="F")),
            _lib.FIELD_E: (_pinned((nx, ny, 3)), np.empty((nx, ny, 2), np.float32, order="F"))}


def _read(ctx, rec, which):
    """One field into its single-precision record (E: the two in-plane components)."""
    full, single = rec[which]
    ctx.field(which, out=full)
    np.copyto(single, full[..., :2] if which == _lib.FIELD_E else full, casting="same_kind")
    return single


def _columns(nx, ny):
    left = np.zeros((nx, ny), bool)
    left[0, :] = True
    right = np.zeros((nx, ny), bool)
    right[-1, :] = True
    return left, right


# ---- two counter-streaming beams --------------------------------------------
def _two_stream_inputs(case, seed):
    nx, n, L = case["nx"], case["np"], 0.1
    dx = L / (nx - 1)
    x, v = _maxwell(_gen(seed), n, L, dx, 1e4)
    v[1:] = 0.0
    v[0, : n // 2] += 1e6
    v[0, n // 2:] -= 1e6
    return dx, x, v, 2e11 * L * dx / n


def _two_stream(case, seed):
    nx = case["nx"]
    dx, x, v, w = _two_stream_inputs(case, seed)
    ctx = device.Context(nx, 2, dx, dx, (1, 1, 1, 1))
    e = ctx.species_create(-QE, ME, w, case["np"])
    ctx.set_boundary(e, _lib.BND_WRAP, _lib.BND_WRAP)
    ctx.upload(e, _host(x), _host(v))
    ctx.set_background(np.full((nx, 2), QE * 2e11))
    ctx.poisson_create(EPS0)
    ctx.apply_periodic(1)
    ctx.apply_periodic(2)
    return {"ctx": ctx, "rec": _record(nx, 2)}


def _two_stream_run(case, s):
    s["ctx"].step(2e-9, case["steps"], seed=0, rtol=1e-10)
    return _read(s["ctx"], s["rec"], _lib.FIELD_E)


# ---- beam source, electrodes, reflecting block ------------------------------
def _boundaries(case, seed):
    n, dt = case["n"], 10e-9
    dh = 1.0 / n
    xs = np.arange(n) * dh
    grid = create_uniform_grid(xs, xs)
    e = pic.create_kinetic_species("e-", 4 * case["np"], -QE, ME, 50e3, grid)
    cfg = pic.Config()
    cfg.grid = grid
    cfg.solver = fdm.create_poisson_solver(grid, EPS0)
    cfg.species = [e]
    pic.wrap(e, grid)
    q = max(1, n // 10)
    bcs = np.zeros((n, n), np.int8)
    bcs[0, 1:n - 1] = 1
    bcs[n - 1, 4 * q:7 * q] = 2
    bcs[n - 2, 0] = 3
    bcs[n - 2, n - 1] = 3
    bcs[5 * q:8 * q, 4 * q:7 * q] = 4
    driven = pic.create_electrode(bcs == 1, cfg, sigma=1 * EPS0)
    floating = pic.create_electrode(bcs == 2, cfg)
    pic.create_electrode(bcs == 3, cfg, fixed=True)
    block = pic.create_reflective_surface()
    pic.track_surface(cfg.tracker, bcs == 4, block)
    beam = pic.create_thermalized_beam(e, [0.25, 0.5], [0.0, 0.0, 0.0], dx=[0.25, 0.25], T=300.0,
                                       rate=case["np"] / dt)
    pic.init(beam, e, dt, seed=seed)
    # the beam keeps feeding the box: about what its walls take
    feed = pic.create_thermalized_beam(e, [0.25, 0.5], [0.0, 0.0, 0.0], dx=[0.25, 0.25], T=300.0,
                                       rate=(case["np"] / 500 + 0.5) / dt)
    cfg.sources = [feed]
    return {"cfg": cfg, "e": e, "dt": dt, "seed": seed, "surfaces": (driven, floating), "rec": _record(n, n)}


def _boundaries_run(case, s):
    cfg = s["cfg"]
    pic.solve(cfg, s["dt"], case["steps"], seed=s["seed"], rtol=1e-8)
    ctx = cfg.grid.device
    return {"phi": _read(ctx, s["rec"], _lib.FIELD_PHI), "rho": _read(ctx, s["rec"], _lib.FIELD_RHO),
            "hits": [cfg.tracker.hits(x, s["e"]) for x in s["surfaces"]]}


# ---- RF discharges -----------------------------------------------------------
def _tables(kind):
    """Argon-like cross sections: log-uniform nodes, or unevenly spaced ones as measured sets have."""
    if kind == "log":
        eps = np.logspace(-2, 4, 1024)
    else:
        eps = np.concatenate([np.linspace(0.01, 2.0, 40), np.linspace(2.5, 20.0, 71), np.linspace(25.0, 100.0, 31),
                              np.geomspace(120.0, 1e4, 24)])
    el = np.where(eps > 100.0, 1e-17 / eps, 1e-19)
    ex = np.where(eps > 11.5, np.minimum((eps - 11.5) / (100.0 - 11.5), 1.0) * 3e-21, 0.0)
    iz = np.where(eps > 15.76, 3e-20 * np.log(np.maximum(eps, 15.76) / 15.76) / np.log(100 / 15.76)
                  * np.sqrt(100 / eps), 0.0)
    return eps, el, ex, iz, np.full(len(eps), 5e-19)


def _collisions(ctx, se, si, nx, ny, kind):
    eps, el, ex, iz, cx = _tables(kind)
    gas = np.full((nx, ny), 3.0 / (KB * 300.0))
    ctx.mcc_create(se, [(_lib.MCC_ELASTIC_ISOTROPIC, 0.0, eps, el), (_lib.MCC_EXCITATION, 11.5, eps, ex),
                        (_lib.MCC_IONIZATION, 15.76, eps, iz)], M_AR, 300.0, gas, product=si)
    ctx.mcc_create(si, [(_lib.MCC_ELASTIC_BACKWARD, 0.0, eps, cx)], M_AR, 300.0, gas)


def _discharge_ctx(nx, cap, np_norm, amp, circuit, table):
    gap = 0.025
    dx = gap / (nx - 1)
    ctx = device.Context(nx, 2, dx, dx)
    w = 1e15 * gap * dx / np_norm
    se = ctx.species_create(-QE, ME, w, cap)
    si = ctx.species_create(QE, M_AR, w, cap)
    for s in (se, si):
        ctx.set_boundary(s, _lib.BND_DISCARD, _lib.BND_WRAP)
    ctx.poisson_create(EPS0)
    ctx.apply_periodic(1)
    left, right = _columns(nx, 2)
    if circuit:
        dof = ctx.add_dof()
        ctx.apply_neumann(left, dof, gauss=True)
        ctx.apply_dirichlet(right, 0.0)
        ctx.circuit_create(50.0, 1e-6, 1e-9, amp, F_RF, 0.0, dof, left, right, dx, 1.0)
    else:
        ctx.apply_dirichlet(left, 0.0)
        ctx.apply_dirichlet(right, 0.0)
        ctx.drive_dirichlet(left, amp, F_RF)
    _collisions(ctx, se, si, nx, 2, table)
    return ctx, se, si, gap, dx


def _discharge(case, seed):
    n = case["np"]
    ctx, se, si, gap, dx = _discharge_ctx(case["nx"], 3 * n, n, 300.0, case["circuit"], case["table"])
    g = _gen(seed)
    for s, T, m in ((se, 0.5, ME), (si, 0.03, M_AR)):
        x, v = _maxwell(g, n, gap, dx, math.sqrt(2 * T * QE / m))
        ctx.upload(s, _host(x), _host(v))
    return {"ctx": ctx, "seed": seed, "rec": _record(case["nx"], 2)}


def _discharge_run(case, s):
    ctx = s["ctx"]
    ctx.step(DT_RF, case["steps"], seed=s["seed"], rtol=1e-8)
    out = {"phi": _read(ctx, s["rec"], _lib.FIELD_PHI), "rho": _read(ctx, s["rec"], _lib.FIELD_RHO)}
    if case["circuit"]:
        out["circuit"] = np.array(list(ctx.circuit_state().values()), np.float32)
    return out


def _ensemble(case, seed):
    nx, R = case["nx"], case["runs"]
    amps = np.linspace(30.0, 150.0, R)
    nps = np.linspace(case["np_lo"], case["np_hi"], R).astype(int)  # denser plasma at larger drive
    ctx, se, si, gap, dx = _discharge_ctx(nx, 16, int(nps.max()), 100.0, False, "log")
    ens = device.Ensemble(ctx, R, int(nps.max() * 1.5) + 1024)
    ens.set_seeds([seed + r for r in range(R)])
    ens.set_drive_amplitude(0, amps)
    g = _gen(seed)
    for r in range(R):
        for s, T, m in ((se, 0.5, ME), (si, 0.03, M_AR)):
            x, v = _maxwell(g, int(nps[r]), gap, dx, math.sqrt(2 * T * QE / m))
            ens.upload(r, s, _host(x), _host(v))
    return {"ens": ens, "ctx": ctx, "phi": np.empty((R, nx, 2), np.float32)}


def _ensemble_run(case, s):
    s["ens"].step(DT_RF, case["steps"])
    for r in range(case["runs"]):
        s["phi"][r] = s["ens"].field(r, _lib.FIELD_PHI)
    return s["phi"]


def _discharge_2d(case, seed):
    n, npart, dx = case["n"], case["np"], 1e-4
    L = (n - 1) * dx
    w = 1e15 * L * L / npart
    ctx = device.Context(n, n, dx, dx, (0, 0, 0, 0))
    sids = []
    for q, m, T in ((-QE, ME, 0.5), (QE, M_AR, 0.03)):
        sid = ctx.species_create(q, m, w, int(npart * 1.25) + 4096)
        ctx.set_boundary(sid, _lib.BND_DISCARD, _lib.BND_WRAP)
        src = ctx.source_create(sid, (npart + 0.5) / DT_RF, (L, L), math.sqrt(2 * T * QE / m))
        ctx.source_sample(src, DT_RF, seed=2 * seed + len(sids))
        sids.append(sid)
    ctx.poisson_create(EPS0)
    ctx.apply_periodic(1)
    left, right = _columns(n, n)
    ctx.apply_dirichlet(left, 0.0)
    ctx.apply_dirichlet(right, 0.0)
    ctx.drive_dirichlet(left, 300.0, F_RF)
    _collisions(ctx, sids[0], sids[1], n, n, "log")
    ctx.set_method(2)
    return {"ctx": ctx, "seed": seed, "rec": _record(n, n)}


def _discharge_2d_run(case, s):
    ctx = s["ctx"]
    ctx.step(DT_RF, case["steps"], seed=s["seed"], rtol=1e-8)
    return {"phi": _read(ctx, s["rec"], _lib.FIELD_PHI), "rho": _read(ctx, s["rec"], _lib.FIELD_RHO)}


# ---- plasma slab -------------------------------------------------------------
def _slab_inputs(case, seed):
    nx, ny, n, dx = case["nx"], case["ny"], case["np"], 1e-4
    lx, ly = (nx - 1) * dx, (ny - 1) * dx
    w = 1e15 * lx * ly / n
    g = _gen(seed)
    return dx, w, [(q, m) + _maxwell(g, n, lx, ly, math.sqrt(2 * T * QE / m))
                   for q, m, T in ((-QE, ME, 2.0), (QE, M_AR, 0.03))]


def _slab(case, seed):
    nx, ny, n = case["nx"], case["ny"], case["np"]
    dx, w, species = _slab_inputs(case, seed)
    ctx = device.Context(nx, ny, dx, dx)
    sids = []
    for q, m, x, v in species:
        s = ctx.species_create(q, m, w, n)
        ctx.set_boundary(s, _lib.BND_DISCARD, _lib.BND_WRAP)
        ctx.upload(s, _host(x), _host(v))
        sids.append(s)
    ctx.poisson_create(EPS0)
    ctx.apply_periodic(1)
    left, right = _columns(nx, ny)
    ctx.apply_dirichlet(left, 0.0)
    ctx.apply_dirichlet(right, 100.0)
    if case["tracker"]:
        ctx.tracker_create(_lib.SURF_PERIODIC)
        block = np.zeros((nx, ny), bool)
        block[nx // 2 - nx // 16:nx // 2 + nx // 16, ny // 2 - ny // 16:ny // 2 + ny // 16] = True
        ctx.tracker_add_surface(block, _lib.SURF_REFLECT)
    return {"ctx": ctx, "sids": sids, "rec": _record(nx, ny)}


def _slab_run(case, s):
    ctx = s["ctx"]
    ctx.step(1e-11, case["steps"], seed=1, rtol=1e-8)
    return {"phi": _read(ctx, s["rec"], _lib.FIELD_PHI), "rho": _read(ctx, s["rec"], _lib.FIELD_RHO),
            "E": _read(ctx, s["rec"], _lib.FIELD_E), "absorbed": [ctx.absorbed(k)[:2] for k in s["sids"]]}


# ---- host arrays in, steps, host arrays out ------------------------------------
def _round_trip(case, seed):
    nx, ny, n = case["nx"], case["ny"], case["np"]
    dx, w, species = _slab_inputs(case, seed)
    ctx = device.Context(nx, ny, dx, dx)
    ctx.poisson_create(EPS0)
    ctx.apply_periodic(1)
    left, right = _columns(nx, ny)
    ctx.apply_dirichlet(left, 0.0)
    ctx.apply_dirichlet(right, 100.0)
    st = {"ctx": ctx, "sp": []}
    for q, m, x, v in species:
        s = ctx.species_create(q, m, w, n)
        ctx.set_boundary(s, _lib.BND_WRAP, _lib.BND_WRAP)
        src = (_pinned((n, 2)), _pinned((n, 3)))
        src[0][...], src[1][...] = _host(x), _host(v)
        st["sp"].append((s, src, (_pinned((n, 2)), _pinned((n, 3)), _pinned((n,), torch.int32).view(np.uint32)),
                         torch.empty((5, n), device="cuda")))
    return st


def _round_trip_run(case, st):
    ctx = st["ctx"]
    for s, (x, v), _, _ in st["sp"]:
        ctx.upload(s, x, v)
    ctx.step(1e-11, case["steps"], seed=1, rtol=1e-8)
    out = []
    for s, _, buf, by_id in st["sp"]:
        x, v, ids = (torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a.T).cuda(non_blocking=True)
                     for a in ctx.download(s, out=buf))
        # particles come back in storage order: put them in the caller's
        by_id[:, ids.long() - 1] = torch.cat([x, v]).float()
        out.append(by_id)
    return out


# ---- a solve by itself -----------------------------------------------------------
def _poisson_masks(case):
    nx, ny = case["nx"], case["ny"]
    blob = np.zeros((nx, ny), bool)
    blob[nx // 3:nx // 3 + 5, ny // 2:ny // 2 + 4] = True
    wall = np.zeros((nx, ny), bool)
    if case["open"]:
        wall[:, 0] = True
    else:
        wall[0, :] = True
    return blob, wall


def _poisson_rhs(case, seed):
    return torch.randn((2, case["ny"], case["nx"]), generator=_gen(seed), device="cuda", dtype=torch.float64) * 1e-6


def _poisson(case, seed):
    nx, ny, dx = case["nx"], case["ny"], 1e-3
    ctx = device.Context(nx, ny, dx, dx)
    ctx.poisson_create(EPS0)
    blob, wall = _poisson_masks(case)
    if not case["open"]:
        ctx.apply_periodic(1)
    ctx.apply_dirichlet(blob, -20.0)
    ctx.apply_dirichlet(wall, 0.0)
    return {"ctx": ctx, "f": [f.T for f in _poisson_rhs(case, seed).cpu().numpy()], "rec": _record(nx, ny)}


def _poisson_run(case, s):
    phi = [s["ctx"].solve_host(f, rtol=1e-11, maxit=2000)[0] for f in s["f"]]
    return {"phi": phi, "E": _read(s["ctx"], s["rec"], _lib.FIELD_E)}


# ---- DSMC --------------------------------------------------------------------------
def _dsmc(case, seed):
    n, npart, dh = case["n"], case["np"], 0.05
    m_o = 8 * 1.67262192e-27
    ctx = device.Context(n, n, dh, dh)
    g = _gen(seed)
    L = (n - 1) * dh
    sids = []
    for q, m, vth in ((-QE, ME, 0.5e6), (0.0, m_o, math.sqrt(2 * KB * 300 / m_o))):
        s = ctx.species_create(q, m, 1.0, 2 * npart)
        x, v = _maxwell(g, npart, L, L, vth)
        ctx.upload(s, _host(x), _host(v))
        sids.append(s)
    k = ctx.dsmc_create(sids[0], sids[1], [3e6, 4e6, 5e6, 6e6], [0.01, 0.1, 2.0, 0.01])
    return {"ctx": ctx, "k": k, "sids": sids, "seed": seed, "step": 0,
            "v": [np.empty((npart, 3), np.float32, order="F") for _ in sids]}


def _dsmc_run(case, s):
    ctx = s["ctx"]
    for _ in range(case["performs"]):
        s["step"] += 1
        ctx.dsmc_perform(s["k"], case["dt"], seed=s["seed"], step=s["step"])
    remaining, nu = ctx.dsmc_state(s["k"])
    for sid, by_id in zip(s["sids"], s["v"]):
        _, v, ids = ctx.download(sid)
        at = ids.astype(np.int64) - 1
        for d in range(3):
            by_id[at, d] = v[:, d]
    return {"remaining": remaining, "nu": nu, "v": s["v"]}


# ---- the warm-start network -----------------------------------------------------------
_LAYERS = [(1, 32)] + 6 * [(32, 32)] + [(32, 1)]  # (input, output) channels of its 3x3 convolutions


def _network_inputs(case, seed):
    g = _gen(seed)
    w = torch.cat([torch.randn(9 * a * b, generator=g, device="cuda") * math.sqrt(2.0 / (9 * a)) for a, b in _LAYERS])
    img = torch.randn((case["ny"], case["nx"]), generator=g, device="cuda")
    return w, img, 0.1 * torch.randn((case["ny"], case["nx"]), generator=g, device="cuda")


def _network(case, seed):
    ctx = device.Context(case["nx"], case["ny"], 1e-4, 1e-4)
    ctx.lws_create(0, seed=1)
    w, img, target = (t.cpu().numpy() for t in _network_inputs(case, seed))
    ctx.lws_weights(w)
    return {"ctx": ctx, "img": img, "target": target}


def _network_run(case, s):
    y = s["ctx"].lws_forward(s["img"])
    loss, grad = s["ctx"].lws_loss_grad(s["img"], s["target"])
    return {"y": y, "loss": np.float32(loss), "grad": grad}


_KINDS = {"two_stream": (_two_stream, _two_stream_run), "boundaries": (_boundaries, _boundaries_run),
          "discharge": (_discharge, _discharge_run), "ensemble": (_ensemble, _ensemble_run),
          "discharge_2d": (_discharge_2d, _discharge_2d_run), "slab": (_slab, _slab_run),
          "round_trip": (_round_trip, _round_trip_run), "poisson": (_poisson, _poisson_run),
          "dsmc": (_dsmc, _dsmc_run), "network": (_network, _network_run)}


def prepare(case, seed):
    s = _KINDS[case["kind"]][0](case, seed)
    s["case"] = case
    return s


def run(state):
    case = state["case"]
    return _KINDS[case["kind"]][1](case, state)


# ---- what a pass cannot do without ------------------------------------------------------
def work(case):
    k = case["kind"]
    if k == "poisson":
        nn = case["nx"] * case["ny"]
        return {"bytes": 2 * 32.0 * nn, "flops": 2 * 40.0 * nn * math.log2(nn)}
    if k == "network":
        px = case["nx"] * case["ny"]
        # multiply-adds of the full, half, quarter and eighth resolution layers
        macs = 9 * (2 * 32 + 32 * 32 * (1 + 2 * (1 / 4 + 1 / 16) + 1 / 64)) * px
        return {"bytes": 4.0 * 4 * px, "flops": 2.0 * macs * 4}  # evaluation, forward, two backward products
    if k == "dsmc":
        npart, n = case["np"], case["n"]
        pairs = npart * (npart / (n - 1) ** 2) * case["dt"] / 0.05 ** 2 * 1e7  # selected per pass over the cells
        return {"bytes": 48.0 * 2 * npart * case["performs"], "flops": 40.0 * pairs * case["performs"]}
    nn = {"two_stream": lambda: case["nx"] * 2, "boundaries": lambda: case["n"] ** 2,
          "discharge": lambda: case["nx"] * 2, "ensemble": lambda: case["runs"] * case["nx"] * 2,
          "discharge_2d": lambda: case["n"] ** 2, "slab": lambda: case["nx"] * case["ny"],
          "round_trip": lambda: case["nx"] * case["ny"]}[k]()
    if k == "ensemble":
        npart = case["runs"] * (case["np_lo"] + case["np_hi"])
    else:
        npart = case["np"] * (1 if k in ("two_stream", "boundaries") else 2)
    steps = case["steps"]
    # a step reads and writes each particle (24 B each way) and each node's charge, potential and field
    b = steps * (48.0 * npart + 32.0 * nn)
    if k == "round_trip":
        b += 2 * 40.0 * npart
    return {"bytes": b, "flops": steps * (60.0 * npart + 20.0 * nn * math.log2(max(nn, 2)))}


# ---- FP64 values --------------------------------------------------------------------------
class _Pic:
    """The collisionless step in FP64 torch: gather, kick, move, walls, deposit, Poisson, field."""

    def __init__(self, nx, ny, dx, species, walls_x, volume_walls, v_right=0.0, background=0.0):
        self.nx, self.ny, self.dx = nx, ny, dx
        self.species, self.walls_x, self.v_right, self.background = species, walls_x, v_right, background
        self.absorbed = [[0, 0] for _ in species]
        vol = torch.full((nx, ny), dx * dx, device="cuda", dtype=torch.float64)
        if volume_walls:
            for k in (0, -1):
                vol[k, :] *= 0.5
                vol[:, k] *= 0.5
        self.vol = vol
        self.E = torch.zeros((2, nx, ny), device="cuda", dtype=torch.float64)

    def _cells(self, x):
        f = x / self.dx
        i = f[0].floor().clamp(0, self.nx - 2)
        j = f[1].floor().clamp(0, self.ny - 2)
        hx, hy = f[0] - i, f[1] - j
        k = (i * self.ny + j).long()
        return [(k, (1 - hx) * (1 - hy)), (k + self.ny, hx * (1 - hy)), (k + 1, (1 - hx) * hy),
                (k + self.ny + 1, hx * hy)]

    def step(self, dt):
        nx, ny, dx = self.nx, self.ny, self.dx
        rho = torch.full((nx, ny), float(self.background), device="cuda", dtype=torch.float64)
        for s, (q, m, w, x, v) in enumerate(self.species):
            cw = self._cells(x)
            for d in range(2):
                Ef = self.E[d].reshape(-1)
                v[d] += (q / m * dt) * sum(wt * Ef[k] for k, wt in cw)
            x = x + v[:2] * dt
            lx, ly = (nx - 1) * dx, (ny - 1) * dx
            if self.walls_x == "discard":
                low, high = x[0] < 0, x[0] >= lx
                self.absorbed[s][0] += int(low.sum())
                self.absorbed[s][1] += int(high.sum())
                keep = ~(low | high)
                x, v = x[:, keep], v[:, keep]
            else:
                x[0] = torch.remainder(x[0], lx)
            x[1] = torch.remainder(x[1], ly)
            self.species[s] = (q, m, w, x, v)
            n = torch.zeros(nx * ny, device="cuda", dtype=torch.float64)
            for k, wt in self._cells(x):
                n.index_add_(0, k, wt)
            rho += q * w * n.reshape(nx, ny) / self.vol
        self.rho = rho
        self.phi = self._solve(-rho / EPS0)
        p = self.phi
        E = torch.empty_like(self.E)
        E[0, 1:-1] = (p[:-2] - p[2:]) / (2 * dx)
        E[0, 0], E[0, -1] = (p[0] - p[1]) / dx, (p[-2] - p[-1]) / dx
        E[1, :, 1:-1] = (p[:, :-2] - p[:, 2:]) / (2 * dx)
        E[1, :, 0], E[1, :, -1] = (p[:, 0] - p[:, 1]) / dx, (p[:, -2] - p[:, -1]) / dx
        self.E = E

    def _solve(self, b):
        nx, ny, h2 = self.nx, self.ny, self.dx ** 2
        ly = 2 * torch.cos(2 * math.pi * torch.arange(ny // 2 + 1, device="cuda", dtype=torch.float64) / ny) - 2
        if self.walls_x == "periodic":  # a ring in x too: the mean-zero potential
            lx = 2 * torch.cos(2 * math.pi * torch.arange(nx, device="cuda", dtype=torch.float64) / nx) - 2
            s = torch.fft.rfft2(b)
            lam = (lx[:, None] + ly[None, :]) / h2
            lam[0, 0] = 1.0
            s = s / lam
            s[0, 0] = 0.0
            return torch.fft.irfft2(s, s=(nx, ny))
        s = torch.fft.rfft(b, dim=1) * h2
        s[0], s[-1] = 0.0, 0.0
        s[-1, 0] = self.v_right * ny
        d, c = ly - 2.0, [torch.zeros_like(ly)]
        y = [s[0]]
        for i in range(1, nx - 1):  # Thomas along x, all modes at once
            f = 1.0 / (d - c[-1])
            c.append(f)
            y.append((s[i] - y[-1]) * f)
        out = torch.empty_like(s)
        out[-1] = s[-1]
        out[0] = s[0]
        for i in range(nx - 2, 0, -1):
            out[i] = y[i] - c[i] * out[i + 1]
        return torch.fft.irfft(out, n=ny, dim=1)


def _exact_two_stream(case, seed):
    dx, x, v, w = _two_stream_inputs(case, seed)
    p = _Pic(case["nx"], 2, dx, [(-QE, ME, w, x, v)], "periodic", False, background=QE * 2e11)
    for _ in range(case["steps"]):
        p.step(2e-9)
    return p.E.permute(1, 2, 0)


def _exact_slab(case, seed, walls="discard"):
    dx, w, species = _slab_inputs(case, seed)
    p = _Pic(case["nx"], case["ny"], dx, [(q, m, w, x, v) for q, m, x, v in species], walls, True, v_right=100.0)
    for _ in range(case["steps"]):
        p.step(1e-11)
    return p


def _exact_poisson(case, seed):
    """Conjugate gradients in FP64 on the five-point operator with its fixed nodes."""
    nx, ny, dx = case["nx"], case["ny"], 1e-3
    blob, wall = (torch.from_numpy(m).cuda() for m in _poisson_masks(case))
    fixed = blob | wall
    free = (~fixed).double()
    phi0 = torch.where(wall, 0.0, torch.where(blob, -20.0, 0.0)).double()

    def lap(p):  # minus the graph Laplacian (open sides have no neighbour), times dx^2
        q = torch.zeros_like(p)
        q[1:] += p[1:] - p[:-1]
        q[:-1] += p[:-1] - p[1:]
        q[:, 1:] += p[:, 1:] - p[:, :-1]
        q[:, :-1] += p[:, :-1] - p[:, 1:]
        if not case["open"]:
            q[:, 0] += p[:, 0] - p[:, -1]
            q[:, -1] += p[:, -1] - p[:, 0]
        return q

    def solve(f):
        r = free * (-f.T * (dx * dx / EPS0) - lap(phi0))
        x, p, rr = torch.zeros_like(r), r.clone(), (r * r).sum()
        stop = float(rr) * 1e-28
        for it in range(20000):
            ap = free * lap(p)
            a = rr / (p * ap).sum()
            x += a * p
            r -= a * ap
            new = (r * r).sum()
            p = r + (new / rr) * p
            rr = new
            if it % 100 == 99 and float(rr) <= stop:
                break
        return phi0 + x

    both = [solve(f) for f in _poisson_rhs(case, seed)]
    phi = both[1]
    E = torch.empty((nx, ny, 2), device="cuda", dtype=torch.float64)
    E[1:-1, :, 0] = (phi[:-2] - phi[2:]) / (2 * dx)
    E[0, :, 0], E[-1, :, 0] = (phi[0] - phi[1]) / dx, (phi[-2] - phi[-1]) / dx
    E[:, 1:-1, 1] = (phi[:, :-2] - phi[:, 2:]) / (2 * dx)
    E[:, 0, 1], E[:, -1, 1] = (phi[:, 0] - phi[:, 1]) / dx, (phi[:, -2] - phi[:, -1]) / dx
    return {"phi": both, "E": E}


def _exact_network(case, seed):
    w, img, target = (t.double() for t in _network_inputs(case, seed))
    w.requires_grad_(True)
    ws, at = [], 0
    for a, b in _LAYERS:
        k = w[at:at + 9 * a * b]
        at += 9 * a * b
        ws.append(k.reshape(3, 3, b, a).permute(2, 3, 0, 1))
    conv = lambda t, k: torch.nn.functional.conv2d(t, k, padding=1)
    pool = lambda t: torch.nn.functional.avg_pool2d(t, 2)
    up = lambda t: t.repeat_interleave(2, 2).repeat_interleave(2, 3)
    a = [torch.relu(conv(img[None, None], ws[0]))]
    for level in (1, 2, 3):
        a.append(torch.relu(conv(pool(a[-1]), ws[level])))
    t = a[3]
    for level in (2, 1, 0):
        t = torch.relu(conv(up(t) + a[level], ws[6 - level]))
    y = conv(t, ws[7])[0, 0]
    loss = ((y - target) ** 2).mean()
    loss.backward()
    return {"y": y.detach(), "loss": loss.detach(), "grad": w.grad}


def exact(case, seed):
    k = case["kind"]
    if k == "two_stream":
        return _exact_two_stream(case, seed)
    if k == "slab" and not case["tracker"]:
        p = _exact_slab(case, seed)
        return {"phi": p.phi, "rho": p.rho, "E": p.E.permute(1, 2, 0), "absorbed": p.absorbed}
    if k == "round_trip":
        p = _exact_slab(case, seed, "wrap")
        return [torch.cat([x, v]) for _, _, _, x, v in p.species]
    if k == "poisson":
        return _exact_poisson(case, seed)
    if k == "network":
        return _exact_network(case, seed)
    return None  # random collisions, or surfaces that particles are followed to
