"""The measured cases: what a user of this framework runs, through its public entry points.

A case is a dict of plain values:

  kind      the entry point: "steps" (time steps on the device-resident state), "dropin" (the traversal
            object on a host grid), "host" (the step on pinned host arrays), "handoff" (mesh and state up,
            one step, flags and state back, as after a remesh), "ensemble" (independent grids, one CUDA
            graph of steps), "reverse" (one step of the discrete adjoint), "gradient" (a checkpointed
            gauge-misfit gradient)
  water     the scenario: "dam" (radial dam break), "shore" (a wave on a beach), "bowl" (parabolic
            bowl with a shore line), "basin" (ocean basin, mostly at rest), "current" (water moving everywhere)
  solver, boundary, log2 (2^log2 cells), discs (local refinements: ragged sizes and mixed depths), steps
"""
import functools
import math

import numpy as np
import torch

from samoa_gb300 import _lib, adjoint, swe

G = 9.80665
DEV = "cuda"


# ---------------------------------------------------------------------------------------------- the cases
def _case(name, kind, water, solver, boundary, log2, discs, steps):
    return dict(name=name, kind=kind, water=water, solver=solver, boundary=boundary, log2=log2, discs=discs,
                steps=steps)


def listed():
    return [
        # the smallest call: a host code steps its own small grid, one traversal per call (latency)
        _case("dropin-dam-4k", "dropin", "dam", "fwave", "slip", 12, 0, 1),
        # a coarse time loop on the device: launches and the latency of one step count
        _case("steps-bowl-4k", "steps", "bowl", "fwave", "outflow", 12, 0, 40),
        # the plain dam break at its usual size, reflecting walls
        _case("steps-dam-64k", "steps", "dam", "fwave", "slip", 16, 0, 20),
        # a locally refined wet/dry grid (ragged size, several depths) with the augmented solver
        _case("steps-bowl-aug-ragged", "steps", "bowl", "aug_riemann", "outflow", 17, 2, 10),
        # the flux of the reference's smoke runs, on a beach: half the cells are dry land
        _case("steps-shore-llfbath-512k", "steps", "shore", "llfbath", "outflow", 19, 0, 10),
        # the large wet/dry case: water moves in every wet cell
        _case("steps-bowl-4m", "steps", "bowl", "fwave", "outflow", 22, 0, 4),
        # a large ocean basin: a source in water otherwise at rest
        _case("steps-basin-16m", "steps", "basin", "fwave", "outflow", 24, 0, 4),
        # a host that keeps the state in its own (pinned) arrays
        _case("host-bowl-1m", "host", "bowl", "fwave", "outflow", 20, 0, 1),
        # the loop around a remesh: mesh and state up, a step, flags and state back
        _case("handoff-bowl-aug-ragged", "handoff", "bowl", "aug_riemann", "outflow", 16, 2, 1),
        # independent scenarios of uneven sizes, stepped together in a CUDA graph
        _case("ensemble-bowls-8-16", "ensemble", "bowl", "fwave", "outflow", 16, 0, 10),
        # one reverse step of the discrete adjoint in moving water
        _case("reverse-current-256k", "reverse", "current", "fwave", "outflow", 18, 0, 1),
        # an inversion's whole gradient: forward, checkpoints and reverse sweep
        _case("gradient-basin-64k", "gradient", "basin", "fwave", "outflow", 16, 0, 24),
    ]


def draw(rng):
    kind = rng.choice(["steps", "steps", "steps", "steps", "dropin", "host", "handoff", "ensemble", "reverse",
                       "gradient"])
    top = {"steps": 21, "dropin": 16, "host": 20, "handoff": 17, "ensemble": 15, "reverse": 18, "gradient": 15}[kind]
    log2 = rng.randint(9, top)
    discs = rng.randint(0, 2) if kind not in ("ensemble",) and log2 < 20 else 0
    solver = rng.choice(["fwave", "fwave", "aug_riemann", "llfbath"])
    if kind == "gradient":
        solver = "fwave"
    water = rng.choice(["dam", "shore", "bowl", "basin", "current"])
    if kind in ("ensemble",):
        water = "bowl"
    if kind in ("reverse", "gradient"):
        water = rng.choice(["basin", "current"])
    steps = {"steps": rng.randint(2, 5) if log2 > 19 else rng.randint(5, 20), "ensemble": 2 * rng.randint(2, 8),
             "gradient": rng.randint(8, 24)}.get(kind, 1)
    return {k: v for k, v in _case("", kind, water, solver, rng.choice(["outflow", "slip", "noslip"]), log2, discs,
                                   steps).items() if k != "name"}


def _sizes(case):
    """Sizes (log2) of an ensemble's instances: four of each from 2^(log2 - 8) to 2^log2 cells."""
    return [k for k in range(case["log2"] - 8, case["log2"] + 1) for _ in range(4)]


def work(case):
    # a step reads h, hu, hv, b and writes h, hu, hv; the flux of an edge and the update of a cell take about
    # 150 operations per cell (f-wave, LLF) or 400 (augmented); the reverse step reads the cotangents and the
    # branch byte too and writes the cotangents and b's; a gradient is a forward and a reverse step per step
    n = sum(1 << k for k in _sizes(case)) if case["kind"] == "ensemble" else _size(case["log2"], case["discs"])
    flops = 400.0 if case["solver"] == "aug_riemann" else 150.0
    k = case["steps"]
    byt = {"dropin": 57.0, "host": 49.0, "handoff": 57.0, "reverse": 97.0, "gradient": 153.0}.get(case["kind"], 56.0)
    fl = {"reverse": 2.5, "gradient": 3.5}.get(case["kind"], 1.0) * flops
    return {"bytes": byt * n * k, "flops": fl * n * k}


# ------------------------------------------------------------------------------------ meshes and scenarios
@functools.lru_cache(maxsize=12)
def _mesh(log2, discs):
    """2^log2 cells; each disc refines the cells within a smaller circle once (with the closure that keeps
    the mesh conforming), so that sizes are ragged and depths mixed."""
    mesh = swe.uniform_mesh(log2 - 1)
    for i in range(discs):
        r = np.hypot(mesh.centroids[:, 0] - 0.43, mesh.centroids[:, 1] - 0.57)
        mesh, _ = swe.adapt(mesh, (r < 0.21 / (i + 1)).astype(np.int8))
    return mesh


def _size(log2, discs):
    return _mesh(log2, discs).n_cells if discs else 1 << log2


def _config(case, log2):
    wide = {"basin": 1.0e6, "current": 1.0e5, "shore": 10.0}.get(case["water"], 1.0)
    return swe.Config(flux_solver=case["solver"], boundary=case["boundary"], courant_number=0.45,
                      dry_tolerance=1e-3 if case["water"] == "bowl" else 0.01, scaling=wide,
                      offset=(-0.5 * wide, -0.5 * wide), i_min_depth=max(0, log2 - 3), i_max_depth=log2 + 2)


def _fields(case, mesh, seed):
    """(h, hu, hv, b) on the GPU at the cells' centroids; h is the surface."""
    rng = np.random.default_rng(seed)
    c = torch.from_numpy(mesh.centroids).to(DEV) - 0.5
    x, y = c[:, 0], c[:, 1]
    x0, y0, amp, width = (float(v) for v in rng.uniform((-0.1, -0.1, 0.5, 0.05), (0.1, 0.1, 2.0, 0.1)))
    r2 = (x - x0) ** 2 + (y - y0) ** 2
    bump = amp * torch.exp(-r2 / (2 * width * width))
    relief = sum(float(a) * torch.sin(6.3 * (float(i) * x + float(j) * y) + float(p))
                 for a, i, j, p in rng.uniform((0.1, -5, -5, 0), (0.3, 5, 5, 6.3), (6, 4)))
    zero = torch.zeros_like(x)
    if case["water"] == "dam":
        b = torch.full_like(x, -10.0)
        return b + torch.where(r2 < (2 * width) ** 2, 10.0 + 2.5 * amp, 10.0), zero, zero, b
    if case["water"] == "shore":
        b = 12.0 * (x - x0)
        return torch.where(b < bump, bump, b), zero, zero, b
    if case["water"] == "bowl":
        b = -10.0 * (1.0 - (x * x + y * y) / 0.16)
        return torch.where(b < bump, bump, b), zero, zero, b
    if case["water"] == "basin":
        b = -4000.0 + 1975.0 * (1.0 + torch.tanh((x - 0.25) / 0.05)) + 300.0 * relief
        near = r2 < 0.15 ** 2  # the source lifts a patch; the rest of the surface is flat
        source = torch.where(near, 2.0 * amp * torch.exp(-r2 / (2 * 0.02 ** 2)), 0.0)
        return source, zero, zero, torch.clamp(b, max=-20.0)
    b = -100.0 + 10.0 * relief
    return 0.5 * bump, (bump * 0.5 - b) * 2.0, (bump * 0.5 - b) * 1.0, b


def _first_dt(case, mesh, cfg, h, hu, hv, b):
    d = h - b
    wet = d > cfg.dry_tolerance
    s = torch.where(wet, torch.sqrt(G * d.clamp(min=0)) + torch.sqrt(hu * hu + hv * hv) / torch.where(wet, d, 1.0), 0.0)
    leg, hyp, vol = _lengths(mesh, cfg)
    return float(cfg.courant_number * (vol / ((hyp + 2 * leg) * s).clamp(min=1e-30)).min())


def _host(fields):
    return [f.cpu().numpy() for f in fields]


class _Memory:
    """A device array of a context, for torch (no copy); a tensor made from it keeps the context."""

    def __init__(self, ctx, ptr, n):
        self.ctx = ctx
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f8", "data": (ptr, False), "version": 2}


def _state_of(ctx, n, views):
    ptrs = tuple(ctx.device_state()[:3])
    if ptrs not in views:
        views[ptrs] = [torch.as_tensor(_Memory(ctx, p, n), device=DEV) for p in ptrs]
    return views[ptrs]


@functools.lru_cache(maxsize=1)
def _stream():
    """The one stream that a program's contexts work on."""
    return torch.cuda.Stream()


def _vp(t):
    return adjoint.C.c_void_p(t.data_ptr())


# --------------------------------------------------------------------------------------------- one pass
class _State:
    """What a program keeps between passes."""

    def __init__(self, **kw):
        self.__dict__.update(kw)


def _ensemble_inputs(case, seed):
    meshes, cfgs, fields, dts = [], [], [], []
    for i, k in enumerate(_sizes(case)):
        mesh = _mesh(k, 0)
        cfg = _config(case, k)
        f = _fields(case, mesh, 1000 * seed + i)
        meshes.append(mesh)
        cfgs.append(cfg)
        fields.append(f)
        dts.append(_first_dt(case, mesh, cfg, *f))
    return meshes, cfgs, fields, dts


def _inputs(case, seed):
    mesh = _mesh(case["log2"], case["discs"])
    cfg = _config(case, case["log2"])
    f = _fields(case, mesh, seed)
    return mesh, cfg, f, _first_dt(case, mesh, cfg, *f)


def _cotangents(n, seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return torch.randn((3, n), dtype=torch.float64, device=DEV, generator=g)


def _gauges(case, n, seed):
    rng = np.random.default_rng(seed)
    return np.sort(rng.choice(n, 32, replace=False)), 0.1 * rng.normal(size=(case["steps"], 32))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        meshes, cfgs, fields, dts = _ensemble_inputs(case, seed)
        ctx = swe.SweEnsemble(0)
        stream = _stream()
        ctx.set_stream(stream.cuda_stream)
        ctx.upload_meshes(meshes)
        ctx.set_params_list([c.params() for c in cfgs])
        ctx.upload_state(*(np.concatenate([_host([f[q]])[0] for f in fields]) for q in range(4)))
        n = ctx.n_cells  # all sizes are even: no padding between the instances
        views = {}
        with torch.cuda.stream(stream):
            start = [v.clone() for v in _state_of(ctx, n, views)]
        return _State(kind=kind, ctx=ctx, stream=stream, start=start, views=views, n=n, steps=case["steps"],
                      zeros=np.zeros(len(dts)), dts=np.array(dts))
    mesh, cfg, f, dt = _inputs(case, seed)
    n = mesh.n_cells
    if kind == "dropin":
        trav = swe.SweEulerTimestepTraversal(cfg)
        grid = swe.Grid(mesh, *(a.copy() for a in _host(f)))
        return _State(kind=kind, trav=trav, grid=grid, start=_host(f), dt=dt)
    if kind == "gradient":
        gauges, obs = _gauges(case, n, seed)
        P = adjoint.GaugeProblem(mesh, cfg.params(), gauges, obs, np.full(case["steps"], dt), snapshots=6)
        h, _, _, b = _host(f)
        return _State(kind=kind, P=P, h=h, b=b)
    ctx = swe.SweContext(0)
    stream = _stream()
    ctx.set_stream(stream.cuda_stream)
    ctx.set_params(cfg.params())
    if kind == "handoff":
        ctx.upload_mesh(mesh)
        return _State(kind=kind, ctx=ctx, mesh=mesh, start=_host(f), dt=dt, stream=stream)
    ctx.upload_mesh(mesh)
    ctx.upload_state(*_host(f))
    ctx.set_time(0.0, dt)
    if kind == "host":
        pinned = [t.cpu().pin_memory() for t in f[:3]]
        out = [torch.empty(n, dtype=torch.float64).pin_memory() for _ in range(3)]
        return _State(kind=kind, ctx=ctx, ins=pinned, out=out, flags=torch.empty(n, dtype=torch.int8).pin_memory(),
                      stream=stream)
    views = {}
    with torch.cuda.stream(stream):
        start = [v.clone() for v in _state_of(ctx, n, views)]
        if kind == "reverse":
            ctx.set_dt_sequence([dt])
            branch = torch.empty((n + 1) & ~1, dtype=torch.uint8, device=DEV)
            _lib.check(ctx.L.swe_traverse_branches(ctx.ptr, 1, _vp(branch), branch.numel()))
            _lib.check(ctx.L.swe_snapshot_restore(ctx.ptr, *(_vp(s) for s in start), 0))
            out = torch.empty((4, n), dtype=torch.float64, device=DEV)
            return _State(kind=kind, ctx=ctx, branch=branch, lam=_cotangents(n, seed), out=out, stream=stream)
    return _State(kind=kind, ctx=ctx, start=start, views=views, n=n, steps=case["steps"], stream=stream)


def run(s):
    if s.kind == "steps":  # from the same state again, as a program that tries several futures does
        _lib.check(s.ctx.L.swe_snapshot_restore(s.ctx.ptr, *(_vp(q) for q in s.start), 0))
        s.ctx.traverse(s.steps)
        return _state_of(s.ctx, s.n, s.views)
    if s.kind == "dropin":
        g = s.grid
        for a, a0 in zip((g.h, g.hu, g.hv, g.b), s.start):
            a[:] = a0
        g.r_time, g.r_dt = 0.0, s.dt
        g.mark_dirty()
        s.trav.traverse(g)
        return {"h": g.h, "hu": g.hu, "hv": g.hv, "dt": g.r_dt, "flags": g.refinement,
                "refined": g.i_refinements_issued}
    if s.kind == "host":
        s.ctx.step_host(*s.ins, None, *s.out, s.flags)
        s.ctx.synchronize()
        return [*s.out, s.flags]
    if s.kind == "handoff":
        s.ctx.upload_mesh(s.mesh)
        s.ctx.upload_state(*s.start)
        s.ctx.set_time(0.0, s.dt)
        s.ctx.traverse(1)
        flags, count = s.ctx.refinements()
        return [*s.ctx.download_state()[:3], flags, count, s.ctx.get_time()[1]]
    if s.kind == "ensemble":
        with torch.cuda.stream(s.stream):
            for v, v0 in zip(_state_of(s.ctx, s.n, s.views), s.start):
                v.copy_(v0)
        s.ctx.set_times(s.zeros, s.dts)
        s.ctx.traverse_graph(s.steps)
        return _state_of(s.ctx, s.n, s.views)
    if s.kind == "reverse":
        with torch.cuda.stream(s.stream):
            s.out[3].zero_()
        _lib.check(s.ctx.L.swe_adjoint_step(s.ctx.ptr, _vp(s.branch), *(_vp(s.lam[q]) for q in range(3)),
                                            *(_vp(s.out[q]) for q in range(4))))
        return s.out
    J, gh, gb = s.P.gradient(s.h, s.b)
    return [J, gh, gb]


# ------------------------------------------------- the same steps in plain torch, 64 bits, differentiable
def _lengths(mesh, cfg):
    d = torch.from_numpy(mesh.depth.astype(np.float64)).to(DEV)
    return cfg.scaling * 2.0 ** (-0.5 * d), cfg.scaling * 2.0 ** (-0.5 * (d - 1)), cfg.scaling ** 2 * 0.5 ** (d + 1)


@functools.lru_cache(maxsize=1)
def _normal_table():
    """Outward normals of the three edges (right leg, hypotenuse, left leg) by orientation, -8..8."""
    out = np.zeros((17, 3, 2))
    for p in range(-8, 9):
        a = math.pi / 4 * abs(p)
        m = [[math.cos(a), -math.sin(a)], [math.sin(a), math.cos(a)]]
        if p < 0:
            m = [[-math.sin(a), math.cos(a)], [math.cos(a), math.sin(a)]]  # reflected
        if p:
            n = np.array([[-1.0, 0.0], [1.0, 1.0], [0.0, -1.0]]) @ np.linalg.inv(np.trunc(1.5 * np.array(m)))
            out[p + 8] = np.where(np.abs(n) < 1e-9, 0.0, n)
            out[p + 8] /= np.sqrt((out[p + 8] ** 2).sum(1, keepdims=True))
    return out


def _root(x):
    ok = x > 0
    return torch.where(ok, torch.sqrt(torch.where(ok, x, 1.0)), 0.0)


def _ratio(a, b):
    return a / torch.where(b != 0, b, 1.0)


def _pick(c, a, b):
    return torch.where(c, a, b)


def _mid_state(hL, hR, uL, uR, dry):
    """Middle depth and the two shock or rarefaction speeds of the Riemann problem (one Newton step)."""
    lo, hi = _pick(hR < hL, hR, hL), _pick(hL < hR, hR, hL)
    du = uR - uL
    cL, cR, clo, chi = _root(G * hL), _root(G * hR), _root(G * lo), _root(G * hi)
    Fmin = du + 2.0 * (clo - chi)
    Fmax = du + (hi - lo) * _root(_ratio((0.5 * G) * (hi + lo), hi * lo))
    t = (-du + 2.0 * (cL + cR)).clamp(min=0)
    hm1 = (1.0 / (16.0 * G)) * (t * t)
    iL, iR, ihi, ilo = _ratio(1.0, hL), _ratio(1.0, hR), _ratio(1.0, hi), _ratio(1.0, lo)
    gL, gR = _root((0.5 * G) * (ihi + iL)), _root((0.5 * G) * (ihi + iR))
    F0 = (du + (hi - hL) * gL) + (hi - hR) * gR
    dF = ((gL - _ratio(G * (hi - hL), (4.0 * (hi * hi)) * gL)) + gR) - _ratio(G * (hi - hR), (4.0 * (hi * hi)) * gR)
    s = _root(hi)
    t = s - _ratio(F0, (2.0 * s) * dF)
    hm2 = t * t
    im = _ratio(1.0, hm2)
    u1 = uL - (hm2 - hL) * _root((0.5 * G) * (im + iL))
    u2 = uR + (hm2 - hR) * _root((0.5 * G) * (im + iR))
    F0 = Fmin + (lo - lo) * _root((0.5 * G) * (ilo + ilo))
    hm3 = lo - _ratio(F0, _ratio(Fmax - F0, hi - lo))
    c1, c2, c3 = _root(G * hm1), _root(G * hm2), _root(G * hm3)
    left = hR < hL
    s1 = _pick(Fmin > 0, (uL + 2.0 * cL) - 3.0 * c1, _pick(Fmax <= 0, u1 - c2, _pick(
        left, (uL + 2.0 * cL) - 3.0 * c3, (uR - 2.0 * cR) + c3)))
    s2 = _pick(Fmin > 0, (uR - 2.0 * cR) + 3.0 * c1, _pick(Fmax <= 0, u2 + c2, _pick(
        left, (uL + 2.0 * cL) - c3, (uR - 2.0 * cR) + 3.0 * c3)))
    hm = _pick(Fmin > 0, hm1, _pick(Fmax <= 0, hm2, hm3))
    none = lo <= dry
    sd = ((uR + uL) - 2.0 * cR) + 2.0 * cL
    return _pick(none, 0.0, hm), _pick(none, sd, s1), _pick(none, sd, s2)


def _f_waves(q):
    dhu = q.huR - q.huL
    dpd = q.dphi + ((0.5 * G) * (q.hR + q.hL)) * (q.bR - q.bL)
    D = q.s2 - q.s1
    b1, b2 = _ratio(q.s2 * dhu - dpd, D), _ratio(dpd - q.s1 * dhu, D)
    z = torch.zeros_like(b1)
    sw = [q.s1, 0.5 * (q.s1 + q.s2), q.s2]
    fw = [[b1, z, b2], [b1 * q.s1, z, b2 * q.s2], [b1 * q.vL, None, b2 * q.vR]]
    fw[2][1] = ((q.huR * q.vR - q.huL * q.vL) - fw[2][0]) - fw[2][2]
    return sw, fw


def _augmented(q):
    db = q.bR - q.bL
    _, s1m, s2m = _mid_state(q.hL, q.hR, q.uL, q.uR, q.dry)
    l0, l2 = _pick(q.s1 < s2m, q.s1, s2m), _pick(q.s2 > s1m, q.s2, s1m)
    D = l2 - l0
    hst = _ratio(((q.huL - q.huR) + l2 * q.hR) - l0 * q.hL, D).clamp(min=0)
    l1 = 0.5 * (l0 + l2)
    l1 = _pick(l1.abs() < 1e-20, 0.0, l1)
    ct = 1e-6
    ghb = G * (0.5 * (q.hL + q.hR)).clamp(min=0)
    sb = 0.25 * ((q.uL + q.uR) * (q.uL + q.uR)) - ghb
    st = (q.uL * q.uR).clamp(min=0) - ghb
    sonic = (sb.abs() <= ct) | (sb * st <= ct) | ((sb * l0) * l2 <= ct) | (torch.minimum(l0.abs(), l2.abs()) < ct)
    sonic |= ((l0 < 0) & (s1m > 0)) | ((l2 > 0) & (s2m < 0))
    sonic |= ((q.uL + q.cL) * (q.uR + q.cR) < 0) | ((q.uL - q.cL) * (q.uR - q.cR) < 0)
    num = db * ghb
    sbs = _pick(sonic, 1.0, sb)
    dh = _pick(sonic, -db, _ratio(num, sbs))
    dphi = _pick(sonic, -(ghb * db), -_ratio(num * st, sbs))
    hsd = hst * D
    A = (l0 < -ct) & (l2 > ct)
    B, Cc = ~A & (l0 >= ct), ~A & (l0 < ct) & (l2 <= -ct)
    hi = _pick(A, _ratio(hsd, l2), _pick(B, _ratio(hsd, l0), _pick(Cc, q.hR, dh)))
    lo = _pick(A, _ratio(hsd, l0), _pick(B, -q.hL, _pick(Cc, _ratio(hsd, l2), dh)))
    x = _pick(dh < hi, dh, hi)
    dh = _pick(A | B | Cc, _pick(x > lo, x, lo), dh)
    pl, pr = -(q.hL * db), -(q.hR * db)
    up, dn = G * _pick(pl > pr, pl, pr), G * _pick(pl < pr, pl, pr)
    y = _pick(dphi < up, dphi, up)
    dphi = _pick(y > dn, y, dn)
    d0, d1, d2 = (q.hR - q.hL) - dh, q.huR - q.huL, q.dphi - dphi
    det = l0 - l2
    r0, r2 = l0 * l0, l2 * l2
    b0, b2 = _ratio(d1 - d0 * l2, det), _ratio(d0 * l0 - d1, det)
    b1 = _ratio(((d1 * r2 - l2 * d2) - d0 * (l0 * r2 - l2 * r0)) + (l0 * d2 - d1 * r0), det)
    fw = [[b0 * l0, 0.0 * b1, b2 * l2], [b0 * r0, b1, b2 * r2], [(b0 * l0) * q.vL, None, (b2 * l2) * q.vR]]
    fw[2][1] = ((((q.hR * q.uR) * q.vR) - ((q.hL * q.uL) * q.vL)) - fw[2][0]) - fw[2][2]
    return [l0, l1, l2], fw


class _Bag:
    pass


def _geoclaw(core, n1, n2, L, R, dry):
    """Net updates (h, hu, hv) of the left and right cell and the largest speed."""
    q = _Bag()
    pL, pR = n1 * L[1] + n2 * L[2], n1 * R[1] + n2 * R[2]
    tL, tR = n1 * L[2] - n2 * L[1], n1 * R[2] - n2 * R[1]
    dL, dR = L[0] - L[3], R[0] - R[3]
    wL, wR = dL > dry, dR > dry
    z = torch.zeros_like(dL)
    q.dry = dry
    q.hL, q.hR = _pick(wL, dL, z), _pick(wR, dR, z)
    q.huL, q.huR = _pick(wL, pL, z), _pick(wR, pR, z)
    hvL, hvR = _pick(wL, tL, z), _pick(wR, tR, z)
    q.uL, q.uR, q.vL, q.vR = _ratio(q.huL, q.hL), _ratio(q.huR, q.hR), _ratio(hvL, q.hL), _ratio(hvR, q.hR)
    q.bL, q.bR = L[3], R[3]
    with torch.no_grad():
        mR, _, _ = _mid_state(q.hL, q.hL, q.uL, -q.uL, dry)
        mL, _, _ = _mid_state(q.hR, q.hR, -q.uR, q.uR, dry)
        wallR = ~wR & (torch.maximum(q.hL, mR) + q.bL < q.bR)
        wallL = wR & ~wL & (torch.maximum(q.hR, mL) + q.bR < q.bL)
        lowR = ~wR & ~wallR & (q.hL + q.bL < q.bR)
        lowL = wR & ~wL & ~wallL & (q.hR + q.bR < q.bL)
    q.hR, q.hL = _pick(wallR, q.hL, q.hR), _pick(wallL, q.hR, q.hL)
    q.huR, q.huL = _pick(wallR, -q.huL, q.huR), _pick(wallL, -q.huR, q.huL)
    q.bR, q.bL = _pick(wallR, q.bL, _pick(lowR, q.hL + q.bL, q.bR)), _pick(wallL, q.bR, _pick(lowL, q.hR + q.bR, q.bL))
    q.uR, q.uL = _pick(wallR, -q.uL, q.uR), _pick(wallL, -q.uR, q.uL)
    q.vR, q.vL = _pick(wallR, q.vL, q.vR), _pick(wallL, q.vR, q.vL)
    hs, db = q.hR + q.hL, q.bR - q.bL
    q.dphi = (((q.huR - q.huL) * (q.uL + q.uR) - (q.uL * q.uR) * (q.hR - q.hL)) +
              ((0.5 * G) * (((q.bR + q.hR) - q.bL) - q.hL)) * hs) - ((0.5 * G) * hs) * db
    q.cL, q.cR = _root(G * q.hL), _root(G * q.hR)
    roe = _ratio(q.cL * q.uL + q.cR * q.uR, q.cR + q.cL)
    ch = _root((0.5 * G) * hs)
    left, right = q.uL - q.cL, q.uR + q.cR
    q.s1, q.s2 = _pick(left < roe - ch, left, roe - ch), _pick(right > roe + ch, right, roe + ch)
    sw, fw = core(q)
    for w, wall in enumerate((wallL, wallL | wallR, wallR)):
        sw[w] = _pick(wall, z, sw[w])
        for e in range(3):
            fw[e][w] = _pick(wall, z, fw[e][w])
    on = wL | wR
    nl, nr = [], []
    for e in range(3):
        a = c = z
        for w in range(3):
            neg, pos = sw[w] < 0, sw[w] > 0
            f = fw[e][w]
            a = a + _pick(neg, f, _pick(pos, z, 0.5 * f))
            c = c + _pick(pos, f, _pick(neg, z, 0.5 * f))
        nl.append(_pick(on, a, z))
        nr.append(_pick(on, c, z))
    s = _pick(on, torch.maximum(torch.maximum(sw[0].abs(), sw[1].abs()), sw[2].abs()), z)
    return ((nl[0], nl[1] * n1 - nl[2] * n2, nl[1] * n2 + nl[2] * n1, s),
            (nr[0], nr[1] * n1 - nr[2] * n2, nr[1] * n2 + nr[2] * n1, s))


def _llf_bath(n1, n2, L, R, dry):
    dL, dR = L[0] - L[3], R[0] - R[3]
    offL, offR = dL < dry, dR < dry
    z = torch.zeros_like(dL)
    hL, hR = dL.clamp(min=0), dR.clamp(min=0)
    sdL, sdR = _pick(offL, 1.0, dL), _pick(offR, 1.0, dR)
    vL, vR = n1 * (L[1] / sdL) + n2 * (L[2] / sdL), n1 * (R[1] / sdR) + n2 * (R[2] / sdR)
    sL, sR = _root(G * hL) + vL.abs(), _root(G * hR) + vR.abs()
    al = _pick(sL > sR, sL, sR)
    F = 0.5 * ((hL * vL + hR * vR) + al * (L[0] - R[0]))
    pr = (0.5 * G) * (hL * hL + hR * hR)
    src = ((0.25 * G) * (hL + hR)) * (R[3] - L[3])
    a, b = [F], [-F]
    for i, n in ((1, n1), (2, n2)):
        f = 0.5 * (((L[i] * vL + R[i] * vR) + pr * n) + al * (L[i] - R[i]))
        gL = ((0.5 * vL) * L[i] + (((0.5 * G) * hL) * hL) * n) + (0.5 * sL) * L[i]
        gR = (-((0.5 * vR) * R[i]) - (((0.5 * G) * hR) * hR) * n) + (0.5 * sR) * R[i]
        a.append(_pick(offL, z, _pick(offR, gL, f + src * n)))
        b.append(_pick(offR, z, _pick(offL, gR, -f + src * n)))
    a[0], b[0] = _pick(offL | offR, z, a[0]), _pick(offL | offR, z, b[0])
    a.append(_pick(offL, z, sL))
    b.append(_pick(offR, z, sR))
    return a, b


class _Steps:
    """Time steps on a mesh in plain torch; on odd steps an edge's other cell is the left one."""

    def __init__(self, mesh, cfg):
        up = lambda a: torch.from_numpy(np.ascontiguousarray(a).astype(np.int64)).to(DEV)  # noqa: E731
        self.cfg, self.n = cfg, mesh.n_cells
        lo = mesh.edge_cells[:, 0] < mesh.edge_cells[:, 1]
        ec = np.where(lo[:, None], mesh.edge_cells, mesh.edge_cells[:, ::-1])
        el = np.where(lo[:, None], mesh.edge_local, mesh.edge_local[:, ::-1])
        table = torch.from_numpy(_normal_table()).to(DEV)
        p = up(mesh.plotter) + 8
        self.c = [up(ec[:, 0]), up(ec[:, 1])]
        self.l = [up(el[:, 0]) - 1, up(el[:, 1]) - 1]
        self.normal = [table[p[c], k] for c, k in zip(self.c, self.l)]
        self.bc, self.bk = up(mesh.bnd_cell), up(mesh.bnd_local) - 1
        self.bn = table[p[self.bc], self.bk]
        self.leg, self.hyp, self.vol = _lengths(mesh, cfg)
        if cfg.flux_solver == "llfbath":
            self.flux = _llf_bath
        else:
            core = _f_waves if cfg.flux_solver == "fwave" else _augmented
            self.flux = lambda *a: _geoclaw(core, *a)

    def step(self, x, b, dt, k):
        """The state after a step of dt and the next dt."""
        cfg, odd = self.cfg, k & 1
        L, R, nn = self.c[odd], self.c[1 - odd], self.normal[odd]
        q = [*x, b]
        fL, fR = self.flux(nn[:, 0], nn[:, 1], [v[L] for v in q], [v[R] for v in q], cfg.dry_tolerance)
        own = [v[self.bc] for v in q]
        n1, n2 = self.bn[:, 0], self.bn[:, 1]
        ghost = list(own)
        if cfg.boundary == "slip":
            d = own[1] * n1 + own[2] * n2
            ghost[1], ghost[2] = own[1] - d * n1, own[2] - d * n2
        elif cfg.boundary == "noslip":
            ghost[1], ghost[2] = -own[1], -own[2]
        fB, _ = self.flux(n1, n2, own, ghost, cfg.dry_tolerance)
        at = torch.cat([L * 3 + self.l[odd], R * 3 + self.l[1 - odd], self.bc * 3 + self.bk])
        first = 2 if odd else 0
        sums = []
        for e in range(4):
            s = torch.zeros(3 * self.n, dtype=torch.float64, device=DEV)
            s = s.index_add(0, at, torch.cat([fL[e], fR[e], fB[e]])).view(-1, 3)
            sums.append((self.leg * s[:, first] + self.hyp * s[:, 1]) + self.leg * s[:, 2 - first])
        new = (self.vol / sums[3].detach().clamp(min=1e-300)).min()
        dh, du, dv = ((-dt / self.vol) * s for s in sums[:3])
        floor = b + cfg.dry_tolerance
        flood = (x[0] < floor) & (dh > 0)
        z = torch.zeros_like(b)
        h = _pick(flood, floor, x[0]) + dh
        u, v = _pick(flood, z, x[1]) + du, _pick(flood, z, x[2]) + dv
        dried = h < floor
        x = [_pick(dried, _pick(b < 0, b, z), h), _pick(dried, z, u), _pick(dried, z, v)]
        return x, cfg.courant_number * float(new)


def _forward(mesh, cfg, f, dt, steps):
    with torch.no_grad():
        S, x = _Steps(mesh, cfg), list(f[:3])
        for k in range(steps):
            x, dt = S.step(x, f[3], dt, k)
    return x, dt


def _pull(S, x, b, dt, k, lam):
    x = [v.detach().requires_grad_(True) for v in x]
    b = b.detach().requires_grad_(True)
    out, _ = S.step(x, b, dt, k)
    return torch.autograd.grad(out, [*x, b], list(lam))


def exact(case, seed):
    kind, steps = case["kind"], case["steps"]
    if kind == "ensemble":
        xs = [_forward(m, c, f, dt, steps)[0] for m, c, f, dt in zip(*_ensemble_inputs(case, seed))]
        return [torch.cat([x[q] for x in xs]) for q in range(3)]
    mesh, cfg, f, dt = _inputs(case, seed)
    if kind == "reverse":
        S = _Steps(mesh, cfg)
        return torch.stack(_pull(S, f[:3], f[3], dt, 0, _cotangents(mesh.n_cells, seed)))
    if kind == "gradient":
        gauges, obs = _gauges(case, mesh.n_cells, seed)
        gauges, obs = torch.from_numpy(gauges).to(DEV), torch.from_numpy(obs).to(DEV)
        S = _Steps(mesh, cfg)
        xs = [[f[0], torch.zeros_like(f[0]), torch.zeros_like(f[0])]]  # the run starts at rest
        with torch.no_grad():
            for k in range(steps):
                xs.append(S.step(xs[-1], f[3], dt, k)[0])
        miss = [xs[k + 1][0][gauges] - obs[k] for k in range(steps)]
        lam, gb = [torch.zeros_like(f[0]) for _ in range(3)], torch.zeros_like(f[0])
        for k in range(steps - 1, -1, -1):
            lam[0] = lam[0].index_add(0, gauges, 2.0 * miss[k])
            *lam, g = _pull(S, xs[k], f[3], dt, k, lam)
            gb = gb + g
        return [float(sum((m * m).sum() for m in miss)), lam[0], gb]
    x, dt = _forward(mesh, cfg, f, dt, steps)
    if kind == "steps":
        return x
    if kind == "dropin":
        h, hu, hv = _host(x)
        return {"h": h, "hu": hu, "hv": hv, "dt": dt, "flags": None, "refined": None}
    x = _host(x)
    return [*x, None] if kind == "host" else [*x, None, None, dt]
