"""Many steps of one call on meshes that fit the GPU at once (the multi-step kernel) against the oracle, bit
for bit: one and few cells, one segment, several with a ragged last one, mixed depths, both parities of
the first step, time limits, ensembles whose instances have one or many segments, and graphs."""
import numpy as np
import pytest

from samoa_gb300 import scenarios, swe
from tests.helpers import assert_state_equal, omp_state, oracle_params

pytestmark = pytest.mark.gpu


def _grid(log2, discs, solver, boundary, seed=3):
    mesh = swe.uniform_mesh(log2 - 1)
    for i in range(discs):
        r = np.hypot(mesh.centroids[:, 0] - 0.4, mesh.centroids[:, 1] - 0.55)
        mesh, _ = swe.adapt(mesh, (r < 0.25 / (i + 1)).astype(np.int8))
    cfg = swe.Config(flux_solver=solver, boundary=boundary, courant_number=0.4, dry_tolerance=1e-3,
                     offset=(-0.5, -0.5), i_min_depth=max(0, log2 - 3), i_max_depth=log2 + 2)
    c = mesh.centroids - 0.5
    rng = np.random.default_rng(seed)
    b = -10.0 * (1.0 - (c ** 2).sum(1) / 0.16)
    eta = 1.5 * np.exp(-((c - rng.uniform(-0.1, 0.1, 2)) ** 2).sum(1) / 0.02)
    h = np.where(b < eta, eta, b)
    hu = np.where(h > b, rng.normal(0.0, 1.0, len(b)), 0.0)
    z = np.zeros(len(b))
    g = swe.Grid(mesh, h, hu, z, b, 0.0, 0.0)
    g.r_dt = swe.initial_dt(mesh, h, hu, z, b, 0.2)
    return g, cfg


def _compare(ctx, S, tag):
    h, hu, hv, _ = ctx.download_state()
    assert_state_equal(tag, h, hu, hv, S.h, S.hu, S.hv)
    flags, count = ctx.refinements()
    t, dt, dt_new = ctx.get_time()
    assert np.array_equal(flags, S.flags) and count == S.n_refine
    assert t == S.scal[0] and dt == S.scal[1] and dt_new == S.dt_new


@pytest.mark.parametrize("log2,discs,solver,boundary", [
    (1, 0, "fwave", "slip"), (2, 0, "aug_riemann", "outflow"), (6, 0, "fwave", "outflow"), (7, 0, "llfbath", "slip"),
    (7, 2, "fwave", "noslip"), (10, 2, "aug_riemann", "slip"), (12, 0, "fwave", "outflow"), (13, 1, "lfbath", "slip"),
    (14, 2, "fwave", "slip"), (16, 1, "fwave", "outflow"), (17, 1, "llfbath", "outflow")])
def test_many_steps_equal_the_oracle(swe_lib, oracle_lib, log2, discs, solver, boundary):
    g, cfg = _grid(log2, discs, solver, boundary)
    S, P = omp_state(g.mesh, g), oracle_params(cfg)
    ctx = swe.SweContext()
    try:
        ctx.set_params(cfg.params())
        ctx.upload_mesh(g.mesh)
        ctx.upload_state(g.h, g.hu, g.hv, g.b)
        ctx.set_time(0.0, g.r_dt)
        for n in (2, 1, 3, 8):  # from even and odd steps, alone and after single ones
            S.steps(P, n)
            ctx.traverse(n)
            ctx.synchronize()
            _compare(ctx, S, "%d steps" % n)
        assert ctx.step_count() == 14
        S.steps(P, 10)
        ctx.traverse_graph(5)
        ctx.traverse_graph(5)
        ctx.synchronize()
        _compare(ctx, S, "graph")
    finally:
        ctx.close()


def test_time_limits_and_dry_land(swe_lib, oracle_lib):
    g, cfg = _grid(9, 1, "fwave", "outflow")
    cfg.r_max_time, cfg.r_output_time_step = 0.7 * g.r_dt, 0.5 * g.r_dt
    for dry in (False, True):
        if dry:
            g.h = g.b + 1e-4
            g.hu[:] = 0.0
        S, P = omp_state(g.mesh, g), oracle_params(cfg)
        ctx = swe.SweContext()
        try:
            ctx.set_params(cfg.params())
            ctx.upload_mesh(g.mesh)
            ctx.upload_state(g.h, g.hu, g.hv, g.b)
            ctx.set_time(0.0, g.r_dt)
            S.steps(P, 6)
            ctx.traverse(6)
            ctx.synchronize()
            _compare(ctx, S, "dry" if dry else "limits")
        finally:
            ctx.close()


def test_uneven_instances(swe_lib, oracle_lib):
    made = [_grid(k, d, "fwave", "slip", seed=k) for k, d in ((1, 0), (5, 0), (11, 2), (6, 1), (9, 0), (2, 0))]
    grids, cfgs = [g for g, _ in made], [c for _, c in made]
    states = [omp_state(g.mesh, g) for g in grids]
    ens = swe.SweEnsemble()
    try:
        ens.upload_meshes([g.mesh for g in grids])
        ens.set_params_list([c.params() for c in cfgs])
        ens.upload_state(*(np.concatenate([getattr(g, q) for g in grids]) for q in ("h", "hu", "hv", "b")))
        ens.set_times([0.0] * len(grids), [g.r_dt for g in grids])
        for k in (3, 4):
            ens.traverse(k)
            for S, c in zip(states, cfgs):
                S.steps(oracle_params(c), k)
            h, hu, hv, _ = ens.download_state()
            flags, counts = ens.refinements_all()
            t, dt, dt_new = ens.get_times()
            for i, (S, x, y, z, f) in enumerate(zip(states, *(ens.split(a) for a in (h, hu, hv, flags)))):
                assert_state_equal("instance %d" % i, x, y, z, S.h, S.hu, S.hv)
                assert np.array_equal(f, S.flags) and counts[i] == S.n_refine
                assert (t[i], dt[i], dt_new[i]) == (S.scal[0], S.scal[1], S.dt_new)
    finally:
        ens.close()
