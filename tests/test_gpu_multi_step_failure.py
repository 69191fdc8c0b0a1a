"""The multi-step kernel's waits between its CTAs run out (an injection makes them count one CTA too few, with a limit
of 20 ms), the wait between two steps or, in a run of one, that for the last: the call reports it, and the context
then steps like the oracle, refinement count included."""
import pytest

from samoa_gb300 import _lib
from tests.helpers import omp_state, oracle_params
from tests.test_gpu_multi_step import _compare, _grid
from tests.test_gpu_multi_step_routes import _context

pytestmark = pytest.mark.gpu

SWE_E_DEVICE = -6
NONE, MEETING, REFUSED_LAUNCH = 0, 2, 3


@pytest.mark.parametrize("steps", [2, 4, 1])
@pytest.mark.parametrize("log2,discs", [(5, 0), (12, 1), (16, 0)])
def test_meeting_runs_out_and_context_recovers(swe_lib, oracle_lib, log2, discs, steps):
    g, cfg = _grid(log2, discs, "fwave", "slip")
    cfg.i_max_depth = log2 + 12  # so that cells do ask for refinement
    L = _lib.load()
    ctx = _context(g, cfg)
    try:
        _lib.check(L.swe_set_fault_injection(ctx.ptr, MEETING))
        assert ctx.launch_count(steps) == 1
        ctx.traverse(steps)
        with pytest.raises(_lib.SweError) as err:
            ctx.synchronize()
        assert err.value.code == SWE_E_DEVICE and "ran out" in str(err.value)
        ctx.synchronize()  # reported once
        _lib.check(L.swe_set_fault_injection(ctx.ptr, NONE))
        ctx.upload_state(g.h, g.hu, g.hv, g.b)  # the time is still that of the state before the failed steps
        S, P = omp_state(g.mesh, g, parity=steps & 1), oracle_params(cfg)
        for n in (2, 3):
            S.steps(P, n)
            ctx.traverse(n)
            ctx.synchronize()
            _compare(ctx, S, "%d steps" % n)
            assert S.n_refine > 0
    finally:
        ctx.close()


@pytest.mark.parametrize("graph", [False, True])
def test_a_refused_launch_is_made_step_by_step(swe_lib, oracle_lib, graph):
    g, cfg = _grid(12, 1, "fwave", "slip")
    L = _lib.load()
    ctx = _context(g, cfg)
    try:
        _lib.check(L.swe_set_fault_injection(ctx.ptr, REFUSED_LAUNCH))
        S, P = omp_state(g.mesh, g), oracle_params(cfg)
        for n in (5, 4):
            S.steps(P, n)
            (ctx.traverse_graph if graph else ctx.traverse)(n)
            ctx.synchronize()
            _compare(ctx, S, "%d steps" % n)
        assert ctx.launch_count(4) == 4 and ctx.step_count() == 9
        _lib.check(L.swe_set_fault_injection(ctx.ptr, NONE))
        ctx.upload_mesh(g.mesh)
        assert ctx.launch_count(4) == 1
    finally:
        ctx.close()


def test_graphs_do_not_outlive_an_injection(swe_lib, oracle_lib):
    g, cfg = _grid(9, 0, "fwave", "slip")
    L = _lib.load()
    ctx = _context(g, cfg)
    try:
        _lib.check(L.swe_set_fault_injection(ctx.ptr, MEETING))
        ctx.traverse_graph(2)
        with pytest.raises(_lib.SweError):
            ctx.synchronize()
        ctx.upload_state(g.h, g.hu, g.hv, g.b)
        ctx.set_time(0.0, g.r_dt)
        _lib.check(L.swe_set_fault_injection(ctx.ptr, NONE))
        S, P = omp_state(g.mesh, g), oracle_params(cfg)
        S.steps(P, 2)
        ctx.traverse_graph(2)
        ctx.synchronize()
        _compare(ctx, S, "after the injection")
    finally:
        ctx.close()
