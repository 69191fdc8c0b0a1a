"""Steps around a dt sequence: in flight on another stream when the next sequence comes (its buffer is kept), across
the sequence's end, and after a gradient, which leaves its sequence set."""
import numpy as np
import pytest

from samoa_gb300 import _lib, adjoint, scenarios
from tests.helpers import assert_state_equal, omp_state, oracle_params
from tests.test_gpu_multi_step import _compare, _grid
from tests.test_gpu_multi_step_routes import _context

pytestmark = pytest.mark.gpu


def test_steps_in_flight_keep_their_sequence(swe_lib):
    import torch
    g, cfg = _grid(20, 0, "fwave", "slip")
    steps = 60
    dts = np.linspace(0.4, 0.8, steps) * g.r_dt
    states = []
    for change in (False, True):
        ctx = _context(g, cfg)
        try:
            streams = [torch.cuda.Stream() for _ in range(2)]
            ctx.set_stream(streams[0].cuda_stream)
            ctx.set_dt_sequence(dts)
            ctx.traverse(steps)
            if change:
                ctx.set_stream(streams[1].cuda_stream)
                ctx.set_dt_sequence(np.zeros(steps))
            torch.cuda.synchronize()
            ctx.synchronize()
            assert ctx.step_count() == steps
            states.append(np.stack(ctx.download_state()))
        finally:
            ctx.close()
    assert np.isfinite(states[0]).all() and not np.array_equal(states[0][0], g.h)
    assert np.array_equal(states[0], states[1])


def _oracle_steps(S, P, dts, n):
    """n steps of the oracle, the first ones with the given dt."""
    for k in range(n):
        if k < len(dts):
            S.scal[1] = dts[k]
        S.steps(P, 1)


@pytest.mark.parametrize("graph", [False, True])
def test_steps_across_the_end_of_a_sequence(swe_lib, oracle_lib, graph):
    g, cfg = _grid(11, 1, "fwave", "slip")
    dts = np.array([0.5, 0.3, 0.6]) * g.r_dt
    ctx = _context(g, cfg)
    try:
        ctx.set_dt_sequence(dts)
        S, P = omp_state(g.mesh, g), oracle_params(cfg)
        _oracle_steps(S, P, dts, 8)
        assert [ctx.launch_count(n) for n in (2, 3, 4, 8)] == [2, 3, 4, 4]
        (ctx.traverse_graph if graph else ctx.traverse)(8)
        ctx.synchronize()
        _compare(ctx, S, "across")
        assert ctx.launch_count(8) == 1
        S.steps(P, 8)
        (ctx.traverse_graph if graph else ctx.traverse)(8)
        ctx.synchronize()
        _compare(ctx, S, "after")
        # back into the sequence
        ctx.set_dt_sequence(None)
        ctx.upload_state(g.h, g.hu, g.hv, g.b)
        ctx.set_time(0.0, g.r_dt)
        ctx.set_dt_sequence(dts)
        ctx.traverse(2)
        _lib.check(_lib.load().swe_step_back(ctx.ptr))
        assert ctx.launch_count(8) == 3
        S = omp_state(g.mesh, g)
        _oracle_steps(S, P, dts, 9)
        ctx.traverse(8)
        ctx.synchronize()
        h, hu, hv, _ = ctx.download_state()
        assert_state_equal("back", h, hu, hv, S.h, S.hu, S.hv)
    finally:
        ctx.close()


def test_steps_after_a_gradient(swe_lib, oracle_lib):
    case = scenarios.adjoint_case(log2_cells=11, steps=6, n_gauges=4, seed=9)
    P = adjoint.GaugeProblem(case["mesh"], case["params"], case["gauges"], case["obs"], case["dts"], snapshots=3)
    try:
        P.gradient(case["h0"], case["b"])
        ctx = P.ctx
        assert ctx.launch_count(6) == 6 and ctx.launch_count(20) == 7
        ctx.traverse(20)
        ctx.synchronize()
        many = ctx.download_state() + list(ctx.get_time())
        P.gradient(case["h0"], case["b"])
        for _ in range(20):
            ctx.traverse(1)
        ctx.synchronize()
        single = ctx.download_state() + list(ctx.get_time())
        for x, y in zip(many, single):
            assert np.array_equal(x, y)
    finally:
        P.close()
