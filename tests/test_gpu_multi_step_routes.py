"""Which kernels the steps of one call take (the multi-step kernel of meshes that fit the GPU at once, or one launch
per step), and that what was picked earlier never outlives what it was picked for."""
import numpy as np
import pytest

from samoa_gb300 import swe
from tests.helpers import omp_state, oracle_params
from tests.test_gpu_multi_step import _compare, _grid

pytestmark = pytest.mark.gpu


def _context(g, cfg):
    ctx = swe.SweContext()
    ctx.set_params(cfg.params())
    ctx.upload_mesh(g.mesh)
    ctx.upload_state(g.h, g.hu, g.hv, g.b)
    ctx.set_time(g.r_time, g.r_dt)
    return ctx


def test_graph_replayed_after_parameters_the_multi_step_kernel_does_not_take(swe_lib, oracle_lib):
    """Cell volumes that are no normal numbers (a scaling of 1e-155) need the step kernel's minimum over the cells;
    a graph captured before they were set must not go on with the multi-step kernel's maximum."""
    g, cfg = _grid(9, 1, "fwave", "slip")
    ctx = _context(g, cfg)
    try:
        ctx.traverse_graph(4)
        ctx.synchronize()
        for scaling in (1e-155, 1.0):
            cfg.scaling = scaling
            g.r_dt = scaling * swe.initial_dt(g.mesh, g.h, g.hu, g.hv, g.b, 0.2)
            S, P = omp_state(g.mesh, g), oracle_params(cfg)
            ctx.set_params(cfg.params())
            ctx.upload_state(g.h, g.hu, g.hv, g.b)
            ctx.set_time(0.0, g.r_dt)
            S.steps(P, 4)
            ctx.traverse_graph(4)
            ctx.synchronize()
            _compare(ctx, S, "scaling %g" % scaling)
    finally:
        ctx.close()


@pytest.mark.parametrize("solver", ["fwave", "aug_riemann", "llfbath"])
@pytest.mark.parametrize("log2,discs", [(1, 0), (9, 1), (13, 1), (16, 1), (17, 1)])
def test_many_steps_of_a_small_mesh_are_one_launch(swe_lib, log2, discs, solver):
    g, cfg = _grid(log2, discs, solver, "slip")
    ctx = _context(g, cfg)
    try:
        assert [ctx.launch_count(n) for n in (0, 1, 2, 4096, 4097)] == [0, 1, 1, 1, 2]
        ctx.set_cross_pass("inkernel")
        assert ctx.launch_count(8) == 8
        ctx.set_cross_pass("pass")
        assert ctx.launch_count(8) == 8 * ctx.task_counts()["launches_per_step"]
    finally:
        ctx.close()


def test_many_steps_of_a_large_mesh_are_a_launch_each(swe_lib):
    g, cfg = _grid(19, 0, "fwave", "slip")
    ctx = _context(g, cfg)
    try:
        assert ctx.launch_count(8) == 8
    finally:
        ctx.close()
