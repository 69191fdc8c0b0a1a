"""A dt sequence's buffer is kept for the next sequence: steps in flight on another stream still get their own."""
import numpy as np
import pytest

from samoa_gb300 import swe
from tests.test_gpu_multi_step import _grid
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
