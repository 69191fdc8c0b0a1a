"""Tilings picked by mesh size and tilings at the limits of what swe_set_tiling and swe_set_staging take."""
import pytest

from samoa_gb300 import swe
from tests.helpers import omp_state, oracle_params
from tests.test_gpu_multi_step import _compare, _grid
from tests.test_gpu_multi_step_routes import _context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells,threads", [(1294, 256), (1298, 128), (1304, 128), (1304, 256)])
def test_longest_segments_with_two_staging_buffers(swe_lib, oracle_lib, cells, threads):
    g, cfg = _grid(12, 2, "fwave", "slip")
    ctx = _context(g, cfg)
    try:
        ctx.set_tiling(64, threads)
        ctx.set_staging(2)
        ctx.set_tiling(cells, threads)
        S, P = omp_state(g.mesh, g), oracle_params(cfg)
        for n in (1, 2):
            S.steps(P, n)
            ctx.traverse(n)
            ctx.synchronize()
            _compare(ctx, S, "%d cells" % cells)
        with pytest.raises(swe._lib.SweError):
            ctx.set_tiling(1306, threads)
    finally:
        ctx.close()
