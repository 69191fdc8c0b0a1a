"""The reverse step in segments of any length (block size and blocks per SM follow from it): the same gradients as
in short ones, bit for bit."""
import ctypes as C

import numpy as np
import pytest

from samoa_gb300 import _lib
from tests.test_gpu_multi_step import _grid
from tests.test_gpu_multi_step_routes import _context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solver", ["fwave", "aug_riemann", "lfbath", "llfbath"])
def test_reverse_step_in_long_segments(swe_lib, solver):
    import torch

    def vp(t):
        return C.c_void_p(t.data_ptr())
    g, cfg = _grid(13, 2, solver, "noslip")
    ctx = _context(g, cfg)
    n = g.mesh.n_cells
    lam = torch.from_numpy(np.random.default_rng(2).normal(size=(3, n))).cuda()
    got = {}
    try:
        for cells in (128, 460, 662, 688, 690, 704, 768, 1024, 1376):
            ctx.set_tiling(cells, 128)
            ctx.upload_state(g.h, g.hu, g.hv, g.b)
            ctx.set_dt_sequence(np.full(4, g.r_dt))
            first = ctx.step_count()
            out = torch.zeros((4, n), dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
            _lib.check(_lib.load().swe_adjoint_step(ctx.ptr, None, *[vp(x) for x in lam], *[vp(x) for x in out]))
            ctx.synchronize()
            got.setdefault(first & 1, {})[cells] = out.cpu().numpy()
        for by_parity in got.values():
            ref = by_parity[min(by_parity)]
            assert np.isfinite(ref).all() and np.abs(ref).max() > 0
            for cells, x in by_parity.items():
                assert np.array_equal(x, ref), cells
    finally:
        ctx.close()
