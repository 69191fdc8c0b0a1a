"""Tilings picked by mesh size and tilings at the limits of what swe_set_tiling and swe_set_staging take."""
import numpy as np
import pytest

from samoa_gb300 import swe
from tests.helpers import assert_state_equal, omp_state, oracle_params
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


@pytest.mark.parametrize("kind", ["uneven", "equal", "tiny", "many"])
def test_ensembles_that_fit_the_gpu_at_once(swe_lib, oracle_lib, kind):
    """Segments never span two instances, so each instance's last one is rounded up: the tiling picked for all of
    them still has to give at most two segments per SM (unless there are more instances than that)."""
    import torch
    made = {"uneven": [(k, 0) for k in (5, 6, 7, 8, 9, 10, 11, 12, 13) for _ in range(4)],
            "equal": [(13, 0)] * 9 + [(12, 1)], "tiny": [(6, 0)] * 200, "many": [(6, 0)] * 700}[kind]
    grids, cfgs = zip(*[_grid(k, d, "fwave", "slip", seed=i) for i, (k, d) in enumerate(made)])
    states = [omp_state(g.mesh, g) for g in grids]
    ens = swe.SweEnsemble()
    try:
        ens.upload_meshes([g.mesh for g in grids])
        resident = 2 * torch.cuda.get_device_properties(0).multi_processor_count
        fits = len(made) <= resident
        assert (ens.task_counts()["segments"] <= resident) == fits
        ens.set_params_list([c.params() for c in cfgs])
        ens.upload_state(*(np.concatenate([getattr(g, q) for g in grids]) for q in ("h", "hu", "hv", "b")))
        ens.set_times([0.0] * len(grids), [g.r_dt for g in grids])
        assert ens.launch_count(3) == (1 if fits else 3)
        ens.traverse(3)
        for S, c in zip(states, cfgs):
            S.steps(oracle_params(c), 3)
        h, hu, hv, _ = ens.download_state()
        for i, (S, x, y, z) in enumerate(zip(states, *(ens.split(a) for a in (h, hu, hv)))):
            assert_state_equal("instance %d" % i, x, y, z, S.h, S.hu, S.hv)
    finally:
        ens.close()


def test_threads_with_a_segment_length_of_the_callers(swe_lib):
    """128 threads unless they were set, whatever an earlier mesh's own tiling had picked."""
    g, cfg = _grid(16, 0, "fwave", "slip")
    ctx = _context(g, cfg)
    try:
        assert ctx.get_tiling()[1] == 256
        ctx.set_tiling(512)
        assert ctx.get_tiling() == (512, 128)
        ctx.upload_mesh(g.mesh)
        assert ctx.get_tiling() == (512, 128)
        ctx.set_tiling(0, 192)
        ctx.set_tiling(256)
        assert ctx.get_tiling() == (256, 192)
    finally:
        ctx.close()
