"""Steps on a stream of a green context, which owns a part of the GPU's SMs: the multi-step kernel is taken only
where its blocks fit that part at once, and the results are the oracle's either way."""
import ctypes as C

import pytest

from tests.helpers import omp_state, oracle_params
from tests.test_gpu_multi_step import _compare, _grid
from tests.test_gpu_multi_step_routes import _context

pytestmark = pytest.mark.gpu

SM = 1  # CU_DEV_RESOURCE_TYPE_SM


@pytest.fixture
def green_stream():
    """A stream on 16 of the GPU's SMs."""
    import torch
    torch.cuda.init()
    torch.zeros(1, device="cuda")
    cu = C.CDLL("libcuda.so.1")
    if not hasattr(cu, "cuGreenCtxStreamCreate"):
        pytest.skip("a driver without green contexts")

    def ok(rc):
        assert rc == 0, "driver error %d" % rc
    whole, part = C.create_string_buffer(256), C.create_string_buffer(256)
    n, desc, green, stream = C.c_uint(1), C.c_void_p(), C.c_void_p(), C.c_void_p()
    ok(cu.cuDeviceGetDevResource(0, whole, SM))
    ok(cu.cuDevSmResourceSplitByCount(part, C.byref(n), whole, None, 0, 16))
    ok(cu.cuDevResourceGenerateDesc(C.byref(desc), part, 1))
    ok(cu.cuGreenCtxCreate(C.byref(green), desc, 0, 1))
    ok(cu.cuGreenCtxStreamCreate(C.byref(stream), green, 1, 0))
    yield stream.value
    ok(cu.cuStreamSynchronize(stream))
    ok(cu.cuStreamDestroy_v2(stream))
    ok(cu.cuGreenCtxDestroy(green))


@pytest.mark.parametrize("log2,fits", [(9, True), (16, False)])
def test_steps_on_a_part_of_the_gpu(swe_lib, oracle_lib, green_stream, log2, fits):
    g, cfg = _grid(log2, 0, "fwave", "slip")
    ctx = _context(g, cfg)
    try:
        assert ctx.launch_count(4) == 1
        ctx.set_stream(green_stream)
        assert ctx.launch_count(4) == (1 if fits else 4)
        S, P = omp_state(g.mesh, g), oracle_params(cfg)
        for steps in (ctx.traverse, ctx.traverse_graph):
            S.steps(P, 4)
            steps(4)
            ctx.synchronize()
            _compare(ctx, S, "green")
        ctx.set_stream(None)
        assert ctx.launch_count(4) == 1
    finally:
        ctx.close()
