"""Edge fluxes with a negative or NaN dry tolerance (the entry points without a context take any): a depth of zero
is then a wet one, whose velocity is 0 / 0, and a negative one has no root; what comes out has to be the oracle's."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O
from samoa_gb300 import _lib, swe

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tolerance", [-1.0, -0.0, float("nan")])
@pytest.mark.parametrize("solver", [swe.FWAVE, swe.AUG_RIEMANN, swe.LF_BATH, swe.LLF_BATH])
def test_any_tolerance(swe_lib, oracle_lib, solver, tolerance):
    rng = np.random.default_rng(3)
    n = 4096
    r = np.sqrt(0.5)
    normals = np.array([(1.0, 0.0), (0.0, -1.0), (r, r), (-r, r), (0.6, 0.8)])[rng.integers(0, 5, n)]
    q = []
    for _ in range(2):
        d = rng.choice([0.0, 0.5, 3.0, -0.25], n)
        p = rng.choice([0.0, -0.0, 1.5], (n, 2)) * (rng.random((n, 1)) < 0.5)
        b = rng.choice([0.0, -2.0], n)
        q.append(np.ascontiguousarray(np.column_stack([b + d, p, b])))
    got, want = np.zeros((2, n, 4)), np.zeros((2, n, 4))
    p = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    _lib.check(_lib.load().swe_riemann_batch(solver, n, p(np.ascontiguousarray(normals)), p(q[0]), p(q[1]), tolerance,
                                             p(got[0]), p(got[1])))
    for i in range(n):
        want[0, i], want[1, i] = O.edge_flux(solver, normals[i], q[0][i], q[1][i], tolerance)
    assert np.array_equal(got, want, equal_nan=True)


@pytest.mark.parametrize("solver", ["fwave", "aug_riemann", "lfbath", "llfbath"])
def test_any_tolerance_without_a_context(swe_lib, oracle_lib, solver):
    from tests.helpers import omp_state, oracle_params
    from tests.test_gpu_multi_step import _grid
    from tests.test_zz_no_alloc import _NoAlloc
    g, cfg = _grid(9, 1, solver, "slip")
    rng = np.random.default_rng(4)
    g.h = g.b + rng.choice([0.0, 0.5, 3.0], len(g.b), p=[0.01, 0.49, 0.5])
    g.hu = np.where(g.h > g.b, rng.choice([0.0, 1.5], len(g.b)), 0.0)
    cfg.dry_tolerance = -1.0
    S, P = omp_state(g.mesh, g), oracle_params(cfg)
    S.steps(P, 1)
    na = _NoAlloc(g.mesh, g)
    na.call(cfg.params(), g.r_dt, 0)
    assert np.isnan(S.h).any() and np.isfinite(S.h).any()
    for got, want in zip(na.out, (S.h, S.hu, S.hv)):
        assert np.array_equal(got.cpu().numpy(), want, equal_nan=True)
