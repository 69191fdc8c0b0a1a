"""Edge fluxes with the mesh's own normals (axis-aligned and diagonal), whose products by 0, 1 and the
diagonal's component take paths of their own: bit for bit against the oracle, signs of zeros included."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O
from samoa_gb300 import _lib, swe

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solver", [swe.FWAVE, swe.AUG_RIEMANN, swe.LF_BATH, swe.LLF_BATH])
def test_fluxes_along_the_mesh_normals(swe_lib, oracle_lib, solver):
    rng = np.random.default_rng(5)
    n = 16384
    r = np.sqrt(0.5)
    kinds = np.array([(1, 0.0), (1, -0.0), (-1, 0.0), (-1, -0.0), (0.0, 1), (-0.0, 1), (0.0, -1), (-0.0, -1),
                      (r, r), (r, -r), (-r, r), (-r, -r)])
    normals = kinds[rng.integers(0, len(kinds), n)]
    bl = rng.uniform(-20, 5, n)
    br = np.where(rng.random(n) < 0.5, bl, bl + rng.uniform(-3, 3, n))
    dl, dr = (rng.choice([0.0, 1e-3, 1.0], n, p=[0.1, 0.05, 0.85]) * rng.uniform(0.0, 20, n) for _ in range(2))
    dr = np.where(rng.random(n) < 0.3, dl + (br - bl) * 0.0, dr)
    ql = np.stack([bl + dl, rng.normal(0, 30, n), rng.normal(0, 30, n), bl], 1)
    qr = np.stack([br + dr, rng.normal(0, 30, n), rng.normal(0, 30, n), br], 1)
    for q in (ql, qr):  # momenta of either zero, of a tiny and of a huge size
        for col in (1, 2):
            k = rng.integers(0, 10, n)
            q[k == 0, col] = 0.0
            q[k == 1, col] = -0.0
            q[(k == 2) & (rng.random(n) < 0.1), col] *= 1e-250
            q[(k == 3) & (rng.random(n) < 0.02), col] *= 1e160
    mirror = rng.random(n) < 0.1  # sums that cancel
    qr[mirror] = ql[mirror] * np.array([1.0, -1.0, -1.0, 1.0])
    gl, gr, ol, orr = (np.zeros((n, 4)) for _ in range(4))
    p = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    _lib.check(_lib.load().swe_riemann_batch(solver, n, p(np.ascontiguousarray(normals)), p(ql), p(qr), 1e-3, p(gl),
                                             p(gr)))
    for i in range(n):
        ol[i], orr[i] = O.edge_flux(solver, normals[i], ql[i], qr[i], 1e-3)
    ok = np.isfinite(ol).all(1) & np.isfinite(orr).all(1)
    assert ok.sum() > 0.9 * n
    assert np.array_equal(gl[ok].view(np.int64), ol[ok].view(np.int64))
    assert np.array_equal(gr[ok].view(np.int64), orr[ok].view(np.int64))
    assert np.array_equal(np.isfinite(gl).all(1) & np.isfinite(gr).all(1), ok)
