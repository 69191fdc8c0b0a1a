"""Mesh checks split over host threads (lists of 2^16 items and more) against meshes just below: valid meshes pass,
and of two broken edges the first in list order is the one reported."""
import ctypes as C

import numpy as np
import pytest

from samoa_gb300 import _lib, swe


def validate(m, edge_cells):
    p = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    a = [np.ascontiguousarray(x, t) for x, t in ((m.depth, np.int8), (m.plotter, np.int8), (edge_cells, np.int64),
                                                 (m.edge_local, np.int8), (m.bnd_cell, np.int64),
                                                 (m.bnd_local, np.int8))]
    return _lib.load().swe_mesh_validate(len(a[0]), p(a[0]), p(a[1]), len(edge_cells), p(a[2]), p(a[3]), len(a[4]),
                                         p(a[4]), p(a[5]))


@pytest.mark.parametrize("depth", [14, 15, 16])
def test_split_checks_report_the_first_bad_edge(swe_lib, depth):
    m = swe.uniform_mesh(depth)
    ec = np.array(m.edge_cells, np.int64).reshape(-1, 2)
    assert validate(m, ec) == 0
    for first in (0, len(ec) // 3, len(ec) - 2):
        bad = ec.copy()
        bad[[first, len(ec) - 1], 1] = m.n_cells
        assert validate(m, bad) == -1
        assert _lib.last_error().startswith("edge %d: cells" % first)
        twice = ec.copy()
        twice[first + 1] = twice[first]
        assert validate(m, twice) == -1
