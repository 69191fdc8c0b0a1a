"""swe_gauge_gradient's buffers stay with the context: a gradient after one of another size, and giving them back."""
import numpy as np
import pytest

from samoa_gb300 import adjoint, scenarios

pytestmark = pytest.mark.gpu


def _case(log2, steps, gauges, seed):
    return scenarios.adjoint_case(log2_cells=log2, steps=steps, n_gauges=gauges, seed=seed)


def _problem(c, snapshots):
    return adjoint.GaugeProblem(c["mesh"], c["params"], c["gauges"], c["obs"], c["dts"], snapshots=snapshots)


def _gradient(P, c):
    J, gh, gb = P.gradient(c["h0"], c["b"])
    return J, gh.cpu().numpy(), gb.cpu().numpy()


def test_gradient_after_one_of_another_size(swe_lib):
    cases = [_case(10, 9, 3, 1), _case(13, 20, 40, 2), _case(6, 5, 1, 3), _case(13, 20, 40, 2), _case(10, 9, 3, 1)]
    want = []
    for c in cases:
        P = _problem(c, 4)
        try:
            want.append(_gradient(P, c))
        finally:
            P.close()
    P = _problem(cases[0], 4)
    try:
        for c, w in zip(cases, want):
            P.retarget(c["mesh"], c["gauges"], c["obs"], c["dts"])
            for _ in range(2):
                got = _gradient(P, c)
                assert got[0] == w[0] and np.array_equal(got[1], w[1]) and np.array_equal(got[2], w[2])
            P.ctx.set_dt_sequence(None)
    finally:
        P.close()


def test_kept_buffers_are_given_back(swe_lib):
    import torch
    c = _case(18, 3, 2, 1)
    P = _problem(c, 6)
    try:
        _gradient(P, c)
        kept = torch.cuda.mem_get_info()[0]
        P.ctx.set_dt_sequence(None)
        # six states of three fields, and two sets of cotangents
        assert torch.cuda.mem_get_info()[0] - kept >= (6 * 3 + 6) * 8 * c["mesh"].n_cells
        J, gh, gb = _gradient(P, c)
        assert np.isfinite(gh).all() and np.isfinite(J)
    finally:
        P.close()
