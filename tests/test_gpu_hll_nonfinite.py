"""HLL flux of a supersonic face whose downwind state is not finite (a vacuum,
an unfilled solid cell): the upwind flux, as in the exact form, and a NaN where
the upwind state itself is not finite."""
import importlib

import numpy as np
import pytest

cfsb = importlib.import_module("2d_compressible_flow_solver_b200")

pytestmark = pytest.mark.gpu

UPWIND = np.array([[1.0, 3.0, 0.25, 7.0], [0.5, 4.0, -1.0, 20.0]])  # (rho, rho un, rho ut, E), Mach 2 and more
DOWNWIND = [[0.0, 0.0, 0.0, 0.0], [0.0, 1.0, 0.0, 1.0], [np.nan] * 4, [1.0, 0.0, 0.0, -1.0], [-1.0, 2.0, 0.0, 1.0],
            [np.inf, 0.0, 0.0, 1.0], [1.0, np.inf, np.inf, np.inf]]  # of all of them the sound speed is a NaN


@pytest.mark.parametrize("form", [cfsb.FP32_MIXED, cfsb.FP64])
@pytest.mark.parametrize("direction", [0, 1])
@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("down", DOWNWIND)
def test_nothing_downwind_enters(form, direction, sign, down):
    n = 1 + direction

    def turned(q):
        q = np.array(q, dtype=float).reshape(-1, 4)
        q = q[:, [0, 2, 1, 3]] if direction else q.copy()
        q[:, n] *= sign
        return q

    up, dn = turned(UPWIND), np.repeat(turned(down), 2, axis=0)
    with cfsb.Solver(16, 16, precision=form, hll=cfsb.HLL_DAVIS) as s:
        got = s.hll_faces(direction, *((up, dn) if sign > 0 else (dn, up)))
        own = s.hll_faces(direction, up, up)  # of two equal states: the physical flux
    assert np.array_equal(got, own)


@pytest.mark.parametrize("form", [cfsb.FP32_MIXED, cfsb.FP64])
def test_a_nan_upwind_is_seen(form):
    up, dn = np.array([[np.nan] * 4]), np.array([[1.0, 0.1, 0.0, 2.5]])
    with cfsb.Solver(16, 16, precision=form, hll=cfsb.HLL_DAVIS) as s:
        assert np.isnan(s.hll_faces(0, up, dn)).all() and np.isnan(s.hll_faces(0, dn, up)).all()
