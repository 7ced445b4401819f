"""FP64 face states of the unit entry (the Dirichlet faces' reconstruction), bit
for bit the written operations: each fused multiply-add, product and the
division rounded once, as rational arithmetic rounds them."""
from fractions import Fraction as Q
import importlib

import numpy as np
import pytest

cfsb = importlib.import_module("2d_compressible_flow_solver_b200")

pytestmark = pytest.mark.gpu


def _fma(a, b, c):
    return float(Q(a) * Q(b) + Q(c))


def _weno5(v, eps):
    v0, v1, v2, v3, v4 = (float(x) for x in v)
    k13 = 13.0 / 12.0
    d = (_fma(-2.0, v1, v0) + v2, _fma(-2.0, v2, v1) + v3, _fma(-2.0, v3, v2) + v4)
    e = (_fma(3.0, v2, _fma(-4.0, v1, v0)), v1 - v3, _fma(3.0, v2, _fma(-4.0, v3, v4)))
    q = [eps + _fma(k13 * x, x, (0.25 * y) * y) for x, y in zip(d, e)]
    q0, q1, q2 = (x * x for x in q)
    a0, a1, a2 = (0.1 * q1) * q2, (0.6 * q0) * q2, (0.3 * q0) * q1
    p0 = _fma(11.0, v2, _fma(-7.0, v1, 2.0 * v0))
    p1 = _fma(2.0, v3, _fma(5.0, v2, -v1))
    p2 = _fma(5.0, v3, _fma(2.0, v2, -v4))
    return _fma(a0, p0, _fma(a1, p1, a2 * p2)) * (1.0 / (6.0 * (a0 + a1 + a2)))


@pytest.mark.parametrize("spread", [1e-6, 0.1, 3.0, 1e4])
def test_fp64_states_are_the_written_operations(spread):
    rng = np.random.default_rng(8)
    st = 1.0 + spread * rng.uniform(0, 1, size=(60, 6, 4))
    st[:10, :3] = st[:10, :1]  # a Dirichlet face's stencil: two values, three times each
    st[:10, 3:] = st[:10, 3:4]
    with cfsb.Solver(16, 16, precision=cfsb.FP64) as s:
        left, right = s.weno5_faces(st)
    for f in range(st.shape[0]):
        for v in range(4):
            x = st[f, :, v]
            assert left[f, v] == _weno5(x[:5], 1e-2)
            assert right[f, v] == _weno5(x[:0:-1], 1e-2)
