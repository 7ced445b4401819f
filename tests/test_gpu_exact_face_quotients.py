"""The exact form's face states, where its quotients (products with a correctly
rounded reciprocal and remainders) change to plain divisions and where a sign
or a subnormal would show: bit for bit the C oracle's plain divisions."""
import ctypes

import numpy as np
import pytest

import oracle_bind as ob

pytestmark = pytest.mark.gpu

LOW, HIGH = 2.0 ** -664, 2.0 ** 199  # the corrected products' range (weno_plain)


def _near(x, rng, size):
    """x and its neighbours, a few units either way."""
    k = rng.integers(-3, 4, size=size)
    return (1.0 + k * 2.0 ** -52 * np.where(k < 0, 0.5, 1.0)) * x


def _stencils(kind, rng, n=3000):
    s = (n, 6, 4)
    sign = rng.choice([-1.0, 1.0], size=s)
    if kind == "random":
        v = rng.uniform(0.1, 3.0, size=s) * sign
    elif kind == "magnitudes":
        v = np.ldexp(rng.uniform(1, 2, size=s), rng.integers(-120, 40, size=s)) * sign
    elif kind == "low limit":      # one slot or more at the low end, some of them beyond it
        v = np.where(rng.uniform(size=s) < 0.5, _near(LOW, rng, s), rng.uniform(0.1, 3.0, size=s)) * sign
    elif kind == "all low":
        v = _near(LOW, rng, s) * sign
    elif kind == "high limit":     # (indicators of 2^398: their squares stay finite)
        v = np.where(rng.uniform(size=s) < 0.5, _near(HIGH, rng, s), rng.uniform(0.1, 3.0, size=s)) * sign
    elif kind == "all high":
        v = _near(HIGH, rng, s) * sign
    elif kind == "lone high":      # a weight 1e-320 of the others, and the only one that is not times 0
        v = np.zeros(s)
        v[np.arange(n), rng.integers(0, 6, n)] = np.ldexp(rng.uniform(1, 2, size=(n, 4)), rng.integers(150, 199, (n, 4)))
        v *= sign
    elif kind == "zeros":
        v = np.where(rng.uniform(size=s) < 0.6, 0.0, rng.uniform(0.1, 3.0, size=s)) * sign
    elif kind == "subnormals":
        v = rng.integers(0, 2 ** 20, size=s) * 2.0 ** -1074 * sign
    else:                          # multiples of 3 and 6, and one unit beside them
        v = _near(1.0, rng, s) * rng.integers(1, 2 ** 20, size=s) * 6 * sign
    return v


@pytest.mark.parametrize("eps", [1e-2, 1e-6, 1e-40])
@pytest.mark.parametrize("kind", ["random", "magnitudes", "low limit", "all low", "high limit", "all high", "lone high",
                                  "zeros", "subnormals", "sixths"])
def test_face_states_are_bitwise_plain_divisions(cfsb, kind, eps):
    rng = np.random.default_rng(sum(map(ord, kind)))
    st = _stencils(kind, rng)
    with cfsb.Solver(16, 16, precision=cfsb.FP64_EXACT, weno_eps=eps) as s:
        got = np.stack(s.weno5_faces(st))[:, :, :4]
    weno5 = ob.orc_lib().orc_weno5
    want = np.empty_like(got)
    for f in range(st.shape[0]):
        for v in range(4):
            x = np.ascontiguousarray(st[f, :, v])
            y = np.ascontiguousarray(x[::-1])
            want[0, f, v] = weno5(x.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), eps)
            want[1, f, v] = weno5(y.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), eps)
    assert np.all(np.isfinite(want))
    assert np.array_equal(got.view(np.uint64), want.view(np.uint64))  # signs of zeros too
