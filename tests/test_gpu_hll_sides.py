"""The throughput forms' HLL flux face by face, judged against each component of
the flux in more bits: flow running either way out of a state up to 1e4 times
the one beside it, supersonic, just subsonic and slow, and its mirror image."""
import importlib

import numpy as np
import pytest

cfsb = importlib.import_module("2d_compressible_flow_solver_b200")

pytestmark = pytest.mark.gpu
GAMMA = 1.4


def _faces(ratio, mach, rng, n=400):
    """Left and right states [n][4] (normal momentum in slot 1), values exact in FP32; the left one `ratio` times larger."""
    out = []
    for scale in (ratio, 1.0):
        rho, p = scale * rng.uniform(0.5, 2.0, n), scale * rng.uniform(0.5, 2.0, n)
        a = np.sqrt(GAMMA * p / rho)
        u, v = mach * a * rng.uniform(0.9, 1.1, n), 0.3 * a * rng.uniform(-1, 1, n)
        q = np.stack([rho, rho * u, rho * v, p / (GAMMA - 1) + 0.5 * rho * (u * u + v * v)], axis=1)
        out.append(q.astype(np.float32).astype(np.float64))
    return out


def _hll(L, R, H):
    """Flux through x-faces with Davis bounds in the type H, and the size of the terms that it is made of."""
    def side(q):
        r, mx, my, E = (np.asarray(x, H) for x in q.T)
        u, ke = mx / r, (mx * mx + my * my) / r / 2
        p, pm = H(GAMMA - 1) * (E - ke), H(GAMMA - 1) * (E + ke)
        au = np.abs(u)
        a = np.sqrt(H(GAMMA) * p / r)
        return (r, mx, my, E, u, p, a, np.stack([mx, mx * u + p, my * u, (E + p) * u]),
                np.stack([np.abs(mx), np.abs(mx) * au + pm, np.abs(my) * au, (E + pm) * au]))
    rL, mL, nL, EL, uL, pL, aL, FL, ML = side(L)
    rR, mR, nR, ER, uR, pR, aR, FR, MR = side(R)
    SL, SR = np.minimum(uL - aL, uR - aR), np.maximum(uL + aL, uR + aR)
    dU = np.stack([rR - rL, mR - mL, nR - nL, ER - EL])
    d = np.where(SR - SL > 0, SR - SL, 1)
    avg = (SL < 0) & (SR > 0)
    F = np.where(SL >= 0, FL, np.where(SR <= 0, FR, (SR * FL - SL * FR + SL * SR * dU) / d))
    # what rounding acts on: the terms of the average, and the derivative of
    # the average by the bounds, which carry roundings of |u| + a
    terms = (np.abs(SR) * ML + np.abs(SL) * MR + np.abs(SL * SR) * np.abs(dU)) / d
    speed = np.maximum(np.abs(uL) + aL, np.abs(uR) + aR)
    bounds = speed * (ML + MR + speed * np.abs(dU)) / d
    size = np.where(avg, terms + bounds, np.where(SL >= 0, ML, MR))
    return F, size, avg


@pytest.mark.parametrize("form,eps", [(cfsb.FP32_MIXED, 2.0 ** -23), (cfsb.FP64, 2.0 ** -52)])
@pytest.mark.parametrize("ratio", [1.0, 1e2, 1e4, 1e-2, 1e-4])
@pytest.mark.parametrize("mach", [-2.5, -0.95, -0.2, 0.2, 0.95, 2.5])
def test_each_component_to_a_few_roundings(form, eps, ratio, mach):
    # per component 6.5 units of the last place for a flux (reciprocal, kinetic
    # energy, pressure, product), 5.5 for a bound, 4 for weight and sums: 16
    L, R = _faces(ratio, mach, np.random.default_rng(5))
    with cfsb.Solver(16, 16, precision=form, hll=cfsb.HLL_DAVIS) as s:
        got = s.hll_faces(0, L, R).T
    F, size, avg = _hll(L, R, np.longdouble)
    assert np.all(np.abs(got - F) <= 16 * eps * size)
    if abs(mach) > 2:
        assert not avg.any()


@pytest.mark.parametrize("form", [cfsb.FP32_MIXED, cfsb.FP64])
@pytest.mark.parametrize("direction", [0, 1])
@pytest.mark.parametrize("ratio", [1.0, 1e4])
@pytest.mark.parametrize("mach", [-2.5, -0.95, -0.2, 0.2, 0.95, 2.5])
def test_the_mirrored_face_has_the_mirrored_flux(form, direction, ratio, mach):
    L, R = _faces(ratio, mach, np.random.default_rng(6))
    n = 1 + direction  # the normal momentum's slot
    if direction:
        L, R = L[:, [0, 2, 1, 3]], R[:, [0, 2, 1, 3]]
    flip = np.ones(4)
    flip[n] = -1.0
    with cfsb.Solver(16, 16, precision=form, hll=cfsb.HLL_DAVIS) as s:
        F = s.hll_faces(direction, L, R)
        G = s.hll_faces(direction, R * flip, L * flip)
    assert np.all(np.isfinite(F))
    assert np.array_equal(G, -F * flip)
