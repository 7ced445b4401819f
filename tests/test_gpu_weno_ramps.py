"""FP32-mixed reconstruction on steep ramps and jumps (energies in SI units):
finite, and the FP64 form's values, in the interior and at Dirichlet sides."""
import importlib

import numpy as np
import pytest

cfsb = importlib.import_module("2d_compressible_flow_solver_b200")

pytestmark = pytest.mark.gpu


def _profile(n, slope, kind, rng):
    """A pressure that climbs and falls by about `slope` a cell, or jumps by it."""
    if kind == "jump":
        return slope * (1.0 + 7.0 * (rng.uniform(size=n // 4 + 1) > 0.5))[np.arange(n) // 4]
    d = slope * rng.uniform(0.5, 1.5, n // 2)
    up = np.concatenate([[0.0], np.cumsum(d)])
    return slope + np.concatenate([up, up[-2::-1]])[:n]


@pytest.mark.parametrize("bc", [0, 1, 2])
@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("kind,slope", [("ramp", 1e4), ("ramp", 2e4), ("ramp", 1e5), ("ramp", 1e6), ("jump", 1e4),
                                        ("jump", 1e6), ("jump", 1e9)])
def test_a_step_stays_finite_and_near_fp64(bc, axis, kind, slope):
    nx, ny = (64, 33) if axis == 0 else (33, 64)
    p = _profile(64, slope, kind, np.random.default_rng(3))
    p = np.broadcast_to(p[:, None] if axis == 0 else p[None, :], (nx, ny))
    U = np.stack([np.full((nx, ny), 1.2), np.zeros((nx, ny)), np.zeros((nx, ny)), p / 0.4])
    prim = [(1.2, 0.0, 0.0, 3.0 * slope)] * 4 if bc == 1 else None
    out, dt = {}, None
    for form in (cfsb.FP64, cfsb.FP32_MIXED):
        with cfsb.Solver(nx, ny, precision=form, rk=cfsb.RK_SSP3, hll=cfsb.HLL_DAVIS, bc=(bc,) * 4, bc_prim=prim) as s:
            s.set_state(U)
            dt = s.compute_dt(0.4) if dt is None else dt
            s.step(dt)
            out[form] = s.get_state()
    # three stages at a Courant number of 0.4, each a few roundings of 2^-24 of
    # the state and of fluxes of up to 5 times the state
    size = np.array([1.2, 1.2, 1.2, 1.0]) * np.sqrt([1.0, slope, slope, 1.0])
    size[3] = np.abs(U[3]).max()
    size[1:3] = np.sqrt(1.2 * p.max()) * 1.2
    err = np.abs(out[cfsb.FP32_MIXED] - out[cfsb.FP64]).max(axis=(1, 2)) / size
    assert np.all(np.isfinite(out[cfsb.FP32_MIXED]))
    assert err.max() < 4e-6


@pytest.mark.parametrize("slope", [1e3, 2e4, 1e6, 1e8])
def test_face_states_of_ramps(slope):
    rng = np.random.default_rng(4)
    st = np.cumsum(slope * rng.uniform(0.5, 1.5, size=(200, 6, 4)), axis=1).astype(np.float32).astype(np.float64)
    st[:, :, 0] = 1.0 + np.abs(st[:, :, 0])
    got = {}
    for form in (cfsb.FP64, cfsb.FP32_MIXED):
        with cfsb.Solver(16, 16, precision=form) as s:
            got[form] = np.stack(s.weno5_faces(st))[:, :, :4]
    assert np.all(np.isfinite(got[cfsb.FP32_MIXED]))
    # candidates of 11/6 + 7/6 + 1/3 of the stencil's largest value, each term rounded twice, weights to 10 roundings
    assert np.abs(got[cfsb.FP32_MIXED] - got[cfsb.FP64]).max() <= 40 * 2.0 ** -24 * np.abs(st).max()
