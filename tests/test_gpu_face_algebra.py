"""The throughput forms' WENO pair and HLL flux where their algebra has edges: flow
supersonic either way in each direction (the HLL weight at 0 and -1), jumps of
a large or small state, equal states, against the engine's exact form (the
reference's arithmetic)."""
import importlib

import numpy as np
import pytest

cfsb = importlib.import_module("2d_compressible_flow_solver_b200")
wl = importlib.import_module("2d_compressible_flow_solver_b200.workloads")

pytestmark = pytest.mark.gpu


def _state(nx, ny, u, v, jump, scale):
    rng = np.random.default_rng(7)
    q = 1.0 + jump * rng.uniform(0, 1, size=(4, 4))[np.arange(nx)[:, None] * 4 // nx, np.arange(ny)[None, :] * 4 // ny]
    p = scale * (1.0 + jump * rng.uniform(0, 1, size=(4, 4)))[np.arange(nx)[:, None] * 4 // nx, np.arange(ny)[None, :] * 4 // ny]
    c = np.sqrt(scale)
    return wl.conserved(q, c * u, c * v, p)


@pytest.mark.parametrize("hll", [cfsb.HLL_REFERENCE, cfsb.HLL_DAVIS])
@pytest.mark.parametrize("u,v", [(4.0, 0.3), (-4.0, -0.3), (0.2, 4.0), (-0.1, -4.0), (0.0, 0.0)])
@pytest.mark.parametrize("jump,scale", [(0.0, 1.0), (1e-3, 1.0), (1.0, 1.0), (1.0, 3e3)])
def test_one_step_against_the_exact_form(hll, u, v, jump, scale):
    nx, ny = 45, 61
    U = _state(nx, ny, u, v, jump, scale)
    size = np.abs(U).max(axis=(1, 2), keepdims=True) + np.sqrt(scale)
    out = {}
    for form in (cfsb.FP64_EXACT, cfsb.FP64, cfsb.FP32_MIXED):
        with cfsb.Solver(nx, ny, precision=form, rk=cfsb.RK_SSP3, hll=hll, bc=(cfsb.BC_PERIODIC,) * 4) as s:
            s.set_state(U)
            dt = s.compute_dt(0.4)
            s.step(dt if form == cfsb.FP64_EXACT else out["dt"])
            out.setdefault("dt", dt)
            out[form] = s.get_state()
    # FP64: the repository's bound of a step; FP32: storage of the deviations
    # (2^-24 of their size) and three stages of fluxes of up to 5 times the
    # state at a Courant number of 0.4, each a few roundings
    assert (np.abs(out[cfsb.FP64] - out[cfsb.FP64_EXACT]) / size).max() < 1e-12
    assert (np.abs(out[cfsb.FP32_MIXED] - out[cfsb.FP64_EXACT]) / size).max() < 4e-6
