"""Every integrator, HLL variant and rounding mode: the default kernels, whose
scheme is compiled in for three combinations and tested at run time for the
others, against the engine's exact form, alone and in a batch."""
import importlib

import numpy as np
import pytest

cfsb = importlib.import_module("2d_compressible_flow_solver_b200")
wl = importlib.import_module("2d_compressible_flow_solver_b200.workloads")

pytestmark = pytest.mark.gpu

N, P = cfsb.BC_NEUMANN, cfsb.BC_PERIODIC


@pytest.mark.parametrize("form,rounding", [(cfsb.FP64, 2), (cfsb.FP32_MIXED, 0), (cfsb.FP32_MIXED, 1), (cfsb.FP32_MIXED, 2)])
@pytest.mark.parametrize("rk", [cfsb.RK_TVD2, cfsb.RK_TVD3_REFERENCE, cfsb.RK_SSP3])
@pytest.mark.parametrize("hll", [cfsb.HLL_REFERENCE, cfsb.HLL_DAVIS])
@pytest.mark.parametrize("bc", [(P, P, P, P), (N, N, N, N)])
def test_steps_against_the_exact_form(form, rounding, rk, hll, bc):
    nx, ny, dt = 70, 61, 1e-3
    rng = np.random.default_rng(3)
    rho, u, v, p = (rng.uniform(a, b, size=(nx, ny)) for a, b in ((0.8, 1.2), (-0.4, 0.4), (-0.4, 0.4), (0.9, 1.1)))
    U = wl.conserved(rho, u, v, p)
    kw = dict(rk=rk, hll=hll)
    with cfsb.Solver(nx, ny, precision=cfsb.FP64_EXACT, bc=bc, **kw) as s:
        s.set_state(U)
        s.advance(3, dt=dt)
        ref = s.get_state()
    with cfsb.Solver(nx, ny, precision=form, bc=bc, rounding=rounding, **kw) as s:
        s.set_state(U)
        s.advance(3, dt=dt)
        got = s.get_state()
    with cfsb.Batch([{"nx": nx, "ny": ny, "bc": bc}], precision=form, rounding=rounding, **kw) as b:
        b.set_state(0, U)
        b.advance(3, dt=dt)
        batched = b.get_state(0)
    # FP64: the repository's bound of a step; FP32: 2^-24 storage and fluxes, three steps
    tol = (1e-12 if form == cfsb.FP64 else 4e-6) * np.abs(U).max()
    assert np.abs(got - ref).max() < tol
    assert np.abs(batched - ref).max() < tol
