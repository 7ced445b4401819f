"""Grids down to the smallest (3 x 3), at the edges of the row march's 30-column
segments and of its shortest row chunks, with every kind of side: one step of
the throughput forms against the engine's exact form."""
import importlib

import numpy as np
import pytest

cfsb = importlib.import_module("2d_compressible_flow_solver_b200")
wl = importlib.import_module("2d_compressible_flow_solver_b200.workloads")

pytestmark = pytest.mark.gpu

N, D, P = cfsb.BC_NEUMANN, cfsb.BC_DIRICHLET, cfsb.BC_PERIODIC


@pytest.mark.parametrize("bc", [(N, N, N, N), (D, N, N, D), (P, P, N, N), (N, D, P, P), (P, P, P, P)])
@pytest.mark.parametrize("nx,ny", [(3, 3), (3, 64), (64, 3), (5, 29), (4, 30), (7, 31), (33, 61), (129, 90)])
def test_one_step_against_the_exact_form(nx, ny, bc):
    rng = np.random.default_rng(nx * 1000 + ny)
    rho, u, v, p = (rng.uniform(a, b, size=(nx, ny)) for a, b in ((0.8, 1.2), (-0.4, 0.4), (-0.4, 0.4), (0.9, 1.1)))
    U = wl.conserved(rho, u, v, p)
    prim = [[1.1, 0.3, -0.1, 1.05]] * 4
    out, dt = {}, None
    for form in (cfsb.FP64_EXACT, cfsb.FP64, cfsb.FP32_MIXED):
        with cfsb.Solver(nx, ny, precision=form, rk=cfsb.RK_TVD3_REFERENCE, bc=bc, bc_prim=prim) as s:
            s.set_state(U)
            dt = dt or s.compute_dt(0.4)
            s.advance(2, dt=dt)
            out[form] = s.get_state()
    size = np.abs(U).max()
    # FP64: the repository's bound of a step; FP32: 2^-24 storage and fluxes, two steps of three stages
    assert np.abs(out[cfsb.FP64] - out[cfsb.FP64_EXACT]).max() < 1e-12 * size
    assert np.abs(out[cfsb.FP32_MIXED] - out[cfsb.FP64_EXACT]).max() < 4e-6 * size
