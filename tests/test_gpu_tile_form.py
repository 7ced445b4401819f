"""The tile form that small grids run in (a warp per row) against the row march
(march_rows fixed): the same device functions with every contraction written
out, so the same bits, at the edges of tiles and segments and with every feature."""
import importlib

import numpy as np
import pytest

cfsb = importlib.import_module("2d_compressible_flow_solver_b200")
wl = importlib.import_module("2d_compressible_flow_solver_b200.workloads")

pytestmark = pytest.mark.gpu

N, D, P = cfsb.BC_NEUMANN, cfsb.BC_DIRICHLET, cfsb.BC_PERIODIC


@pytest.mark.parametrize("prec", [cfsb.FP64, cfsb.FP32_MIXED])
@pytest.mark.parametrize("kw", [
    {"bc": (P, P, P, P)},
    {"bc": (N, N, N, N), "rk": cfsb.RK_TVD3_REFERENCE, "hll": cfsb.HLL_REFERENCE},
    {"bc": (D, N, N, D), "rk": cfsb.RK_TVD2, "hll": cfsb.HLL_REFERENCE, "positivity": cfsb.POSITIVITY_FLOOR},
    {"bc": (P, P, P, P), "viscous": cfsb.VISCOUS_NS, "keep_rhs": True},
    {"bc": (N, N, P, P), "rounding": cfsb.ROUND_NEAREST, "positivity": cfsb.POSITIVITY_FACE},
])
@pytest.mark.parametrize("nx,ny", [(3, 3), (2 * 3, 30), (5, 31), (17, 29), (64, 61), (150, 130), (230, 200)])
def test_tile_form_equals_the_march(prec, kw, nx, ny):
    rng = np.random.default_rng(nx + 7 * ny)
    rho, u, v, p = (rng.uniform(a, b, size=(nx, ny)) for a, b in ((0.8, 1.2), (-0.4, 0.4), (-0.4, 0.4), (0.9, 1.1)))
    U = wl.conserved(rho, u, v, p)
    outs = []
    for rows in (0, 2):
        with cfsb.Solver(nx, ny, precision=prec, march_rows=rows, bc_prim=[[1.1, 0.2, -0.1, 1.0]] * 4,
                         **{"rk": cfsb.RK_SSP3, "hll": cfsb.HLL_DAVIS, **kw}) as s:
            s.set_state(U)
            t = s.advance(3, cfl=0.4)
            outs.append((s.get_state(), t, s.get_rhs() if kw.get("keep_rhs") else 0.0))
    assert np.all(np.isfinite(outs[0][0]))
    assert np.array_equal(outs[0][0], outs[1][0]) and outs[0][1] == outs[1][1]
    assert np.array_equal(outs[0][2], outs[1][2])
