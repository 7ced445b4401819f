"""Row chunks in two lengths (the launcher's own choice on grids past the tile
form's) against chunks of one fixed length: the same bits, on grids whose rows
and segments neither divides, and every row of the split parts of a stage."""
import importlib

import numpy as np
import pytest

cfsb = importlib.import_module("2d_compressible_flow_solver_b200")
wl = importlib.import_module("2d_compressible_flow_solver_b200.workloads")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [cfsb.FP64, cfsb.FP32_MIXED])
@pytest.mark.parametrize("nx,ny", [(613, 701), (4001, 95), (97, 3001), (1201, 1031), (2503, 1777)])
def test_two_lengths_change_no_bit(prec, nx, ny):
    rng = np.random.default_rng(nx)
    x = np.arange(nx)[:, None] / nx
    y = np.arange(ny)[None, :] / ny
    rho = 1.0 + 0.2 * np.sin(2 * np.pi * (x + y)) + 0.05 * rng.uniform(size=(nx, 1))
    U = wl.conserved(rho, 0.4 + 0 * y, -0.3 + 0 * x, 1.0)
    outs = []
    for rows in (0, 13):
        with cfsb.Solver(nx, ny, precision=prec, rk=cfsb.RK_SSP3, hll=cfsb.HLL_DAVIS, march_rows=rows) as s:
            s.set_state(U)
            t = s.advance(2, cfl=0.4)
            outs.append((s.get_state(), t))
    assert np.all(np.isfinite(outs[0][0]))
    assert np.array_equal(outs[0][0], outs[1][0]) and outs[0][1] == outs[1][1]
