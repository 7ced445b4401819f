"""Work units of a batch cut by the work left against units of one fixed
length: every row of every case is stepped once (the same bits), from batches
of one tiny case to ones whose longest units reach the limit."""
import importlib

import numpy as np
import pytest

cfsb = importlib.import_module("2d_compressible_flow_solver_b200")
wl = importlib.import_module("2d_compressible_flow_solver_b200.workloads")

pytestmark = pytest.mark.gpu

SIZES = {
    "one": [(6, 6)],
    "uneven": [(64, 31), (33, 65), (7, 301), (500, 97), (301, 64), (16, 16)],
    "large": [(2049, 1023), (1999, 777), (1021, 1537), (96, 96), (3000, 61), (509, 2003), (64, 64)],
}


def states(sizes):
    out = []
    for k, (nx, ny) in enumerate(sizes):
        x = np.arange(nx)[:, None] / nx
        y = np.arange(ny)[None, :] / ny
        rho = 1.0 + 0.2 * np.sin(2 * np.pi * (x + y) + k)
        out.append(wl.conserved(rho, 0.4 + 0 * y, -0.3 + 0 * x, 1.0))
    return out


@pytest.mark.parametrize("prec", [cfsb.FP64, cfsb.FP32_MIXED])
@pytest.mark.parametrize("name", sorted(SIZES))
def test_units_change_no_bit(prec, name):
    sizes = SIZES[name]
    got = []
    # no case fixed; all; some
    for rows in ([0] * len(sizes), [11] * len(sizes), [0 if k % 2 else 17 for k in range(len(sizes))]):
        cases = [dict(nx=nx, ny=ny, bc=(cfsb.BC_PERIODIC,) * 4 if k % 3 == 0 else (cfsb.BC_NEUMANN,) * 4, rows=r)
                 for k, ((nx, ny), r) in enumerate(zip(sizes, rows))]
        with cfsb.Batch(cases, precision=prec) as b:
            for k, U in enumerate(states(sizes)):
                b.set_state(k, U)
            b.advance(2, cfl=0.4)
            got.append([b.get_state(k) for k in range(len(sizes))])
    for k in range(len(sizes)):
        assert np.all(np.isfinite(got[0][k]))
        assert np.array_equal(got[0][k], got[1][k]) and np.array_equal(got[0][k], got[2][k])
