"""Row chunks in two lengths against chunks of one fixed length, bit for bit,
where the launcher's choice meets a row range (stages in parts), cell flags and
floors, viscous terms, and the scheme that reads U^1."""
import importlib

import numpy as np
import pytest

cfsb = importlib.import_module("2d_compressible_flow_solver_b200")
wl = importlib.import_module("2d_compressible_flow_solver_b200.workloads")

pytestmark = pytest.mark.gpu
SCHEMES = {"ssp3": dict(rk=cfsb.RK_SSP3, hll=cfsb.HLL_DAVIS), "tvd3": dict(rk=cfsb.RK_TVD3_REFERENCE, hll=cfsb.HLL_REFERENCE),
           "tvd2": dict(rk=cfsb.RK_TVD2, hll=cfsb.HLL_REFERENCE), "odd": dict(rk=cfsb.RK_TVD3_REFERENCE, hll=cfsb.HLL_DAVIS)}


def _state(nx, ny):
    rng = np.random.default_rng(nx + ny)
    x, y = np.arange(nx)[:, None] / nx, np.arange(ny)[None, :] / ny
    rho = 1.0 + 0.2 * np.sin(2 * np.pi * (x + y)) + 0.05 * rng.uniform(size=(nx, 1))
    return wl.conserved(rho, 0.4 + 0 * y, -0.3 + 0 * x, 1.0)


@pytest.mark.parametrize("prec", [cfsb.FP64, cfsb.FP32_MIXED])
@pytest.mark.parametrize("scheme", sorted(SCHEMES))
@pytest.mark.parametrize("nx,ny", [(1201, 1031), (2503, 601)])
@pytest.mark.parametrize("bc", [cfsb.BC_NEUMANN, cfsb.BC_PERIODIC])
def test_stages_in_parts(prec, scheme, nx, ny, bc):
    U, outs = _state(nx, ny), []
    stages = 2 if scheme == "tvd2" else 3
    for rows, split in ((0, True), (13, False)):
        with cfsb.Solver(nx, ny, precision=prec, bc=(bc,) * 4, march_rows=rows, **SCHEMES[scheme]) as s:
            s.set_state(U)
            s.steps_begin(cfl=0.4)
            for _ in range(2 * stages):
                for part in ((cfsb.PART_INTERIOR, cfsb.PART_EDGES) if split else (cfsb.PART_ALL,)):
                    s.steps_stage(part)
            t = s.steps_end()
            outs.append((s.get_state(), t))
    assert np.all(np.isfinite(outs[0][0])) and not np.array_equal(outs[0][0], U)
    assert np.array_equal(outs[0][0], outs[1][0]) and outs[0][1] == outs[1][1]


@pytest.mark.parametrize("prec", [cfsb.FP64, cfsb.FP32_MIXED])
@pytest.mark.parametrize("nx,ny", [(1301, 651), (1999, 1003)])
def test_body_and_floors(prec, nx, ny):
    prim = [(1.4, 2.5, 0.0, 1.0)] * 4
    U = wl.conserved(np.full((nx, ny), 1.4), 2.5, 0.0, 1.0)
    outs = []
    for rows in (0, 13):
        with cfsb.Solver(nx, ny, 2.0, 1.0, precision=prec, bc=(1, 0, 0, 0), bc_prim=prim, march_rows=rows,
                         positivity=cfsb.POSITIVITY_FLOOR, **SCHEMES["ssp3"]) as s:
            s.build_circle(0.07, 0.4, 0.5, mode=cfsb.IB_BILINEAR_SLIP)
            s.set_state(U)
            t = s.advance(7, cfl=0.4)
            outs.append((s.get_state(), t))
    assert np.all(np.isfinite(outs[0][0]))
    assert np.array_equal(outs[0][0], outs[1][0]) and outs[0][1] == outs[1][1]


@pytest.mark.parametrize("prec", [cfsb.FP64, cfsb.FP32_MIXED])
@pytest.mark.parametrize("nx,ny", [(1031, 1201)])
def test_viscous_terms(prec, nx, ny):
    U, outs = _state(nx, ny), []
    for rows in (0, 13):
        with cfsb.Solver(nx, ny, precision=prec, bc=(cfsb.BC_PERIODIC,) * 4, viscous=cfsb.VISCOUS_NS, mu=5e-4,
                         march_rows=rows, **SCHEMES["ssp3"]) as s:
            s.set_state(U)
            t = s.advance(3, cfl=0.4)
            outs.append((s.get_state(), t))
    assert np.all(np.isfinite(outs[0][0]))
    assert np.array_equal(outs[0][0], outs[1][0]) and outs[0][1] == outs[1][1]
