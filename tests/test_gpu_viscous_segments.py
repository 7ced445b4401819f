"""Navier-Stokes terms at the edges of the viscous march's 26-column segments
and shortest row chunks, against the C oracle's restatement, per RK step:
the bounds of test_gpu_viscous.py."""
import numpy as np
import pytest

import oracle_bind as ob

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,tol", [(0, 1e-12), (1, 2e-5)])
@pytest.mark.parametrize("bc", [(2, 2, 2, 2), (0, 1, 0, 0)])
@pytest.mark.parametrize("nx,ny", [(3, 3), (4, 26), (40, 25), (7, 27), (9, 52), (130, 53)])
def test_step_matches_oracle(cfsb, workloads, prec, tol, bc, nx, ny):
    prim = [(1.1, 0.2, 0.1, 1.0)] * 4
    rng = np.random.default_rng(nx + 1000 * ny)
    rho, u, v, p = (rng.uniform(a, b, size=(nx, ny)) for a, b in ((0.8, 1.2), (-0.4, 0.4), (-0.4, 0.4), (0.9, 1.1)))
    U = workloads.conserved(rho, u, v, p)
    cfg = ob.make_orc_config(nx, ny, rk=2, hll=1, bc=bc, bc_prim=prim, viscous=1, mu=2e-3, prandtl=0.72, mach=1.0)
    dt = ob.orc_cfl_dt(cfg, U, 0.3)
    with cfsb.Solver(nx, ny, precision=prec, rk=cfsb.RK_SSP3, hll=cfsb.HLL_DAVIS, bc=bc, bc_prim=prim,
                     viscous=cfsb.VISCOUS_NS, mu=2e-3, prandtl=0.72, mach=1.0) as s:
        s.set_state(U)
        s.step(dt)
        got = s.get_state()
    ref, _ = ob.orc_run(cfg, U, 1, 3, dt=dt)
    for k in range(4):
        assert np.abs(got[k] - ref[k]).max() <= tol * max(np.abs(ref[k]).max(), 1e-300)
