"""A body whose ghost cells lie next to a Dirichlet side (the boundary faces'
fluxes then read what the immersed-ghost fill writes) and one inside the grid
(both run in one launch): FP64 steps, alone and in a batch, against the C
oracle on the same lists."""
import numpy as np
import pytest

import oracle_bind as ob

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cx,cy", [(0.04, 0.5), (0.5, 0.97), (0.5, 0.5)])
@pytest.mark.parametrize("bc", [(1, 0, 0, 0), (1, 1, 1, 1)])
def test_steps_match_the_oracle(cfsb, workloads, cx, cy, bc):
    nx, ny = 64, 57
    prim = [[1.4, 0.6, 0.1, 1.0]] * 4
    rng = np.random.default_rng(5)
    rho, u, v, p = (rng.uniform(a, b, size=(nx, ny)) for a, b in ((1.2, 1.6), (0.4, 0.8), (0.0, 0.2), (0.9, 1.1)))
    U = workloads.conserved(rho, u, v, p)
    types, cells, donors, images, normals = cfsb.circle_setup(nx, ny, 1.0, 1.0, 0.12, cx, cy)
    i, j = cells // ny, cells % ny
    at_side = bool(((i == 0) | (i == nx - 1) | (j == 0) | (j == ny - 1)).any())
    assert at_side == ((cx, cy) != (0.5, 0.5))
    cfg = ob.make_orc_config(nx, ny, rk=2, hll=1, bc=bc, bc_prim=prim, positivity=2)
    ib = ob.OrcIBList(cells, donors, images, normals, mode=1, types=types)
    dt = 1e-3
    ref, _ = ob.orc_run(cfg, U, 1, 9, dt=dt, types=types, ib=ib)
    assert np.all(np.isfinite(ref))
    with cfsb.Solver(nx, ny, precision=cfsb.FP64, rk=cfsb.RK_SSP3, hll=cfsb.HLL_DAVIS, bc=bc, bc_prim=prim,
                     positivity=cfsb.POSITIVITY_BODY) as s:
        s.build_circle(0.12, cx, cy, 400, cfsb.IB_BILINEAR_SLIP)
        s.set_state(U)
        s.advance(3, dt=dt)
        got = s.get_state()
    with cfsb.Batch([{"nx": nx, "ny": ny, "bc": bc, "bc_prim": prim, "circle": (0.12, cx, cy)}], precision=cfsb.FP64,
                    positivity=cfsb.POSITIVITY_BODY) as b:
        b.set_state(0, U)
        b.advance(3, dt=dt)
        batched = b.get_state(0)
    # the repository's bound of a step, three of them
    for k in range(4):
        size = np.abs(ref[k]).max()
        assert np.abs(got[k] - ref[k]).max() <= 3e-12 * size
        assert np.abs(batched[k] - ref[k]).max() <= 3e-12 * size
