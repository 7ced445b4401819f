"""A stage in parts on the narrowest slab that takes them (6 rows: no interior
rows): the whole stages' state, time and time step."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(s, cfsb, steps, stages, split, **dt):
    s.steps_begin(**dt)
    for _ in range(steps * stages):
        if split:
            s.steps_stage(cfsb.PART_INTERIOR)
            s.steps_stage(cfsb.PART_EDGES)
        else:
            s.steps_stage()
    return s.steps_end()


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("nx,ny", [(6, 64), (6, 301), (7, 64)])
@pytest.mark.parametrize("rk,stages", [(0, 2), (2, 3)])
@pytest.mark.parametrize("dt", [{"cfl": 0.4}, {"dt": 1e-3}])
def test_parts_without_interior_rows_equal_whole_stages(cfsb, workloads, prec, nx, ny, rk, stages, dt):
    U = workloads.riemann_quadrants(nx, ny, seed=9).U0
    got = []
    for split in (False, True):
        with cfsb.Solver(nx, ny, nx / ny, 1.0, precision=prec, rk=rk, hll=cfsb.HLL_DAVIS, bc=(cfsb.BC_PERIODIC,) * 4) as s:
            s.set_state(U)
            t = _run(s, cfsb, 3, stages, split, **dt)
            t2 = _run(s, cfsb, 2, stages, split, **dt)
            got.append((s.get_state(), t, t2))
    assert got[0][1][0] > 0 and got[0][1:] == got[1][1:]
    assert np.array_equal(got[0][0], got[1][0])
