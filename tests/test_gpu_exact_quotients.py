"""The exact form's quotients by 3, 6 and the weight sum (formed from products
and remainders) against plain divisions, where they could differ: signed zeros,
values at the ends of the range they are used in and beyond it, subnormals,
equal states -- bit for bit the C oracle (the reference's operations)."""
import numpy as np
import pytest

import oracle_bind as ob

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1.0, 1e-3, 1e-250, 1e-199, 3e-200, 1e-310, 1e40, 4e59, 1e61, 1e100])
@pytest.mark.parametrize("shape", [(40, 33), (8, 32), (9, 65)])
def test_stages_are_bitwise_the_oracle(cfsb, scale, shape):
    nx, ny = shape
    rng = np.random.default_rng(int(abs(np.log10(scale))) + nx)
    rho, p = rng.uniform(0.5, 2.0, size=(2, nx, ny))
    mx, my = rng.uniform(-1, 1, size=(2, nx, ny)) * scale
    mx[rng.uniform(size=(nx, ny)) < 0.2] = 0.0
    my[rng.uniform(size=(nx, ny)) < 0.3] = -0.0
    U = np.stack([rho, mx, my, p / 0.4 + 0.5 * (mx * mx + my * my) / rho])
    with np.errstate(all="ignore"):
        dt = 1e-4 / max(1.0, scale)
        with cfsb.Solver(nx, ny, precision=cfsb.FP64_EXACT, rk=cfsb.RK_TVD3_REFERENCE) as s:
            s.set_state(U)
            for k in range(1, 4):
                s.stage(k, dt)
            got = s.get_state()
        ref, _ = ob.orc_run(ob.make_orc_config(nx, ny), U, 1, 3, dt=dt)
    assert np.array_equal(got, ref, equal_nan=True)
