"""The longest work unit of a batch's cases, set by a case (negative rows) or by
the autotuner's table (Batch's default): more units where it is shorter, and
the same bits."""
import importlib

import numpy as np
import pytest

cfsb = importlib.import_module("2d_compressible_flow_solver_b200")
autotune = importlib.import_module("2d_compressible_flow_solver_b200.autotune")
wl = importlib.import_module("2d_compressible_flow_solver_b200.workloads")

pytestmark = pytest.mark.gpu
SIZES = [(2049, 1023), (64, 64), (777, 1999), (3, 3), (500, 97)]


def _run(prec, rows, tuned):
    cases = [dict(nx=nx, ny=ny, bc=(cfsb.BC_PERIODIC,) * 4, rows=rows) for nx, ny in SIZES]
    with cfsb.Batch(cases, precision=prec, tuned_rows=tuned) as b:
        for k, (nx, ny) in enumerate(SIZES):
            b.set_state(k, wl.riemann_quadrants(nx, ny, seed=k).U0)
        b.advance(2, cfl=0.4)
        return b.info()[1], [b.get_state(k) for k in range(len(SIZES))]


def _least(rows):
    return sum((ny + 29) // 30 * ((nx + rows - 1) // rows) for nx, ny in SIZES)


@pytest.mark.parametrize("prec", [cfsb.FP64, cfsb.FP32_MIXED])
def test_limits_and_table(prec, monkeypatch):
    plain, ref = _run(prec, 0, False)
    got = {}
    for name, rows, tuned in (("limit", -5, False), ("huge", -2**31, False), ("table", 0, True), ("fixed", 5, True)):
        if name == "table":
            asked = []
            monkeypatch.setattr(autotune, "batch_rows_for", lambda p, nx, ny: asked.append((p, nx, ny)) or 5)
        got[name], states = _run(prec, rows, tuned)
        for a, b in zip(states, ref):
            assert np.array_equal(a, b)
    assert asked == [("f32" if prec == cfsb.FP32_MIXED else "f64", nx, ny) for nx, ny in SIZES]
    assert got["limit"] == got["table"] > plain >= got["huge"]
    assert got["limit"] >= got["fixed"] == _least(5)
