"""The snapshot writer's contents against the C oracle's state and RHS, for
places where the reference's own classes (test_snapshot.py) are not built."""
import importlib
import json

import numpy as np
import pytest

import oracle_bind as ob

snap = importlib.import_module("2d_compressible_flow_solver_b200.snapshot")


def _oracle(nx, ny, U0, steps, dt):
    """State after `steps` TVD3 steps and the last stage's RHS."""
    cfg = ob.make_orc_config(nx, ny)
    U = np.ascontiguousarray(U0).copy()
    rhs = np.zeros_like(U)
    for _ in range(steps):
        u0 = U.copy()
        u1 = U.copy()
        for stage in range(3):
            if stage == 1:
                u1 = U.copy()
            ob.orc_stage(cfg, U, u0, u1, stage, dt, rhs=rhs)
    return U, rhs


def _matches(d, U, rhs):
    for k, name in enumerate(("Rho", "Mu", "Mv", "Energy")):
        assert np.array_equal(d[name], U[k])
    for k, name in enumerate(("FluxRho", "FluxMu", "FluxMv", "FluxEnergy")):
        assert np.array_equal(d[name], rhs[k])


def test_raw_round_trip_of_an_oracle_state(tmp_path, workloads):
    w = workloads.riemann_quadrants(24, 16, seed=2)
    U, rhs = _oracle(24, 16, w.U0, 1, 1e-3)
    p = snap.write_snapshot(tmp_path / "s", U, rhs, time=1e-3, fmt="raw")
    index = json.loads((p / "index.json").read_text())
    assert index["datasets"] == list(snap.DATASETS) and index["shape"] == [24, 16]
    assert np.fromfile(p / "Mu.f64", dtype="<f8")[5 * 16 + 7] == U[1][5, 7]  # x-major
    _matches(snap.read_snapshot(p), U, rhs)


@pytest.mark.gpu
def test_solver_snapshot_holds_the_oracle_state_and_rhs(cfsb, workloads, tmp_path):
    w = workloads.riemann_quadrants(64, 40, seed=6)
    U, rhs = _oracle(64, 40, w.U0, 2, 1e-3)
    with cfsb.Solver(64, 40, precision=cfsb.FP64_EXACT, keep_rhs=True) as s:
        s.set_state(w.U0)
        for k in range(1, 7):
            s.stage(k, 1e-3)
        p = snap.write_solver_snapshot(s, tmp_path / "g", fmt="raw")
    _matches(snap.read_snapshot(p), U, rhs)
