"""Performance cases of the stage engine: what its users have it do, through
``Solver`` and ``Batch``.

A pass is a stretch of a real run: (for a study of many initial states) a state
up from host memory, a number of time steps, and the new state down to host
memory, where a program keeps its frames.  The FP64 forms' frames are kept in
64 bits, the FP32-mixed form's in 32 (what the form stores).

A case is a dict:
  flow    "quadrants" (four-quadrant Riemann states, transmissive sides), "advection" (smooth, periodic),
          "cylinder" (supersonic flow past a slip-wall circle, Dirichlet inflow, positivity floors), "shear" (periodic
          Navier-Stokes shear layer), "batch" (uneven quadrant and cylinder grids advanced together)
  nx, ny  cells (batch: ``cases`` grids with edges drawn from 64..``edge`` in steps of 16 by ``layout``)
  form    "f64", "f32" (FP32-mixed) or "exact" (the reference's arithmetic bit for bit)
  rk      "tvd2", "tvd3" (as the reference writes it) or "ssp3";  hll "reference" or "davis"
  steps   time steps of a pass;  per_call: steps of one ``advance`` call (0: the drop-in's loop, one
          ``compute_dt`` a step and one ``stage`` call a stage)
  restart true: every pass begins with a state from the host; false: it goes on from the last one
  pinned  host frames in pinned memory (else ordinary pageable arrays)
"""
import importlib
import math
import random

import numpy as np
import torch

cfsb = importlib.import_module("2d_compressible_flow_solver_b200")

GAMMA = 1.4
EPS = 1e-2
PRANDTL, MACH, MU = 0.72, 1.0, 1.0 / 2000.0
FLOOR = 1e-6
CFL = {"quadrants": 0.5, "advection": 0.4, "cylinder": 0.5, "shear": 0.5, "batch": 0.5}
FORMS = {"f64": cfsb.FP64, "f32": cfsb.FP32_MIXED, "exact": cfsb.FP64_EXACT}
RKS = {"tvd2": cfsb.RK_TVD2, "tvd3": cfsb.RK_TVD3_REFERENCE, "ssp3": cfsb.RK_SSP3}
HLLS = {"reference": cfsb.HLL_REFERENCE, "davis": cfsb.HLL_DAVIS}
BCS = {"quadrants": (0, 0, 0, 0), "advection": (2, 2, 2, 2), "cylinder": (1, 0, 0, 0), "shear": (2, 2, 2, 2)}


def _case(name, flow, nx, ny, form, steps, per_call=None, rk="ssp3", hll="davis", restart=True, pinned=False, **more):
    return {"name": name, "flow": flow, "nx": nx, "ny": ny, "form": form, "rk": rk, "hll": hll, "steps": steps,
            "per_call": steps if per_call is None else per_call, "restart": restart, "pinned": pinned, **more}


def listed():
    ref = {"rk": "tvd3", "hll": "reference"}
    return [
        # a small grid stepped one call at a time by a program that looks at every step: latency and launches
        _case("quad_64x48_f64_single", "quadrants", 64, 48, "f64", 8, per_call=1, **ref),
        # the drop-in inside the reference's own loop (its TVD2), bit for bit the reference
        _case("dropin_256_exact", "quadrants", 256, 256, "exact", 10, per_call=0, rk="tvd2", hll="reference"),
        # the 256 x 256 Riemann configuration, one of a study of many initial states
        _case("quad_256_f32", "quadrants", 256, 256, "f32", 40, **ref),
        # the same in the plain FP64 form, TVD2, on an odd grid
        _case("quad_251x333_f64", "quadrants", 251, 333, "f64", 40, rk="tvd2", hll="reference"),
        # smooth advection on a ragged middle-sized grid
        _case("adv_1021x1537_f32", "advection", 1021, 1537, "f32", 60, restart=False, pinned=True),
        # the plain FP64 form on a large grid
        _case("adv_2048_f64", "advection", 2048, 2048, "f64", 60, restart=False, pinned=True),
        # the largest configuration: 4096 x 4096 FP32-mixed between two frames
        _case("adv_4096_f32", "advection", 4096, 4096, "f32", 80, restart=False, pinned=True),
        # the Mach-3 cylinder configuration, host arrays as a C++ caller's vectors
        _case("cyl_2048x1024_f32", "cylinder", 2048, 1024, "f32", 60),
        # a coarse odd cylinder grid in FP64
        _case("cyl_605x301_f64", "cylinder", 605, 301, "f64", 40),
        # the Navier-Stokes shear layer configuration
        _case("shear_1024_f32", "shear", 1024, 1024, "f32", 60, restart=False, pinned=True),
        # the same terms in FP64 on a ragged grid
        _case("shear_517x389_f64", "shear", 517, 389, "f64", 40, restart=False),
        # a sweep of uneven grids advanced together
        _case("batch_48_f32", "batch", 0, 0, "f32", 80, restart=False, cases=48, edge=768, layout=1),
    ]


def draw(rng):
    flow = rng.choice(["quadrants", "quadrants", "advection", "advection", "cylinder", "shear", "batch"])
    form = rng.choice(["f32", "f32", "f64"])
    if flow == "batch":
        n = int(round(math.exp(rng.uniform(math.log(4), math.log(48)))))
        return {k: v for k, v in _case("", flow, 0, 0, form, rng.randint(40, 80), restart=False, cases=n,
                                       edge=rng.choice([256, 512, 768]), layout=rng.randint(2, 1 << 20)).items() if k != "name"}
    top = {"quadrants": 1500, "advection": 3000, "cylinder": 1500, "shear": 1400}[flow]
    nx, ny = (int(round(math.exp(rng.uniform(math.log(64 if flow == "cylinder" else 33), math.log(top))))) for _ in range(2))
    if flow == "cylinder":
        nx = max(96, 2 * ny + rng.randint(-ny // 4, ny // 4))
    if flow == "quadrants" and rng.random() < 0.15:
        form = "exact"
    rk, hll = ("ssp3", "davis")
    if flow == "quadrants":
        rk, hll = rng.choice([("tvd2", "reference"), ("tvd3", "reference"), ("ssp3", "davis")])
    steps = max(6, min(40, int(4e8 / (nx * ny))))
    per_call = steps
    if form == "exact":
        nx, ny, steps, per_call = min(nx, 600), min(ny, 600), 6, 0
    elif nx * ny < 40000 and rng.random() < 0.4:
        per_call = 1
    restart = flow in ("quadrants", "cylinder") or rng.random() < 0.3
    c = _case("", flow, nx, ny, form, steps, per_call=per_call, rk=rk, hll=hll, restart=restart, pinned=rng.random() < 0.5)
    del c["name"]
    return c


# ------------------------------------------------------------------ inputs
def _conserved(rho, u, v, p):
    mx, my = rho * u, rho * v
    return np.stack(np.broadcast_arrays(rho, mx, my, p / (GAMMA - 1) + 0.5 * (mx * mx + my * my) / rho))


def _centres(nx, ny, lx, ly):
    return ((np.arange(nx) + 0.5) * (lx / nx))[:, None], ((np.arange(ny) + 0.5) * (ly / ny))[None, :]


def _quadrants(nx, ny, rng, strong):
    """Four-quadrant states; not ``strong``: drawn milder, so that the reference's scheme, which has no positivity
    fallback, carries every draw."""
    x, y = _centres(nx, ny, 1.0, 1.0)
    low, fast = (0.1, 1.0) if strong else (0.5, 0.5)
    q = [[rng.uniform(2 * low if strong else low, 2.0), rng.uniform(-fast, fast), rng.uniform(-fast, fast),
          rng.uniform(low, 2.0)] for _ in range(4)]
    at = (x >= 0.5).astype(int) + 2 * (y >= 0.5).astype(int)
    w = np.array(q)[at]
    return _conserved(w[..., 0], w[..., 1], w[..., 2], w[..., 3])


def _inflow(rng, slow, fast):
    rho, p, mach = 1.4, 1.0, rng.uniform(slow, fast)
    return [rho, mach * math.sqrt(GAMMA * p / rho), 0.0, p]


def _grid(case, seed):
    """(state, bc_prim, circle, lx) of a single grid."""
    nx, ny, flow = case["nx"], case["ny"], case["flow"]
    rng = random.Random(1000003 * int(seed) + 17)
    if flow == "quadrants":
        return _quadrants(nx, ny, rng, False), None, None, 1.0
    if flow == "advection":
        x, y = _centres(nx, ny, 1.0, 1.0)
        ph, amp = rng.uniform(0, 2 * math.pi), rng.uniform(0.15, 0.25)
        rho = (torch.from_numpy(x) + torch.from_numpy(y)).mul_(2 * math.pi).add_(ph).sin_().mul_(amp).add_(1.0).numpy()
        return np.stack([rho, rho, rho, rho + 1.0 / (GAMMA - 1)]), None, None, 1.0
    if flow == "shear":
        x, y = _centres(nx, ny, 1.0, 1.0)
        u = np.tanh((np.abs(y - 0.5) - 0.25) / 0.02) * np.where(y >= 0.5, 1.0, -1.0)
        v = 0.01 * sum(rng.uniform(-1, 1) * np.sin(2 * np.pi * (k + 1) * x) for k in range(8))
        return _conserved(np.ones((nx, ny)), u, v, 2.5), None, None, 1.0
    prim = _inflow(rng, 2.0, 3.0)
    lx = 2.0
    circle = (rng.uniform(0.04, 0.08), rng.uniform(0.35, 0.45), rng.uniform(0.45, 0.55))
    return _conserved(np.full((nx, ny), prim[0]), prim[1], prim[2], prim[3]), [prim] * 4, circle, lx


def _batch_sizes(case):
    rng = random.Random(case["layout"])
    edges = range(64, case["edge"] + 1, 16)
    return [(rng.choice(edges), rng.choice(edges)) for _ in range(case["cases"])]


def _batch(case, seed):
    """Case descriptions and states: half quadrants, half cylinders."""
    rng = random.Random(1000003 * int(seed) + 29)
    descs, states = [], []
    for k, (nx, ny) in enumerate(_batch_sizes(case)):
        d = {"nx": nx, "ny": ny, "lx": 1.0, "ly": 1.0, "bc": (0, 0, 0, 0)}
        if k % 2 == 0:
            states.append(_quadrants(nx, ny, rng, True))
        else:
            prim = _inflow(rng, 1.5, 2.2)  # (a run goes on for hundreds of steps; faster, a coarse case now and then blows up)
            r = rng.uniform(0.03, 0.1)
            d.update(bc=(1, 0, 0, 0), bc_prim=[prim] * 4, ib_mode=cfsb.IB_BILINEAR_SLIP,
                     circle=(r, rng.uniform(3 * r, 1 - 3 * r), rng.uniform(3 * r, 1 - 3 * r)))
            states.append(_conserved(np.full((nx, ny), prim[0]), prim[1], prim[2], prim[3]))
        descs.append(d)
    return descs, states


# -------------------------------------------------------------------- runs
def _host(shape, pinned, dtype=torch.float64):
    return torch.empty(shape, dtype=dtype, pin_memory=pinned)


def prepare(case, seed):
    form = FORMS[case["form"]]
    if case["flow"] == "batch":
        descs, states = _batch(case, seed)
        b = cfsb.Batch(descs, precision=form, rk=RKS[case["rk"]], hll=HLLS[case["hll"]], positivity=cfsb.POSITIVITY_FLOOR)
        for k, u in enumerate(states):
            b.set_state(k, u)
        kept = [np.zeros(u.shape, np.float32) for u in states] if case["form"] == "f32" else None
        return {"case": case, "batch": b, "frames32": kept}
    u0, prim, circle, lx = _grid(case, seed)
    s = cfsb.Solver(case["nx"], case["ny"], lx, 1.0, precision=form, rk=RKS[case["rk"]], hll=HLLS[case["hll"]],
                    bc=BCS[case["flow"]], bc_prim=prim,
                    positivity=cfsb.POSITIVITY_FLOOR if circle else cfsb.POSITIVITY_OFF,
                    viscous=cfsb.VISCOUS_NS if case["flow"] == "shear" else cfsb.VISCOUS_OFF,
                    mu=MU, prandtl=PRANDTL, mach=MACH)
    if circle:
        s.build_circle(*circle, mode=cfsb.IB_BILINEAR_SLIP)
    first = _host(u0.shape, case["pinned"])
    first.copy_(torch.from_numpy(u0))
    s.set_state(first.numpy())
    st = {"case": case, "solver": s, "first": first if case["restart"] else None, "frame": _host(u0.shape, case["pinned"])}
    if case["form"] == "f32":
        st["frame32"] = _host(u0.shape, False, torch.float32)
    return st


def run(state):
    case = state["case"]
    cfl, steps, per = CFL[case["flow"]], case["steps"], case["per_call"]
    if "batch" in state:
        b = state["batch"]
        t = b.advance(steps, cfl=cfl)
        frames = [b.get_state(k) for k in range(len(b.shapes))]
        if case["form"] == "f32":
            for to, f in zip(state["frames32"], frames):
                np.copyto(to, f, casting="same_kind")
            frames, t = state["frames32"], t.astype(np.float32)
        return {"frames": frames, "t": t}
    s = state["solver"]
    if case["restart"]:
        s.set_state(state["first"].numpy())
    t = 0.0
    if per == 0:
        stages = 2 if case["rk"] == "tvd2" else 3
        for i in range(1, steps * stages + 1):
            if i % stages == 1:
                dt = s.compute_dt(cfl)
                t += dt
            s.stage(i, dt)
    else:
        for _ in range(steps // per):
            t += s.advance(per, cfl=cfl)[0]
        if steps % per:
            t += s.advance(steps % per, cfl=cfl)[0]
    s.get_state(state["frame"].numpy())
    if case["form"] != "f32":
        return {"frame": state["frame"], "t": t}
    state["frame32"].copy_(state["frame"])
    return {"frame": state["frame32"], "t": np.float32(t)}


def work(case):
    """Bytes: per step every stored state value read and written once, and the host's states in and out.  Flops: per
    cell and stage both biased WENO5 states of four variables in two directions, their pressures and sound speeds, two
    HLL fluxes and the update (about 800), and the viscous terms (about 180)."""
    cells = sum(a * b for a, b in _batch_sizes(case)) if case["flow"] == "batch" else case["nx"] * case["ny"]
    word = 4 if case["form"] == "f32" else 8
    stages = 2 if case["rk"] == "tvd2" else 3
    per = 800 + (180 if case["flow"] == "shear" else 0)
    copies = (2 if case["restart"] else 1) * 32
    return {"bytes": float(cells * (case["steps"] * 8 * word + copies)), "flops": float(cells * case["steps"] * stages * per)}


# ------------------------------------------- the same scheme in plain torch
def _weno(a, b, c, d, e):
    """WENO5-JS value at the upper face of the cell c from five cell values."""
    b0 = 13 / 12 * (a - 2 * b + c) ** 2 + 0.25 * (a - 4 * b + 3 * c) ** 2
    b1 = 13 / 12 * (b - 2 * c + d) ** 2 + 0.25 * (b - d) ** 2
    b2 = 13 / 12 * (c - 2 * d + e) ** 2 + 0.25 * (3 * c - 4 * d + e) ** 2
    w0, w1, w2 = 0.1 / (EPS + b0) ** 2, 0.6 / (EPS + b1) ** 2, 0.3 / (EPS + b2) ** 2
    return (w0 * (2 * a - 7 * b + 11 * c) + w1 * (-b + 5 * c + 2 * d) + w2 * (2 * c + 5 * d - e)) / (6 * (w0 + w1 + w2))


def _pressure(u):
    return (GAMMA - 1) * (u[3] - 0.5 * (u[1] ** 2 + u[2] ** 2) / u[0])


def _flux(L, R, d, davis):
    """HLL flux in direction d (0 x, 1 y)."""
    def phys(u):
        un, p = u[1 + d] / u[0], _pressure(u)
        f = torch.stack([u[1 + d], u[1] * un, u[2] * un, (u[3] + p) * un])
        f[1 + d] += p
        return f, un, p, torch.sqrt(GAMMA * p / u[0])

    FL, uL, pL, aL = phys(L)
    FR, uR, pR, aR = phys(R)
    if davis:
        SL, SR = torch.fmin(uL - aL, uR - aR), torch.fmax(uL + aL, uR + aR)
    else:
        qL, a, r = L[1 + d], 0.5 * (aL + aR), 0.5 * (L[0] + R[0])
        ps, us = 0.5 * (pL + pR) - 0.5 * (uR - uL) * r * a, 0.5 * (uR + uL) - 0.5 * (pR - pL) / (r * a)
        lo = us - torch.sqrt(GAMMA * ps / (L[0] + (uL - us) * r / a))
        hi = us + torch.sqrt(GAMMA * ps / (R[0] - (uR - us) * r / a))
        SL, SR = torch.where(lo < qL - aL, lo, qL - aL), torch.where(hi > qL + aL, hi, qL + aL)
    mid = (SR * FL - SL * FR + SL * SR * (R - L)) / (SR - SL)
    return torch.where(SL >= 0, FL, torch.where(SR <= 0, FR, mid))


class _Plain:
    """The engine's scheme on one grid in 64 bits."""

    def __init__(self, case, u0, bc, prim, circle, lx, dev):
        self.rk, self.davis, self.bc, self.dev = case["rk"], case["hll"] == "davis", bc, dev
        self.viscous, self.floors = case["flow"] == "shear", case["flow"] in ("cylinder", "batch")
        self.nx, self.ny = u0.shape[1:]
        self.dx, self.dy = lx / self.nx, 1.0 / self.ny
        self.U = torch.from_numpy(u0).to(dev)
        self.ghost = None if prim is None else torch.from_numpy(_conserved(*(np.array(v) for v in prim[0]))).to(dev)
        self.body = circle is not None
        self.solid, self.low = torch.zeros((self.nx, self.ny), dtype=torch.bool, device=dev), (False, False)
        if self.body:
            self._circle(*circle)

    def _circle(self, radius, cx, cy):
        """Solid and ghost cells, image points and slip weights of a 400-point circle."""
        nx, ny, dx, dy = self.nx, self.ny, self.dx, self.dy
        x, y = (np.arange(nx) + 0.5) * dx, (np.arange(ny) + 0.5) * dy
        solid = np.sqrt((x[:, None] - cx) ** 2 + (y[None, :] - cy) ** 2) <= radius
        pad = np.pad(~solid, 3)
        near = np.zeros_like(solid)
        for k in (1, 2, 3):
            for a, b in ((k, 0), (-k, 0), (0, k), (0, -k)):
                near |= pad[3 + a:3 + a + nx, 3 + b:3 + b + ny]
        gi, gj = np.nonzero(solid & near)
        ang = 2 * np.pi * np.arange(400) / 400
        px, py = cx + radius * np.cos(ang), cy + radius * np.sin(ang)
        sx, sy = np.roll(px, -1) - px, np.roll(py, -1) - py
        n = np.sqrt(sx * sx + sy * sy)
        sx, sy = sx / n, sy / n
        ax, ay = x[gi][:, None], y[gj][:, None]
        dd = sx * (ax - px) + sy * (ay - py)
        qx, qy = dd * sx + px, dd * sy + py
        dist = np.sqrt((qx - ax) ** 2 + (qy - ay) ** 2)
        k = dist.argmin(1)
        rows = np.arange(len(gi))
        dist, ex, ey = dist[rows, k], qx[rows, k] - ax[:, 0], qy[rows, k] - ay[:, 0]
        n = np.sqrt(ex * ex + ey * ey)
        n = np.where(n > 0, n, 1.0)
        ex, ey = ex / n, ey / n
        X, Y = ax[:, 0] + 2 * dist * ex, ay[:, 0] + 2 * dist * ey
        fx, fy = (X - 0.5 * dx) / dx, (Y - 0.5 * dy) / dy
        i0, j0 = np.floor(fx).astype(int), np.floor(fy).astype(int)
        tx, ty = fx - i0, fy - j0
        ci, cj = np.stack([i0, i0 + 1, i0, i0 + 1], 1), np.stack([j0, j0, j0 + 1, j0 + 1], 1)
        w = np.stack([(1 - tx) * (1 - ty), tx * (1 - ty), (1 - tx) * ty, tx * ty], 1)
        ok = (ci >= 0) & (ci < nx) & (cj >= 0) & (cj < ny)
        ci, cj = ci.clip(0, nx - 1), cj.clip(0, ny - 1)
        ok &= ~solid[ci, cj]
        w = np.where(ok, w, 0.0)
        for g in np.nonzero(w.sum(1) <= 1e-3)[0]:  # no fluid block: inverse distances of the 4 nearest fluid cells
            a, b = int((X[g] - x[0]) / dx), int((Y[g] - y[0]) / dy)
            wi = [(i, j) for i in range(a - 5, a + 6) for j in range(b - 5, b + 6) if 0 <= i < nx and 0 <= j < ny and not solid[i, j]]
            wi = sorted(wi, key=lambda c: (x[c[0]] - X[g]) ** 2 + (y[c[1]] - Y[g]) ** 2)[:4]
            ci[g], cj[g] = [c[0] for c in wi], [c[1] for c in wi]
            w[g] = [1 / ((x[i] - X[g]) ** 2 + (y[j] - Y[g]) ** 2 + 1e-300) for i, j in wi]
        w /= w.sum(1, keepdims=True)
        up = lambda v: torch.from_numpy(np.ascontiguousarray(v)).to(self.dev)  # noqa: E731
        self.solid, self.gi, self.gj, self.ci, self.cj, self.w, self.ex, self.ey = map(up, (solid, gi, gj, ci, cj, w, ex, ey))
        s = np.pad(solid, 3)
        s[:3], s[-3:], s[:, :3], s[:, -3:] = False, False, False, False
        lx = np.stack([s[k:k + nx + 1, 3:-3] for k in range(6)]).any(0)
        ly = np.stack([s[3:-3, k:k + ny + 1] for k in range(6)]).any(0)
        lx[0], lx[-1], ly[:, 0], ly[:, -1] = solid[0], solid[-1], solid[:, 0], solid[:, -1]
        self.low = (up(lx), up(ly))

    def fill(self, U):
        if self.body:
            v = (U[:, self.ci, self.cj] * self.w).sum(2)
            mn = v[1] * self.ex + v[2] * self.ey
            v[1] -= 2 * mn * self.ex
            v[2] -= 2 * mn * self.ey
            U[:, self.gi, self.gj] = v

    def padded(self, U):
        nx, ny = self.nx, self.ny
        if self.bc[0] == 2:
            P = torch.cat([U[:, -3:], U, U[:, :3]], 1)
            return torch.cat([P[:, :, -3:], P, P[:, :, :3]], 2)
        P = torch.empty((4, nx + 6, ny + 6), dtype=U.dtype, device=U.device)
        P[:, 3:-3, 3:-3] = U
        P[:, :3, 3:-3] = self.ghost.view(4, 1, 1) if self.bc[0] == 1 else U[:, :1]
        P[:, -3:, 3:-3] = U[:, -1:]
        P[:, :, :3], P[:, :, -3:] = P[:, :, 3:4], P[:, :, -4:-3]
        return P

    def direction(self, P, d):
        """Fluxes through the faces of direction d, [4][n+1][cells across]."""
        V = P[:, :, 3:-3] if d == 0 else P[:, 3:-3, :].transpose(1, 2)
        n = V.shape[1] - 6
        s = [V[:, k:k + n + 1] for k in range(6)]
        L, R = _weno(*s[:5]), _weno(*s[5:0:-1])
        if self.bc[0] != 2:  # a physical face's stencil repeats the cell and the ghost beside it
            for f in (0, n):
                a, b = s[2][:, f], s[3][:, f]
                L[:, f], R[:, f] = _weno(a, a, a, b, b), _weno(b, b, b, a, a)
        if self.floors:
            low = self.low[d] if d == 0 or not self.body else self.low[1].transpose(0, 1)
            L = torch.where(low | ~((L[0] > 0) & (_pressure(L) > 0)), s[2], L)
            R = torch.where(low | ~((R[0] > 0) & (_pressure(R) > 0)), s[3], R)
        F = _flux(L, R, d, self.davis)
        return F if d == 0 else F.transpose(1, 2)

    def viscous_rhs(self, P):
        u, v = P[1] / P[0], P[2] / P[0]
        T = GAMMA * MACH ** 2 * _pressure(P) / P[0]
        w = torch.stack([u, v, T])
        kT = MU / ((GAMMA - 1) * MACH ** 2 * PRANDTL)
        out = None
        for d, h, g in ((0, self.dx, self.dy), (1, self.dy, self.dx)):
            q = w if d == 0 else w.transpose(1, 2)  # rows along the face normal
            n, m = q.shape[1] - 6, q.shape[2] - 6
            c = q[:, :, 3:3 + m]
            dn = (-3 / 640 * (c[:, 0:n + 1] - c[:, 5:n + 6]) + 25 / 384 * (c[:, 1:n + 2] - c[:, 4:n + 5])
                  - 75 / 64 * (c[:, 2:n + 3] - c[:, 3:n + 4])) / h
            t = ((q[:, :, 1:1 + m] - q[:, :, 5:5 + m]) / 12 - 8 / 12 * (q[:, :, 2:2 + m] - q[:, :, 4:4 + m])) / g
            mid = lambda z: (9 * (z[:, 2:n + 3] + z[:, 3:n + 4]) - (z[:, 1:n + 2] + z[:, 4:n + 5])) / 16  # noqa: E731
            cr, f = mid(t), mid(c)
            a, b = (0, 1) if d == 0 else (1, 0)  # normal and transverse velocity
            snn = MU * (4 / 3 * dn[a] - 2 / 3 * cr[b])
            snt = MU * (cr[a] + dn[b])
            e = f[a] * snn + f[b] * snt + kT * dn[2]
            F = torch.stack([torch.zeros_like(e), snn, snt, e] if d == 0 else [torch.zeros_like(e), snt, snn, e])
            D = (F[:, 1:] - F[:, :-1]) / h
            out = D if d == 0 else out + D.transpose(1, 2)
        return out

    def rhs(self, U):
        P = self.padded(U)
        F, G = self.direction(P, 0), self.direction(P, 1)
        r = -(F[:, 1:] - F[:, :-1]) / self.dx - (G[:, :, 1:] - G[:, :, :-1]) / self.dy
        return r + self.viscous_rhs(P) if self.viscous else r

    def update(self, old, new):
        if not self.floors:
            return new
        rho = new[0]
        bad = ~(rho > FLOOR) | torch.isnan(new).any(0)
        new[0] = torch.where(bad, FLOOR, rho)
        new[1:3] = torch.where(bad, 0.0, new[1:3])
        new[3] = torch.where(bad, FLOOR / (GAMMA - 1), new[3])
        ke = 0.5 * (new[1] ** 2 + new[2] ** 2) / new[0]
        new[3] = torch.where((GAMMA - 1) * (new[3] - ke) > FLOOR, new[3], FLOOR / (GAMMA - 1) + ke)
        return torch.where(self.solid, old, new)

    def dt(self, cfl):
        U = self.U
        a = torch.sqrt(GAMMA * _pressure(U) / U[0])
        w = ((U[1] / U[0]).abs() + a) / self.dx + ((U[2] / U[0]).abs() + a) / self.dy
        return cfl / float(w[~self.solid].max())

    def advance(self, steps, cfl):
        t = 0.0
        for _ in range(steps):
            self.fill(self.U)
            U0, dt = self.U, self.dt(cfl)
            t += dt
            U1 = self.update(U0, U0 + dt * self.rhs(U0))
            self.fill(U1)
            if self.rk == "tvd2":
                self.U = self.update(U1, 0.5 * U0 + 0.5 * U1 + 0.5 * dt * self.rhs(U1))
                continue
            U2 = self.update(U1, 0.75 * U0 + 0.25 * U1 + 0.25 * dt * self.rhs(U1))
            self.fill(U2)
            self.U = self.update(U2, U0 / 3 + 2 / 3 * (U1 if self.rk == "tvd3" else U2) + 2 / 3 * dt * self.rhs(U2))
        return t


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    stages = case["steps"] * (2 if case["rk"] == "tvd2" else 3)
    if case["flow"] == "batch":  # the first grids; all of them would take minutes
        descs, states = _batch(case, seed)
        frames = [None] * len(descs)
        for k in range(min(4, len(descs))):
            d = descs[k]
            p = _Plain(case, states[k], d["bc"], d.get("bc_prim"), d.get("circle"), 1.0, dev)
            p.advance(case["steps"], CFL["batch"])
            frames[k] = p.U.cpu().numpy()
        return {"frames": frames, "t": None}
    if stages * max(6e-3, case["nx"] * case["ny"] * 5e-9) > 25:
        return None
    u0, prim, circle, lx = _grid(case, seed)
    p = _Plain(case, u0, BCS[case["flow"]], prim, circle, lx, dev)
    t = p.advance(case["steps"], CFL[case["flow"]])
    return {"frame": p.U.cpu(), "t": t}
