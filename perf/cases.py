"""Timed workloads of the library, through its public entry points.

What a user of this framework has it do: barotropic-vorticity RK4 steps on
icosahedral grids in FP64 and FP32C (single steps between remeshes, runs of
several steps, grids refined where the vorticity is, from a few hundred panels
to several hundred thousand), single Biot-Savart sums, the forced
stratosphere model, the Voronoi (SoA) step, ensembles of uneven grids, and the
adjoint. Sizes follow configs.py and the tests; grids are refined by an
arbitrary number of panels, so tile remainders are ragged.

listed() names the workloads, draw() gives others of the same ranges,
prepare() makes inputs, run() is one pass, work() is the floor of a pass (22
algorithmic flops per interaction; inputs read and results written once), and
exact() is the same pass in plain torch in 64 bits.
"""
import ctypes
import functools
import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

from thesiscode_b200 import _native as N
from thesiscode_b200 import ics
from thesiscode_b200.batch import batch_rk4
from thesiscode_b200.configs import Workload
from thesiscode_b200.grid import new_icos_grid
from thesiscode_b200.panel_velocity import Context
from thesiscode_b200.voronoi_velocity import BVERK4, VorPanels

OMEGA = 2.0 * math.pi
FLOPS_PER_PAIR = 22.0  # dot 5, denominator 1, weight 1, cross product 9, accumulation 6
# interactions of the largest listed case (627,689 panels): draws stay below half of it
MOST_PAIRS = {"fp32c": 1.1e12, "fp64": 2.5e11}


def listed():
    return [
        # the drop-in BVERK4 call on the smallest grid the drivers' namelists use, all three target
        # classes: launches and host work
        dict(name="step_l2_fp64", kind="bve", precision="fp64", ic="rh4", level=2, refine=0, parity=True, delta=0.0,
             dt=0.01, steps=1),
        # Rossby-Haurwitz wave, level 4, ten steps: the plain-method benchmark
        dict(name="ten_steps_l4_fp64", kind="bve", precision="fp64", ic="rh4", level=4, refine=0, parity=False,
             delta=0.0, dt=0.01, steps=10),
        # a production FP64 step on a refined grid: panels, vertices and divided panels
        dict(name="step_l6_refined_fp64", kind="bve", precision="fp64", ic="rh4", level=6, refine=9001, parity=True,
             delta=0.01, dt=0.005, steps=1),
        # one velocity sum at the particles, arrays already on the device
        dict(name="vertex_sum_l5_fp64", kind="sum", target="vertex", precision="fp64", ic="gauss", level=5, refine=1111,
             delta=0.0),
        # the forced stratosphere model, a few steps
        dict(name="forced_l4_fp64", kind="forced", precision="fp64", level=4, refine=301, t=3.9, dt=0.01, steps=3),
        # the Voronoi step on its SoA generators (numbered as the particles of a level-5 grid)
        dict(name="voronoi_l5_fp64", kind="voronoi", precision="fp64", ic="gauss", level=5, dt=0.01, steps=1),
        # vector-Jacobian product of a run (cotangents of its end state, as data assimilation has
        # them): forward sweep, checkpoint recomputation, backward sweep
        dict(name="adjoint_l5_fp64", kind="adjoint", level=5, refine=0, delta=0.02, dt=0.005, steps=10, every=5),
        # FP32C on a small grid: the steps between two remeshes of a coarse run
        dict(name="five_steps_l4_fp32c", kind="resident", precision="fp32c", ic="gauss", level=4, refine=777, delta=0.01,
             dt=0.0025, steps=5),
        # FP32C, level 6 refined around the vortex
        dict(name="step_l6_refined_fp32c", kind="resident", precision="fp32c", ic="jet", level=6, refine=10007,
             delta=0.02, dt=0.005, steps=1),
        # FP32C, the level-7 Gaussian benchmark
        dict(name="step_l7_fp32c", kind="resident", precision="fp32c", ic="gauss", level=7, refine=0, delta=0.01,
             dt=0.005, steps=1),
        # FP32C, the largest: level 7 refined to 627,689 panels and about 314,000 particles
        dict(name="step_l7_refined_fp32c", kind="resident", precision="fp32c", ic="rh4", level=7, refine=100003,
             delta=0.005, dt=0.01, steps=1),
        # an ensemble of uneven grids advanced together
        dict(name="ensemble_fp32c", kind="ensemble", precision="fp32c", count=24, low=3, high=5, delta=0.0, dt=0.0025,
             steps=2),
    ]


def draw(rng):
    kind = rng.choice(["bve", "bve", "sum", "forced", "voronoi", "adjoint", "resident", "resident", "resident", "ensemble"])
    ic = rng.choice(["rh4", "gauss", "jet"])
    delta = rng.choice([0.0, 0.005, 0.01, 0.02])
    dt = rng.choice([0.005, 0.01])

    def size(lowest, highest):  # log-uniform active panels between 20*4^lowest and 20*4^highest
        n = 20.0 * 4.0 ** rng.uniform(lowest, highest)
        level = min(highest, max(lowest, int(math.log(n / 20.0, 4.0) + 1e-9)))
        return level, max(0, min(20 * 4 ** level, int((n - 20 * 4 ** level) / 3.0)))

    while True:
        if kind == "bve":
            level, refine = size(2, 6)
            case = dict(kind=kind, precision="fp64", ic=ic, level=level, refine=refine, parity=rng.random() < 0.5,
                        delta=delta if level < 6 else max(delta, 0.005), dt=dt if level < 6 else 0.005,
                        steps=rng.choice([1, 2, 4, 10]) if level < 5 else 1)
        elif kind == "sum":
            level, refine = size(2, 6)
            case = dict(kind=kind, target=rng.choice(["active", "vertex", "passive"]), precision="fp64", ic=ic,
                        level=level, refine=refine, delta=delta)
        elif kind == "forced":
            level, refine = size(2, 5)
            case = dict(kind=kind, precision="fp64", level=level, refine=refine, t=round(rng.uniform(0.0, 15.0), 3),
                        dt=0.01, steps=rng.choice([1, 2, 3]))
        elif kind == "voronoi":
            case = dict(kind=kind, precision="fp64", ic=ic, level=rng.randint(3, 6), dt=dt, steps=rng.choice([1, 2]))
        elif kind == "adjoint":
            level, refine = size(2, 4)
            case = dict(kind=kind, level=level, refine=refine, delta=max(delta, 0.01), dt=0.005,
                        steps=rng.choice([4, 7, 10]), every=rng.choice([2, 3, 5]))
        elif kind == "resident":
            level, refine = size(3, 7)
            case = dict(kind=kind, precision="fp32c", ic=ic, level=level, refine=refine,
                        delta=delta if level < 6 else max(delta, 0.005), dt=0.001 if level < 5 else 0.0025,
                        steps=rng.choice([1, 2, 5]) if level < 6 else 1)
        else:
            low = rng.randint(2, 4)
            case = dict(kind=kind, precision="fp32c", count=rng.randint(3, 40), low=low, high=low + rng.randint(1, 2),
                        delta=delta, dt=0.0025, steps=rng.choice([1, 2]))
        if pairs(case) <= MOST_PAIRS["fp32c" if kind in ("resident", "ensemble") else "fp64"]:
            return case


# ---------------------------------------------------------------------------
# grids and initial conditions
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=4)
def _icos(level):
    parts, pans = new_icos_grid(level)
    leaf = ~pans.hasChildren
    return parts.x, pans.vertices[leaf], pans.x[leaf], pans.area[leaf], pans.x[~leaf]


def _unit(v):
    return v / np.linalg.norm(v, axis=1, keepdims=True)


def _grid(level, refine, centre):
    """(xA, areaA, xV, xQ): the icosahedral grid with the `refine` leaf panels nearest to `centre`
    divided once more, as the drivers' refinement does: their four children go to the end of the
    list, the parents become divided panels."""
    V, tri, xA, area, xQ = _icos(level)
    if refine == 0:
        return xA.copy(), area.copy(), V.copy(), xQ.copy()
    pick = np.sort(np.argpartition(-(xA @ centre), refine - 1)[:refine])
    keep = np.ones(len(xA), bool)
    keep[pick] = False
    t = tri[pick]
    edges = np.sort(np.stack([t[:, [0, 1]], t[:, [1, 2]], t[:, [2, 0]]], 1), axis=2)
    key = edges[..., 0].astype(np.int64) * len(V) + edges[..., 1]
    uniq, inv = np.unique(key.ravel(), return_inverse=True)
    mids = _unit(V[uniq // len(V)] + V[uniq % len(V)])
    m = len(V) + inv.reshape(-1, 3)
    P = np.concatenate([V, mids])
    kids = np.stack([np.stack(c, 1) for c in ((t[:, 0], m[:, 0], m[:, 2]), (m[:, 0], t[:, 1], m[:, 1]),
                                              (m[:, 2], m[:, 1], t[:, 2]), (m[:, 0], m[:, 1], m[:, 2]))], 1).reshape(-1, 3)
    a, b, c = P[kids[:, 0]], P[kids[:, 1]], P[kids[:, 2]]
    num = np.abs(np.einsum("ij,ij->i", a, np.cross(b, c)))
    den = 1.0 + np.einsum("ij,ij->i", a, b) + np.einsum("ij,ij->i", b, c) + np.einsum("ij,ij->i", c, a)
    return (np.concatenate([xA[keep], _unit(a + b + c)]), np.concatenate([area[keep], 2.0 * np.arctan2(num, den)]),
            P, np.concatenate([xQ, xA[pick]]))


def _inputs(case, seed):
    """A grid as it is after some time of advection (every point moved by up to a tenth of the
    spacing, on the sphere) with its relative vorticity: (xA, zeta, areaA, xV, xQ)."""
    rng = np.random.default_rng(seed)
    patch = ics.sphere_point(np.deg2rad(22.5), 0.1 * case.get("refine", 0))  # the refined region
    centre = _unit((patch + rng.uniform(-0.1, 0.1, 3))[None])[0]              # the vortex in it
    xA, area, xV, xQ = _grid(case["level"], case.get("refine", 0), patch)
    h = 0.1 * math.sqrt(4.0 * math.pi / len(xA)) * (0.5 if case.get("refine") else 1.0)
    xA, xV, xQ = (_unit(x + h * rng.uniform(-1.0, 1.0, x.shape)) if len(x) else x for x in (xA, xV, xQ))
    ic = case.get("ic", "jet")
    if ic == "rh4":
        turn = rng.uniform(0.0, 2.0 * np.pi)
        c, s = np.cos(turn), np.sin(turn)
        z = ics.rh4_config(xA @ np.array([[c, -s, 0.0], [s, c, 0.0], [0.0, 0.0, 1.0]]))
    elif ic == "gauss":
        d = xA - centre
        z = np.exp(-16.0 * np.einsum("ij,ij->i", d, d))
        z -= ics.remove_area_mean(z, area)
    else:
        z = ics.jet_config(xA) + 1e-2 * rng.standard_normal(len(xA))
    return tuple(np.ascontiguousarray(v) for v in (xA, z, area, xV, xQ))


def _levels(case):
    """The levels of an ensemble's members, by the case alone."""
    rng = np.random.default_rng(case["count"] * 64 + case["low"] * 8 + case["high"])
    return [int(v) for v in rng.integers(case["low"], case["high"] + 1, case["count"])]


def _ensemble(case, seed):
    rng = np.random.default_rng(seed)
    out = []
    for k, level in enumerate(_levels(case)):
        xA, z, area, xV, _ = _inputs(dict(level=level, ic="gauss"), int(rng.integers(1 << 30)))
        out.append(Workload("m%d" % k, level, xA, z * rng.uniform(0.5, 2.0), area, xV, np.zeros((0, 3)), OMEGA,
                            (case["delta"],) * 3, case["dt"], case["steps"]))
    return out


def _deltas(case):
    if case["kind"] == "forced" or case.get("parity"):
        return (0.0 if case["kind"] == "forced" else case["delta"],) * 2 + (0.05,)
    return (case.get("delta", 0.0),) * 3


def _forced(case, seed):
    xA, _, area, xV, xQ = _inputs(case, seed)
    g = ics.stratosphere_rel_vort(xA)
    mean = ics.remove_area_mean(g, area)
    absA = np.ascontiguousarray(g - mean + 2.0 * OMEGA * xA[:, 2])
    absV = np.ascontiguousarray(ics.stratosphere_rel_vort(xV) - mean + 2.0 * OMEGA * xV[:, 2])
    return xA, absA, area, xV, absV, xQ


def _context(case):
    ctx = Context(0, case.get("precision", "fp64"))
    ctx.set_omega(OMEGA)
    ctx.set_deltas(*_deltas(case))
    return ctx


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    state = dict(case=case, ctx=_context(case))
    if kind == "ensemble":
        state["members"] = _ensemble(case, seed)
    elif kind == "forced":
        state["inputs"] = _forced(case, seed)
    elif kind == "voronoi":
        _, _, _, xV, _ = _inputs(dict(level=case["level"]), seed)
        n = len(xV)
        state["panels"] = _voronoi(case, xV, seed), n
    elif kind == "sum":
        xA, z, area, xV, xQ = _inputs(case, seed)
        X = xA if case["target"] == "active" else xV if case["target"] == "vertex" else xQ
        state["inputs"] = [torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (X, xA, z, area)]
        state["dX"] = torch.zeros((len(X), 3), dtype=torch.float64, device="cuda")
        state["dV"] = torch.zeros(len(X), dtype=torch.float64, device="cuda")
    elif kind == "adjoint":
        state["inputs"] = _cotangents(case, seed)
    else:
        xA, z, area, xV, xQ = _inputs(case, seed)
        if kind == "bve" and not case["parity"] or kind == "resident":
            xQ = np.zeros((0, 3))
        state["inputs"] = (xA, z, area, xV, xQ)
    return state


def _cotangents(case, seed):
    """A state and the cotangents of the state at the end: a misfit's gradient at every panel."""
    xA, z, area, _, _ = _inputs(case, seed)
    rng = np.random.default_rng(seed + 2)
    return xA, z, area, area[:, None] * rng.standard_normal(xA.shape), area * rng.standard_normal(len(xA))


def _voronoi(case, x, seed):
    """Generators as SoA arrays with a few unused slots, as type(VorPanels) holds them."""
    rng = np.random.default_rng(seed + 1)
    n, pad = len(x), 13
    centre = ics.sphere_point(np.deg2rad(rng.uniform(10.0, 40.0)), rng.uniform(0.0, 2.0 * np.pi))
    area = np.full(n, 4.0 * np.pi / n)
    if case["ic"] == "gauss":
        z = np.exp(-16.0 * np.sum((x - centre) ** 2, axis=1))
        z -= z.mean()
    else:
        z = ics.rh4_config(x) if case["ic"] == "rh4" else ics.jet_config(x)
    hold = [np.concatenate([v, np.zeros(pad)]) for v in (x[:, 0], x[:, 1], x[:, 2], z, np.zeros(n), area)]
    return VorPanels(*hold, N=n)


def run(state):
    case, ctx = state["case"], state["ctx"]
    kind = case["kind"]
    if kind == "bve":  # the drop-in call: host arrays in and out
        xA, z, area, xV, xQ = state["inputs"]
        xA, z, xV, xQ = xA.copy(), z.copy(), xV.copy(), xQ.copy()
        tke, ke = ctx.rk4_step(xA, z, area, xV, xQ, case["dt"], case["steps"])
        return dict(xA=xA, zeta=z, xV=xV, xQ=xQ, totalKE=tke, kineticEnergy=ke)
    if kind == "resident":  # a state kept on the device over the steps: what they leave is the state
        xA, z, area, xV, xQ = state["inputs"]
        ctx.rk4_load(xA, z, area, xV, xQ)
        ctx.rk4_advance(case["dt"], case["steps"])
        xA, z, xV, xQ = ctx.rk4_store(len(xA), len(xV), len(xQ))
        return dict(xA=xA, zeta=z, xV=xV)
    if kind == "forced":
        xA, absA, area, xV, absV, xQ = state["inputs"]
        xA, xV, xQ = xA.copy(), xV.copy(), xQ.copy()
        relA, relV, tke, ke = ctx.strat_rk4_step(xA, absA, area, xV, xQ, case["t"], case["dt"], case["steps"],
                                                 absVortV=absV)
        return dict(xA=xA, xV=xV, xQ=xQ, relA=relA, relV=relV, totalKE=tke, kineticEnergy=ke)
    if kind == "voronoi":
        p, n = state["panels"]
        q = VorPanels(p.x.copy(), p.y.copy(), p.z.copy(), p.relVort.copy(), p.absVort, p.area, n)
        tke, ke = BVERK4(ctx, q, case["dt"], case["steps"])
        return dict(x=q.x, y=q.y, z=q.z, zeta=q.relVort, totalKE=tke, kineticEnergy=ke)
    if kind == "sum":
        X, xA, z, area = state["inputs"]
        active = case["target"] == "active"
        cls = dict(active=N.TC_ACTIVE, vertex=N.TC_VERTEX, passive=N.TC_PASSIVE)[case["target"]]
        p = [ctypes.c_void_p(v.data_ptr()) for v in (X, xA, z, area, state["dX"], state["dV"])]
        N.call("tc_bs_velocity_device", ctx.handle, cls, None if active else p[0], len(X), p[1], p[2], p[3], len(xA),
               0, len(X), p[4], p[5] if active else None)
        return dict(dX=state["dX"], dV=state["dV"])
    if kind == "ensemble":
        members = [w.copy() for w in state["members"]]
        batch_rk4(ctx, members, case["dt"], case["steps"])
        return {k: np.concatenate([getattr(w, k) for w in members]) for k in ("xA", "zetaA", "xV")}
    if kind == "adjoint":
        xA, z, area, gTx, gTz = state["inputs"]
        J, gz, gx = np.zeros(1), np.zeros(len(xA)), np.zeros((len(xA), 3))
        N.call("tc_rk4_vjp", ctx.handle, N.dptr(xA), N.dptr(z), N.dptr(area), len(xA), case["dt"], case["steps"],
               case["every"], N.dptr(gTx), N.dptr(gTz), N.dptr(J), N.dptr(gz), N.dptr(gx))
        return dict(J=J, zeta=gz, x=gx)
    raise ValueError(kind)


# ---------------------------------------------------------------------------
# the floor of a pass
# ---------------------------------------------------------------------------
def _sizes(case):
    """(active, vertex, divided) points of the case's grid."""
    n, r = 20 * 4 ** case["level"], case.get("refine", 0)
    # a refined patch adds about 1.5 edges' midpoints per panel
    return n + 3 * r, n // 2 + 2 + (3 * r) // 2, (n - 20) // 3 + r


def pairs(case):
    """Interactions of one pass (adjoint: the forward sweep's and the backward sweep's)."""
    kind = case["kind"]
    if kind == "ensemble":
        return sum(4 * case["steps"] * n * (n + n // 2 + 2) for n in (20 * 4 ** v for v in _levels(case)))
    nA, nV, nQ = _sizes(case)
    if kind == "sum":
        return nA * dict(active=nA, vertex=nV, passive=nQ)[case["target"]]
    if kind == "voronoi":
        return 4 * case["steps"] * nV * nV
    if kind == "adjoint":
        return 8 * case["steps"] * nA * nA
    if kind == "resident" or kind == "bve" and not case["parity"]:
        nQ = 0
    return 4 * case["steps"] * nA * (nA + nV + nQ)


def work(case):
    if case["kind"] == "ensemble":
        points = sum(20 * 4 ** v * 3 // 2 for v in _levels(case))
    else:
        points = sum(_sizes(case))
    return {"bytes": 2.0 * 32.0 * points, "flops": FLOPS_PER_PAIR * pairs(case)}


# ---------------------------------------------------------------------------
# the same in 64 bits with plain torch
# ---------------------------------------------------------------------------
def _sum64(X, x, G, d2, same):
    """u_i = -1/(4 pi) sum_k x_i x x_k G_k / (1 - x_i.x_k + d2), k = i left out where `same`."""
    u = torch.empty_like(X)
    rows = max(1, (1 << 29) // max(1, len(x)))
    for a in range(0, len(X), rows):
        b = min(len(X), a + rows)
        w = X[a:b] @ x.T
        w.neg_().add_(1.0 + d2)
        if same:
            i = torch.arange(a, b, device=X.device)
            w[i - a, i] = math.inf
        w.reciprocal_().mul_(G)
        u[a:b] = torch.linalg.cross(X[a:b], w @ x)
    return u / (-4.0 * math.pi)


def _forcing64(x, t):
    tan1 = math.tan(math.pi / 3.0) ** 2
    if 0.0 <= t < 4.0:
        a = 0.5 * (1.0 - math.cos(math.pi / 4.0 * t))
    elif 4.0 <= t < 11.0:
        a = 1.0
    elif 11.0 <= t < 15.0:
        a = 0.5 * (1.0 - math.cos(math.pi / 4.0 * (t - 11.0) + math.pi))
    else:
        a = 0.0
    r = torch.hypot(x[:, 0], x[:, 1])
    lat = torch.atan2(x[:, 2], r)
    q = tan1 / torch.tan(lat) ** 2
    b = torch.where(lat > 0.0, q * torch.exp(1.0 - q), torch.zeros_like(q))
    b = torch.nan_to_num(b, nan=0.0)
    return 0.3 * 4.0 * math.pi * a * b * torch.where(r > 0.0, x[:, 0] / r, torch.ones_like(r))


def _rk4_64(xs, zeta, area, deltas, dt, steps, forced=None):
    """RK4 steps of [xA, xV, xQ] and zeta; `forced`: (absolute vorticity, start time)."""
    energies, ke = [], None
    for step in range(steps):
        X, Z, k_x, k_z = xs, zeta, [], []
        for s in range(4):
            if forced:
                t = forced[1] + step * dt + (0.0, 0.5, 0.5, 1.0)[s] * dt
                Z = forced[0] - 2.0 * OMEGA * X[0][:, 2] - _forcing64(X[0], t)
            u = [_sum64(X[c], X[0], Z * area, deltas[c] ** 2, c == 0) for c in range(3)]
            if s == 0:
                ke = (u[0] ** 2).sum(1)
                energies.append(0.5 * (ke * area).sum())
            k_x.append([dt * v for v in u])
            k_z.append(-2.0 * OMEGA * dt * u[0][:, 2])
            if s < 3:
                c = (0.5, 0.5, 1.0)[s]
                X = [a + c * k for a, k in zip(xs, k_x[s])]
                Z = zeta + c * k_z[s]
        w = (1.0 / 6.0, 1.0 / 3.0, 1.0 / 3.0, 1.0 / 6.0)
        xs = [a + sum(w[s] * k_x[s][c] for s in range(4)) for c, a in enumerate(xs)]
        zeta = zeta + sum(w[s] * k_z[s] for s in range(4))
    return xs, zeta, torch.stack(energies), ke


def _on_gpu(*arrays):
    return [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in arrays]


def exact(case, seed):
    kind = case["kind"]
    if pairs(case) > 3.0e11:
        return None
    with torch.no_grad():
        if kind == "bve" or kind == "resident":
            xA, z, area, xV, xQ = prepare_arrays(case, seed)
            xs, zeta, tke, ke = _rk4_64([xA, xV, xQ], z, area, _deltas(case), case["dt"], case["steps"])
            if kind == "resident":
                return dict(xA=xs[0], zeta=zeta, xV=xs[1])
            return dict(xA=xs[0], zeta=zeta, xV=xs[1], xQ=xs[2], totalKE=tke, kineticEnergy=ke)
        if kind == "forced":
            xA, absA, area, xV, absV, xQ = _on_gpu(*_forced(case, seed))
            xs, _, tke, ke = _rk4_64([xA, xV, xQ], absA, area, _deltas(case), case["dt"], case["steps"],
                                     (absA, case["t"]))
            t = case["t"] + case["steps"] * case["dt"]
            rel = [a - 2.0 * OMEGA * x[:, 2] - _forcing64(x, t) for a, x in ((absA, xs[0]), (absV, xs[1]))]
            return dict(xA=xs[0], xV=xs[1], xQ=xs[2], relA=rel[0], relV=rel[1], totalKE=tke, kineticEnergy=ke)
        if kind == "voronoi":
            p = _voronoi(case, _inputs(dict(level=case["level"]), seed)[3], seed)
            x, z, area = _on_gpu(np.stack([p.x, p.y, p.z], 1)[:p.N], p.relVort[:p.N], p.area[:p.N])
            none = x[:0]
            xs, zeta, tke, ke = _rk4_64([x, none, none], z, area, (0.0,) * 3, case["dt"], case["steps"])
            pad = torch.zeros(len(p.x) - p.N, dtype=torch.float64, device="cuda")
            soa = [torch.cat([v, pad]) for v in (xs[0][:, 0], xs[0][:, 1], xs[0][:, 2], zeta)]
            return dict(x=soa[0], y=soa[1], z=soa[2], zeta=soa[3], totalKE=tke, kineticEnergy=ke)
        if kind == "sum":
            xA, z, area, xV, xQ = _on_gpu(*_inputs(case, seed))
            X = xA if case["target"] == "active" else xV if case["target"] == "vertex" else xQ
            u = _sum64(X, xA, z * area, case["delta"] ** 2, case["target"] == "active")
            dV = -2.0 * OMEGA * u[:, 2] if case["target"] == "active" else torch.zeros_like(u[:, 0])
            return dict(dX=u, dV=dV)
        if kind == "ensemble":
            got = []
            for w in _ensemble(case, seed):
                xA, z, area, xV = _on_gpu(w.xA, w.zetaA, w.areaA, w.xV)
                xs, zeta, _, _ = _rk4_64([xA, xV, xA[:0]], z, area, (case["delta"],) * 3, case["dt"], case["steps"])
                got.append((xs[0], zeta, xs[1]))
            return {k: torch.cat([g[j] for g in got]) for j, k in enumerate(("xA", "zetaA", "xV"))}
    return _adjoint64(case, seed)


def prepare_arrays(case, seed):
    xA, z, area, xV, xQ = _inputs(case, seed)
    if case["kind"] == "resident" or not case["parity"]:
        xQ = np.zeros((0, 3))
    return _on_gpu(xA, z, area, xV, xQ)


def _adjoint64(case, seed):
    xA, z, area, gTx, gTz = _on_gpu(*_cotangents(case, seed))
    if len(xA) > 25000:
        return None
    d2, dt = case["delta"] ** 2, case["dt"]
    own = torch.eye(len(xA), dtype=torch.bool, device="cuda")

    def rate(x, zeta):
        D = (1.0 + d2 - x @ x.T).masked_fill(own, math.inf)
        u = torch.linalg.cross(x, (zeta * area / D) @ x) / (-4.0 * math.pi)
        return u, -2.0 * OMEGA * u[:, 2]

    xA.requires_grad_(True)
    z.requires_grad_(True)
    x, zeta = xA, z
    for _ in range(case["steps"]):
        X, Z, ks = x, zeta, []
        for s in range(4):
            k = checkpoint(rate, X, Z, use_reentrant=False)
            ks.append(k)
            if s < 3:
                c = (0.5, 0.5, 1.0)[s] * dt
                X, Z = x + c * k[0], zeta + c * k[1]
        w = (dt / 6.0, dt / 3.0, dt / 3.0, dt / 6.0)
        x = x + sum(c * k[0] for c, k in zip(w, ks))
        zeta = zeta + sum(c * k[1] for c, k in zip(w, ks))
    J = (gTx * x).sum() + (gTz * zeta).sum()
    J.backward()
    return dict(J=J.detach().reshape(1), zeta=z.grad, x=xA.grad)
