"""What a user of the framework has it do, as cases that can be timed and checked.

Each case goes through the package's public entry points.  The kinds:

* ``triangles``: 2D Euler on a triangle mesh.  The plain FP64 form is stepped
  as the reference's run loop steps it (``Solver.run``: the CFL step, then an
  SSP-RK3 step with its limiter); the mixed form with device-resident steps
  (``Solver.advance``); or, with ``host``, one step as the drop-in case model
  makes it, with the host vector as the state of record.
* ``scalar``: 2D scalar advection on triangles.
* ``line``: 1D advection or Euler on a line mesh, a whole small run in one
  launch (``run_resident``) or device-resident steps.
* ``batch``: many independent cases of uneven size and order in one batch.
* ``train``: training steps of the learned troubled-cell indicator.

``exact`` evaluates the same discretization in 64 bits with plain torch, from
the method's definition alone (bases, quadrature, HLLC, SSP-RK3, the WENO and
positivity limiter, the network).
"""
from __future__ import annotations

import math

import numpy as np
import torch

import wasl_b200
from wasl_b200 import cases as workloads
from wasl_b200 import meshgen

GAMMA = 1.4
CFL = 0.1
SENSOR, FLOOR, MIXED_FLOOR = 1e-3, 1e-10, 1e-5
BAND = (0.005, 0.999)  # the learned indicator's confidence band
DEVICE = "cuda" if torch.cuda.is_available() else "cpu"
F64 = torch.float64


def listed():
    return [
        # A tutorial-sized limited run with the drop-in form: every launch and
        # host round trip of the loop counts.
        {"name": "small limited drop-in", "kind": "triangles", "form": "plain", "order": 1,
         "quads": 24, "problem": "mild quadrant", "limited": True, "steps": 10},
        # The drop-in on the vortex benchmark's mesh (131,072 triangles).
        {"name": "vortex drop-in", "kind": "triangles", "form": "plain", "order": 2,
         "quads": 256, "problem": "vortex", "limited": False, "steps": 4},
        # The headline: the same mesh in the mixed form, device-resident steps.
        {"name": "vortex mixed", "kind": "triangles", "form": "mixed", "order": 2,
         "quads": 256, "problem": "vortex", "limited": False, "steps": 10},
        # One step of a case model whose state of record is the host's.
        {"name": "vortex host step", "kind": "triangles", "form": "mixed", "order": 2,
         "quads": 151, "problem": "vortex", "limited": False, "steps": 1, "host": True},
        # The largest: shocks with the limiter, P3 (500,000 triangles).
        {"name": "quadrants mixed", "kind": "triangles", "form": "mixed", "order": 3,
         "quads": 500, "problem": "quadrant", "limited": True, "steps": 4},
        # Milder quadrants in the drop-in form (which limits positivity in
        # troubled cells only), on an odd, smaller mesh.
        {"name": "quadrants drop-in", "kind": "triangles", "form": "plain", "order": 3,
         "quads": 161, "problem": "mild quadrant", "limited": True, "steps": 4},
        # Shock-vortex interaction with the learned indicator.
        {"name": "shock-vortex learned", "kind": "triangles", "form": "mixed", "order": 3,
         "quads": 300, "problem": "shock-vortex", "limited": True, "learned": True, "steps": 4},
        # A parameter study: independent cases of uneven size and order.
        {"name": "batch", "kind": "batch", "cases": 32, "smallest": 1000, "largest": 16000,
         "steps": 16},
        # The 400-cell advected pulse, a stretch of its one-launch run.
        {"name": "line pulse", "kind": "line", "equation": "scalar", "order": 2, "cells": 400,
         "resident": True, "steps": 3000},
        # Long 1D gas dynamics run, an odd cell count.
        {"name": "line gas", "kind": "line", "equation": "euler", "order": 2, "cells": 1000003,
         "resident": False, "steps": 4},
        # Scalar transport on triangles.
        {"name": "scalar square", "kind": "scalar", "order": 2, "quads": 509, "steps": 4},
        # Training the indicator on P3 features.
        {"name": "indicator training", "kind": "train", "order": 3, "samples": 60000,
         "batch": 4096, "steps": 16},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["triangles"] * 6 + ["scalar", "line", "line", "batch", "train"])
    if kind == "triangles":
        form = rng.choice(["plain", "mixed", "mixed"])
        problem = rng.choice(["vortex", "quadrant" if form == "mixed" else "mild quadrant",
                              "shock-vortex"])
        limited = problem != "vortex"
        case = {"kind": kind, "form": form, "order": rng.randint(1, 3),
                "quads": _log_int(rng, 20, 160 if form == "plain" else 350),
                "problem": problem, "limited": limited, "steps": rng.randint(2, 4)}
        if problem == "shock-vortex":
            case["quads"] = max(12, case["quads"] * 5 // 7)  # twice as many along x
            case["learned"] = form == "mixed" and rng.random() < 0.5
        elif not limited and rng.random() < 0.2:
            case.update(host=True, steps=1)
        return case
    if kind == "scalar":
        return {"kind": kind, "order": rng.randint(1, 3), "quads": _log_int(rng, 40, 500),
                "steps": rng.randint(2, 4)}
    if kind == "line":
        if rng.random() < 0.5:
            # three buffers of order + 1 modes a cell fit one CTA's shared memory
            return {"kind": kind, "equation": rng.choice(["scalar", "scalar", "euler"]),
                    "order": rng.randint(1, 3), "cells": _log_int(rng, 50, 480),
                    "resident": True, "steps": _log_int(rng, 200, 3000)}
        return {"kind": kind, "equation": rng.choice(["scalar", "euler"]),
                "order": rng.randint(1, 4), "cells": _log_int(rng, 3000, 1000000),
                "resident": False, "steps": rng.randint(2, 4)}
    if kind == "batch":
        return {"kind": kind, "cases": rng.randint(4, 32), "smallest": _log_int(rng, 200, 1000),
                "largest": _log_int(rng, 2000, 16000), "steps": rng.randint(2, 16)}
    return {"kind": kind, "order": rng.randint(1, 3), "samples": _log_int(rng, 5000, 60000),
            "batch": 64 * _log_int(rng, 4, 64), "steps": rng.randint(6, 16)}


# ---- inputs ----------------------------------------------------------------------

def _mesh(case, seed):
    n = case["quads"]
    if case["problem"] == "vortex":
        return meshgen.jittered_box(n, 0.0, 10.0, 0.0, 10.0, jitter=0.15, seed=seed)
    if case["problem"] == "shock-vortex":
        return meshgen.jittered_box(2 * n, 0.0, 2.0, 0.0, 1.0, jitter=0.15, seed=seed, ny=n)
    return meshgen.jittered_box(n, jitter=0.15, seed=seed)


def _conserved(rho, u, v, p):
    return torch.stack([rho, rho * u, rho * v, p / (GAMMA - 1.0) + 0.5 * rho * (u * u + v * v)], -1)


def _field(problem, seed):
    """Conserved values as a function of (x, y)."""
    rng = np.random.Generator(np.random.PCG64(seed))
    if problem == "vortex":
        cx, cy = rng.uniform(3.0, 7.0, 2)
        eps = 5.0

        def vortex(x, y):
            dx, dy = torch.remainder(x - cx + 5.0, 10.0) - 5.0, torch.remainder(y - cy + 5.0, 10.0) - 5.0
            bump = torch.exp(0.5 * (1.0 - dx * dx - dy * dy))
            t = 1.0 - (GAMMA - 1.0) * eps ** 2 / (8.0 * GAMMA * math.pi ** 2) * bump * bump
            rho = t ** (1.0 / (GAMMA - 1.0))
            k = eps / (2.0 * math.pi)
            return _conserved(rho, 1.0 - k * bump * dy, 1.0 + k * bump * dx, rho * t)
        return vortex
    if problem.endswith("quadrant"):
        if problem == "quadrant":
            states = workloads.QuadrantRiemann(seed=seed).states
        else:
            states = np.stack([workloads.conserved(rng.uniform(0.5, 1.2), *rng.uniform(-0.3, 0.3, 2),
                                                   rng.uniform(0.5, 1.2)) for _ in range(4)])
        states = torch.tensor(states, dtype=F64, device=DEVICE)
        return lambda x, y: states[(x >= 0.5).long() + 2 * (y >= 0.5).long()]
    if problem == "planar":
        w = workloads.PlanarRiemann(seed=seed)
        two = torch.tensor(np.stack([w.left, w.right]), dtype=F64, device=DEVICE)
        ca, sa = math.cos(w.angle), math.sin(w.angle)
        return lambda x, y: two[((x - w.cx) * ca + (y - w.cy) * sa >= 0.0).long()]
    w = workloads.ShockVortex(seed=seed)

    def shock(x, y):
        (ru, uu, _, pu), (rd, ud, _, pd) = w.upstream, w.downstream
        dx, dy = x - 0.25, y - 0.5
        bump = torch.exp(0.5 * (1.0 - (dx * dx + dy * dy) / 0.05 ** 2))
        c = math.sqrt(GAMMA * pu / ru)
        k = w.strength * c / 0.05
        t = 1.0 - (GAMMA - 1.0) * w.strength ** 2 / (2.0 * GAMMA) * bump * bump
        left = _conserved(ru * t ** (1.0 / (GAMMA - 1.0)), uu - k * bump * dy, k * bump * dx,
                          pu * t ** (GAMMA / (GAMMA - 1.0)))
        one = torch.ones_like(x)
        return torch.where((x < 0.5)[..., None], left, _conserved(rd * one, ud * one, 0.0 * one, pd * one))
    return shock


def _network(features, seed):
    """Seeded weights of the indicator: most smooth cells fall clearly below the band."""
    rng = np.random.Generator(np.random.PCG64(seed + 77))
    w1 = rng.normal(0.0, 1.0, (64, features)) * math.sqrt(2.0 / features)
    w2 = rng.normal(0.0, 1.0, (64, 64)) * math.sqrt(2.0 / 64)
    w3 = rng.normal(0.0, 1.0, 64) * math.sqrt(2.0 / 64)
    zeros = np.zeros(64)
    return np.concatenate([w1.ravel(), zeros, w2.ravel(), zeros, 4.0 * np.abs(w3), [-7.0]]).astype(np.float32)


def _features(order):
    raw = 4 * ((order + 1) * (order + 2) // 2 - 1) + 3
    return (raw + 15) // 16 * 16


def _samples(case, seed):
    """Features and flags as the sensor's data has them: modes over the mean,
    small in smooth cells, a quarter of the cells near a jump."""
    rng = np.random.Generator(np.random.PCG64(seed))
    n, order, f = case["samples"], case["order"], _features(case["order"])
    h = (order + 1) * (order + 2) // 2 - 1
    top = order + 1
    rough = rng.random(n) < 0.25
    size = np.where(rough, 10.0 ** rng.uniform(-1.5, -0.3, n), 10.0 ** rng.uniform(-5.0, -1.5, n))
    x = np.zeros((n, f), dtype=np.float32)
    x[:, :4 * h] = rng.normal(size=(n, 4 * h)) * size[:, None]
    x[:, 4 * h:4 * h + 3] = rng.normal(size=(n, 3)) * size[:, None]
    high = np.square(x[:, h - top:h].astype(np.float64)).sum(1)
    y = (high > SENSOR * (1.0 + np.square(x[:, :h].astype(np.float64)).sum(1))).astype(np.uint8)
    return np.clip(x, -8.0, 8.0), y


def _batch_shapes(case):
    """(quads per side, order) of each case: triangle counts spread over their
    logarithm, out of order."""
    n = case["cases"]
    ratio = case["largest"] / case["smallest"]
    return [(max(2, int(round(math.sqrt(0.5 * case["smallest"] * ratio ** (c * 7 % n / max(1, n - 1)))))),
             c % 3 + 1) for c in range(n)]


def _batch_inputs(case, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    out = []
    for n, order in _batch_shapes(case):
        s = int(rng.integers(1 << 30))
        arrays = meshgen.jittered_box(n, jitter=0.15, seed=s)
        out.append((arrays, order, _project(arrays, order, _field("planar", s))))
    return out


def _pulse(case, seed):
    """Smooth periodic modes on a line: the pulse, or an acoustic wave train."""
    rng = np.random.Generator(np.random.PCG64(seed))
    tags, x, segs = meshgen.jittered_line(case["cells"], jitter=0.2, seed=seed)
    phase = rng.uniform(0.0, 1.0)
    g, w = np.polynomial.legendre.leggauss(7)
    phi = _legendre(g, case["order"])
    at = 0.5 * (x[:-1] + x[1:])[:, None] + 0.5 * (x[1:] - x[:-1])[:, None] * g[None, :]
    y = np.mod(at - phase, 1.0)
    if case["equation"] == "scalar":
        u = (np.sin(2.0 * math.pi * y) + np.exp(-300.0 * (y - 0.5) ** 2))[None]
    else:
        rho = 1.0 + 0.2 * np.sin(2.0 * math.pi * y)
        v = 0.3 + 0.1 * np.cos(2.0 * math.pi * y)
        p = 1.0 + 0.1 * np.sin(4.0 * math.pi * y)
        u = np.stack([rho, rho * v, 0.0 * rho, p / (GAMMA - 1.0) + 0.5 * rho * v * v])
    return (tags, x, segs), np.einsum("q,veq,qm->vme", w, u, phi)


def _scalar_field(x, y):
    return (torch.sin(2.0 * math.pi * x) * torch.cos(2.0 * math.pi * y)
            + torch.exp(-100.0 * ((x - 0.5) ** 2 + (y - 0.5) ** 2)))[..., None]


VELOCITY = (1.0, 0.5)


class _Device:
    """The state's device memory as torch sees it: it lives as long as the
    solver, which a tensor over it keeps."""

    def __init__(self, solver):
        self.solver = solver
        self.__cuda_array_interface__ = {
            "shape": (solver.variables, solver.modes, solver.elements), "typestr": "<f8",
            "data": (solver.state_device_pointer(), False), "version": 3}


def _handle(solver):
    return {"solver": solver, "view": torch.as_tensor(_Device(solver), device="cuda"),
            "stream": torch.cuda.ExternalStream(solver.stream_handle())}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "triangles":
        arrays = _mesh(case, seed)
        mixed = case["form"] == "mixed"
        s = wasl_b200.Solver(*arrays, polynomial_order=case["order"], precision=case["form"],
                             boundary="periodic" if case["problem"] == "vortex" else "transmissive",
                             limiting=case["limited"], volume_rule_order=-1 if mixed else 0,
                             positivity_all=mixed and case["limited"])
        state = _project(arrays, case["order"], _field(case["problem"], seed)).cpu().numpy()
        s.set_state(state)
        if case["limited"]:
            s.limit()
        if case.get("learned"):
            s.set_indicator(_network(s.indicator_features(), seed), *BAND)
        h = _handle(s)
        h["host"] = s.get_state() if case.get("host") else None
        h["saved"] = h["view"].clone()
    elif kind == "scalar":
        arrays = meshgen.jittered_box(case["quads"], jitter=0.15, seed=seed)
        s = wasl_b200.Solver(*arrays, polynomial_order=case["order"], equation="scalar",
                             velocity=VELOCITY)
        s.set_state(_project(arrays, case["order"], _scalar_field).cpu().numpy())
        h = _handle(s)
    elif kind == "line":
        arrays, state = _pulse(case, seed)
        s = wasl_b200.Solver(*arrays, dimensions=1, equation=case["equation"],
                             polynomial_order=case["order"], velocity=(1.0, 0.0))
        s.set_state(state)
        h = _handle(s)
    elif kind == "batch":
        inputs = _batch_inputs(case, seed)
        b = wasl_b200.Batch([(*a, p) for a, p, _ in inputs], limiting=True, positivity_all=True)
        for c, (_, _, state) in enumerate(inputs):
            b.set_state(c, state.cpu().numpy())
        b.limit()
        h = {"batch": b}
    else:
        x, y = _samples(case, seed)
        net = wasl_b200.Mlp(x.shape[1], seed=seed)
        net.set_weights(_first_weights(case, seed))
        net.set_data(x, y)
        h = {"net": net}
    return {"case": case, **h}


def _first_weights(case, seed):
    w = _network(_features(case["order"]), seed)
    w[-65:-1] *= np.where(np.arange(64) % 2, 0.25, -0.25)
    w[-1] = 0.0
    return w


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "batch":
        b = state["batch"]
        b.advance(CFL, case["steps"])
        t, dt = b.times()
        return {"states": [b.get_state(c) for c in range(b.cases)], "time": t, "dt": dt}
    if kind == "train":
        loss = state["net"].train(case["steps"], batch=case["batch"], learning_rate=2e-3,
                                  positive_weight=8.0)
        return {"weights": state["net"].weights(), "loss": loss}
    s = state["solver"]
    if kind == "line" and case["resident"]:
        steps, t = s.run_resident(CFL, 0.0, 1e9, max_steps=case["steps"])
        return {"state": state["view"], "steps": steps, "time": t}
    if kind != "triangles":
        s.advance(CFL, case["steps"])
        return {"state": state["view"]}
    if case.get("host"):
        s.set_state(state["host"])
        dt = s.stable_dt(CFL)
        s.step(dt)
        return {"state": s.get_state(), "dt": dt}
    if case["limited"]:
        # From the same state each time: a flow with shocks does not run on for ever.
        with torch.cuda.stream(state["stream"]):
            state["view"].copy_(state["saved"])
    if case["form"] == "mixed":
        s.advance(CFL, case["steps"])
        return {"state": state["view"]}
    steps, t = s.run(CFL, 0.0, 1e9, max_steps=case["steps"])
    return {"state": state["view"], "steps": steps, "time": t}


# ---- what a pass cannot do without ------------------------------------------------

def _stage_work(elements, order, variables, dims, volume_points):
    """One RK step: each stage reads its input state and writes its output,
    stages 2 and 3 also read u^n; the mesh once per stage."""
    modes = (order + 1) * (order + 2) // 2 if dims == 2 else order + 1
    dof = elements * modes * variables
    mesh = 92.0 if dims == 2 else 8.0
    per_point = variables * modes * 2 * (3 if dims == 2 else 2) + 10 * variables
    faces = 1.5 * (order + 1) if dims == 2 else 1.0
    per_face = variables * modes * 8 + 40 * variables
    return {"bytes": 64.0 * dof + 3 * mesh * elements,
            "flops": 3.0 * elements * (volume_points * per_point + faces * per_face)}


def _elements(case):
    return 2 * case["quads"] ** 2 * (2 if case.get("problem") == "shock-vortex" else 1)


def work(case):
    kind, order = case["kind"], case.get("order", 2)
    if kind == "train":
        f = _features(order)
        weights = 64 * f + 64 * 64 + 3 * 64 + 1
        return {"bytes": case["steps"] * (4.0 * case["batch"] * f + 24.0 * weights),
                "flops": case["steps"] * case["batch"] * 6.0 * weights}
    if kind == "batch":
        each = [_stage_work(2 * n * n, p, 4, 2, (p + 1) ** 2) for n, p in _batch_shapes(case)]
        return {k: case["steps"] * sum(w[k] for w in each) for k in ("bytes", "flops")}
    if kind == "line":
        v = 4 if case["equation"] == "euler" else 1
        w = _stage_work(case["cells"], order, v, 1, order + 1)
        if case["resident"]:  # the state stays on the chip
            w["bytes"] = 16.0 * case["cells"] * (order + 1) * v / case["steps"]
    elif kind == "scalar":
        w = _stage_work(2 * case["quads"] ** 2, order, 1, 2, (order + 1) ** 2)
    else:
        points = (order + 3) ** 2 if case["form"] == "plain" else {1: 3, 2: 6, 3: 12}[order]
        w = _stage_work(_elements(case), order, 4, 2, points)
    return {k: case["steps"] * v for k, v in w.items()}


# ---- the method in 64 bits ----------------------------------------------------------

def _legendre(x, p):
    return np.stack([np.polynomial.legendre.legval(x, [0] * m + [1]) * math.sqrt(m + 0.5)
                     for m in range(p + 1)], -1)


def _jacobi(x, n, a):
    """Jacobi polynomials P_n^(a, 0)."""
    before, now = np.zeros_like(x), np.ones_like(x)
    for k in range(n):
        if k == 0:
            before, now = now, 0.5 * (a + (a + 2.0) * x)
            continue
        s = 2 * k + a
        nxt = ((s + 1) * (s * (s + 2) * x + a * a) * now - 2 * (k + a) * k * (s + 2) * before)
        before, now = now, nxt / (2 * (k + 1) * (k + a + 1) * s)
    return now


def _dubiner(xi, eta, p):
    """Orthonormal modes on the triangle (-1,-1), (1,-1), (-1,1), by degree n,
    then i; the collapsed coordinate a is -1 from the apex on (eta >= 1)."""
    half = 0.5 * (1.0 - eta)
    a = np.where(half > 0.0, (1.0 + xi) / np.where(half > 0.0, half, 1.0) - 1.0, -1.0)
    return np.stack([math.sqrt((2 * i + 1) * (n + 1) / 2.0) * _jacobi(a, i, 0) * half ** i
                     * _jacobi(eta, n - i, 2 * i + 1) for n in range(p + 1) for i in range(n + 1)], -1)


def _powers(p):
    return [(n - k, k) for n in range(p + 1) for k in range(n + 1)]


def _monomial_modes(p):
    """coefficients[power, mode] of the modes in the monomials xi^a eta^b."""
    g, _ = np.polynomial.legendre.leggauss(p + 2)
    b, a = np.meshgrid(g, g, indexing="ij")
    xi, eta = (0.5 * (a + 1.0) * (1.0 - b) - 1.0).ravel(), b.ravel()
    v = np.stack([xi ** i * eta ** j for i, j in _powers(p)], -1)
    return np.linalg.lstsq(v, _dubiner(xi, eta, p), rcond=None)[0]


def _gradient(xi, eta, p):
    zero = np.zeros_like(xi)
    dx = np.stack([i * xi ** (i - 1) * eta ** j if i else zero for i, j in _powers(p)], -1)
    dy = np.stack([j * xi ** i * eta ** (j - 1) if j else zero for i, j in _powers(p)], -1)
    c = _monomial_modes(p)
    return dx @ c, dy @ c


def _collapsed(order):
    g, w = np.polynomial.legendre.leggauss(order + 1)
    b, a = np.meshgrid(g, g, indexing="ij")
    wb, wa = np.meshgrid(w, w, indexing="ij")
    return (0.5 * (a + 1.0) * (1.0 - b) - 1.0).ravel(), b.ravel(), (wb * wa * 0.5 * (1.0 - b)).ravel()


def _symmetric(degree):
    """The fully symmetric rules of 3, 6 and 12 points (Dunavant, 1985), their
    published digits carried to 64 bits on the moment equations."""
    u = {2: [1 / 6, 1 / 3], 4: [0.44594849, 0.22338159, 0.09157621, 0.10995174],
         6: [0.24928675, 0.11678628, 0.06308901, 0.05084491, 0.31035245, 0.05314505, 0.08285108]}[degree]
    pairs = {2: 1, 4: 2, 6: 2}[degree]

    def points(x):
        out = []
        for k in range(pairs):
            a, w = x[2 * k], x[2 * k + 1]
            b = 1.0 - 2.0 * a
            out += [(a, a, b, w), (a, b, a, w), (b, a, a, w)]
        for k in range((len(x) - 2 * pairs) // 3):
            a, b, w = x[2 * pairs + 3 * k:2 * pairs + 3 * k + 3]
            c = 1.0 - a - b
            out += [(r, s, t, w) for r, s, t in ((a, b, c), (a, c, b), (b, a, c), (b, c, a), (c, a, b), (c, b, a))]
        return np.array(out)

    def moments(x):
        l = points(x)
        return np.array([(l[:, 3] * l[:, 0] ** i * l[:, 1] ** j).sum() - 2.0 * math.factorial(i)
                         * math.factorial(j) / math.factorial(i + j + 2)
                         for i in range(degree + 1) for j in range(degree + 1 - i)])

    u = np.array(u, dtype=np.float64)
    for _ in range(20):
        jac = np.stack([(moments(u + h) - moments(u - h)) / 2e-7
                        for h in 1e-7 * np.eye(len(u))], -1)
        u = u - np.linalg.lstsq(jac, moments(u), rcond=None)[0]
    l = points(u)
    return -1.0 + 2.0 * l[:, 1], -1.0 + 2.0 * l[:, 2], 2.0 * l[:, 3]


def _edges(p):
    """p + 1 Gauss points on each edge (0-1, 1-2, 2-0), in the direction round
    the triangle: (xi, eta) [3][p+1] and the 1D weights."""
    g, w = np.polynomial.legendre.leggauss(p + 1)
    t = 0.5 * (g + 1.0)
    corner = np.array([(-1.0, -1.0), (1.0, -1.0), (-1.0, 1.0)])
    at = np.stack([corner[k] + t[:, None] * (corner[(k + 1) % 3] - corner[k]) for k in range(3)])
    return at[..., 0], at[..., 1], w


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=F64, device=DEVICE)


def _project(arrays, order, field):
    """L2 projection of field(x, y) -> [..., variables] onto the modes."""
    _, xy, tris = arrays
    xi, eta, w = _collapsed(max(order, 5))
    v = _t(xy)[torch.as_tensor(tris - 1, device=DEVICE)]
    a, b = v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    at = v[:, None, 0] + 0.5 * (a[:, None] * _t(xi + 1.0)[:, None] + b[:, None] * _t(eta + 1.0)[:, None])
    weighted = _t(w[:, None] * _dubiner(xi, eta, order))
    return torch.einsum("eqv,qm->vme", field(at[..., 0], at[..., 1]), weighted).contiguous()


class _Triangles:
    """A triangle mesh's geometry, neighbours across edges and limiter stencil."""

    def __init__(self, arrays, periodic):
        _, xy, tris = arrays
        n = len(tris)
        v = xy[tris - 1]
        self.ne, self.v = n, _t(v)
        self.a, self.b = self.v[:, 1] - self.v[:, 0], self.v[:, 2] - self.v[:, 0]
        self.det = 0.25 * (self.a[:, 0] * self.b[:, 1] - self.a[:, 1] * self.b[:, 0])
        edge = torch.stack([self.v[:, (k + 1) % 3] - self.v[:, k] for k in range(3)], 1)
        self.length = torch.linalg.vector_norm(edge, dim=-1)
        self.nx, self.ny = edge[..., 1] / self.length, -edge[..., 0] / self.length
        self.altitude = 4.0 * self.det / self.length.amax(1)
        # The side across each side (element * 3 + edge), -1 on the boundary.
        ends = np.stack([tris, np.roll(tris, -1, 1)], -1).reshape(-1, 2)
        key = ends.min(1) * (len(xy) + 1) + ends.max(1)
        other = self._pairs(key, 3 * n)
        first = np.where(other >= 0, np.minimum(np.arange(3 * n), other), np.arange(3 * n))
        if periodic:
            lo, hi = xy.min(0), xy.max(0)
            mid = 0.5 * (xy[ends[:, 0] - 1] + xy[ends[:, 1] - 1])
            bound = np.nonzero(other < 0)[0]
            m = mid[bound]
            tol = 1e-9 * (hi - lo)
            on_x = (np.abs(m[:, 0] - lo[0]) < tol[0]) | (np.abs(m[:, 0] - hi[0]) < tol[0])
            along = np.where(on_x, m[:, 1], m[:, 0])
            key = np.round(along / (hi - lo).max() * 1e7).astype(np.int64) * 2 + on_x
            p = self._pairs(key, len(bound))
            other[bound] = bound[p]
            box = hi - lo
        else:
            box = np.zeros(2)
        self.box = box
        self.other = torch.as_tensor(other, device=DEVICE).view(n, 3)
        self.neighbour = torch.where(self.other >= 0, self.other // 3, -1)
        # The characteristic direction: the first face, in face order, with a neighbour.
        rank = torch.as_tensor(first, device=DEVICE).view(n, 3)
        rank = torch.where(self.other >= 0, rank, 1 << 60)
        best = rank.argmin(1, keepdim=True)
        self.cx, self.cy = self.nx.gather(1, best)[:, 0], self.ny.gather(1, best)[:, 0]

    @staticmethod
    def _pairs(key, n):
        order = np.argsort(key, kind="stable")
        same = np.nonzero(key[order[:-1]] == key[order[1:]])[0]
        other = np.full(n, -1, dtype=np.int64)
        other[order[same]], other[order[same + 1]] = order[same + 1], order[same]
        return other


def _primitive(s):
    inv = 1.0 / s[..., 0]
    u, v = s[..., 1] * inv, s[..., 2] * inv
    return u, v, (GAMMA - 1.0) * (s[..., 3] - 0.5 * (s[..., 1] * u + s[..., 2] * v))


def _flux(s, nx, ny):
    u, v, p = _primitive(s)
    un = u * nx + v * ny
    return torch.stack([s[..., 0] * un, s[..., 1] * un + p * nx, s[..., 2] * un + p * ny,
                        (s[..., 3] + p) * un], -1)


def _hllc(l, r, nx, ny):
    (ul, vl, pl), (ur, vr, pr) = _primitive(l), _primitive(r)
    a, b = ul * nx + vl * ny, ur * nx + vr * ny
    cl, cr = torch.sqrt(GAMMA * pl / l[..., 0]), torch.sqrt(GAMMA * pr / r[..., 0])
    sl, sr = torch.minimum(a - cl, b - cr), torch.maximum(a + cl, b + cr)
    ql, qr = l[..., 0] * (sl - a), r[..., 0] * (sr - b)
    star = (pr - pl + a * ql - b * qr) / (ql - qr)

    def side(s, u, v, p, un, wave, q):
        rho = q / (wave - star)
        shift = star - un
        e = s[..., 3] / s[..., 0] + shift * (star + p / q)
        t = torch.stack([rho, rho * (u + shift * nx), rho * (v + shift * ny), rho * e], -1)
        return _flux(s, nx, ny) + wave[..., None] * (t - s)

    f = torch.where((star >= 0.0)[..., None], side(l, ul, vl, pl, a, sl, ql),
                    side(r, ur, vr, pr, b, sr, qr))
    f = torch.where((sr <= 0.0)[..., None], _flux(r, nx, ny), f)
    return torch.where((sl >= 0.0)[..., None], _flux(l, nx, ny), f)


class _Method:
    """The modal discontinuous Galerkin residual and limiter on one mesh;
    states are [element][variable][mode]."""

    def __init__(self, mesh, order, rule, scalar=False):
        self.mesh, self.p, self.scalar = mesh, order, scalar
        xi, eta, w = rule
        self.phi, self.w = _t(_dubiner(xi, eta, order)), _t(w)
        gx, gy = _gradient(xi, eta, order)
        self.gx, self.gy = _t(gx), _t(gy)
        ex, ey, ew = _edges(order)
        self.edge, self.ew = _t(_dubiner(ex, ey, order)), _t(ew)
        self.top = order * (order + 1) // 2
        cx, cy, cw = _collapsed(order)
        self.rule = (_t(cx), _t(cy), _t(cw))
        self.target = _t(_dubiner(cx, cy, order))
        self.check = torch.cat([self.target, self.edge.reshape(-1, self.edge.shape[-1])])

    def residual(self, c):
        m = self.mesh
        s = torch.einsum("evm,qm->eqv", c, self.phi)
        if self.scalar:
            fx, fy = VELOCITY[0] * s, VELOCITY[1] * s
        else:
            zero, one = torch.zeros_like(s[..., 0]), torch.ones_like(s[..., 0])
            fx, fy = _flux(s, one, zero), _flux(s, zero, one)
        col = lambda x: (0.5 * x)[:, None, None] * self.w[:, None]
        fxi = col(m.b[:, 1]) * fx - col(m.b[:, 0]) * fy
        feta = col(m.a[:, 0]) * fy - col(m.a[:, 1]) * fx
        r = torch.einsum("eqv,qm->evm", fxi, self.gx) + torch.einsum("eqv,qm->evm", feta, self.gy)
        own = torch.einsum("evm,kqm->ekqv", c, self.edge)
        side = m.other.clamp(min=0)
        across = own.reshape(-1, *own.shape[2:])[side].flip(2)
        across = torch.where((m.other >= 0)[..., None, None], across, own)
        nx, ny = m.nx[..., None], m.ny[..., None]
        if self.scalar:
            speed = (VELOCITY[0] * nx + VELOCITY[1] * ny)[..., None]
            f = torch.where(speed >= 0.0, speed * own, speed * across)
        else:
            f = _hllc(own, across, nx, ny)
        weight = 0.5 * m.length[..., None] * self.ew
        r = r - torch.einsum("ekqv,kqm->evm", f * weight[..., None], self.edge)
        return r / m.det[:, None, None]

    def sensor(self, c):
        total, high = c[:, 0].square().sum(1), c[:, 0, self.top:].square().sum(1)
        return ~((total == 0.0) | (high / total <= SENSOR))

    def transforms(self, e, nb):
        """Projection matrices of the neighbours' modes onto the elements e."""
        m, (xi, eta, w) = self.mesh, self.rule
        at = m.v[e][:, None, 0] + 0.5 * (m.a[e][:, None] * (xi + 1.0)[:, None]
                                         + m.b[e][:, None] * (eta + 1.0)[:, None])
        away = m.v[e].mean(1) - m.v[nb].mean(1)
        box = _t(m.box)
        shift = torch.where(away.abs() > 0.5 * box, torch.sign(away) * box, 0.0) if m.box.any() else 0.0 * away
        d = at - (m.v[nb][:, 0] + shift)[:, None]
        a, b = m.a[nb][:, None], m.b[nb][:, None]
        det = a[..., 0] * b[..., 1] - a[..., 1] * b[..., 0]
        s = 2.0 * (b[..., 1] * d[..., 0] - b[..., 0] * d[..., 1]) / det - 1.0
        t = 2.0 * (a[..., 0] * d[..., 1] - a[..., 1] * d[..., 0]) / det - 1.0
        # (outside the neighbour the basis is its collapsed form's, not the polynomial)
        source = _t(_dubiner(s.cpu().numpy(), t.cpu().numpy(), self.p))
        return torch.einsum("q,qt,eqs->ets", w, self.target, source)

    def weno(self, c, e):
        """The limited modes of the troubled elements e."""
        m = self.mesh
        own = c[e]
        nx, ny = m.cx[e][:, None], m.cy[e][:, None]
        nb = m.neighbour[e]
        there = nb >= 0
        avg = own[:, None, :, 0] / math.sqrt(2.0)
        u, v, p = _primitive(avg)
        rho = avg[..., 0]
        un, ut = u * nx + v * ny, v * nx - u * ny
        c2 = GAMMA * p / rho
        cs, ke = torch.sqrt(c2), 0.5 * (un * un + ut * ut)

        def characteristic(d):
            nm, tm = d[:, 1] * nx + d[:, 2] * ny, d[:, 2] * nx - d[:, 1] * ny
            common = (GAMMA - 1.0) / c2 * (ke * d[:, 0] - un * nm - ut * tm + d[:, 3])
            diff = (un * d[:, 0] - nm) / cs
            return torch.stack([0.5 * (common + diff), d[:, 0] - common, tm - ut * d[:, 0],
                                0.5 * (common - diff)], 1)

        tc = characteristic(own)
        smooth = lambda d: d[:, :, 1:].square().sum(2, keepdim=True)
        count = there.sum(1)[:, None, None]
        weight = 0.5 / (1e-12 + smooth(tc)) ** 2
        total, value = weight, weight * tc
        for k in range(3):
            j = nb[:, k].clamp(min=0)
            cand = torch.einsum("ets,evs->evt", self.transforms(e, j), c[j])
            cand[:, :, 0] = own[:, :, 0]
            cc = characteristic(cand)
            w = torch.where(there[:, k, None, None], 0.5 / count.clamp(min=1) / (1e-12 + smooth(cc)) ** 2, 0.0)
            total, value = total + w, value + w * cc
        w = torch.where(count > 0, value / total, tc)
        h = (avg[..., 3] + p) / rho
        d0 = w[:, 0] + w[:, 1] + w[:, 3]
        nm = (un - cs) * w[:, 0] + un * w[:, 1] + (un + cs) * w[:, 3]
        tm = ut * d0 + w[:, 2]
        en = (h - un * cs) * w[:, 0] + ke * w[:, 1] + ut * w[:, 2] + (h + un * cs) * w[:, 3]
        out = torch.stack([d0, nx * nm - ny * tm, ny * nm + nx * tm, en], 1)
        out[:, :, 0] = own[:, :, 0]
        return out

    def positive(self, c, relative):
        """Density, then pressure, scaled towards the mean at the check points."""
        avg = c[:, :, 0] / math.sqrt(2.0)
        rf = (relative * avg[:, 0]).clamp(min=FLOOR)[:, None]
        pf = (relative * avg[:, 3]).clamp(min=FLOOR)[:, None]
        rho = torch.einsum("em,qm->eq", c[:, 0], self.check)
        scale = torch.where(rho < rf, (avg[:, :1] - rf) / (avg[:, :1] - rho), 1.0).amin(1)
        c = torch.cat([c[:, :, :1], c[:, :, 1:] * scale[:, None, None]], 2)
        s = torch.einsum("evm,qm->eqv", c, self.check)
        bad = _primitive(s)[2] < pf
        e, q = bad.nonzero(as_tuple=True)
        if len(e) == 0:
            return c
        mean, point, floor = avg[e], s[e, q], pf[e, 0]
        lower, upper = torch.zeros_like(floor), torch.ones_like(floor)
        for _ in range(64):
            middle = 0.5 * (lower + upper)
            ok = _primitive(mean + middle[:, None] * (point - mean))[2] >= floor
            lower, upper = torch.where(ok, middle, lower), torch.where(ok, upper, middle)
        scale = torch.ones_like(avg[:, 0]).scatter_reduce(0, e, lower, "amin")
        return torch.cat([c[:, :, :1], c[:, :, 1:] * scale[:, None, None]], 2)

    def network(self, c, weights, sensor):
        """The learned decision, the sensor's where the network is not confident."""
        rounded = lambda x: x.float().bfloat16().to(F64)
        f = _features(self.p)
        w = torch.as_tensor(weights, device=DEVICE)
        w1, b1, w2, b2, w3, b3 = (x.to(F64) for x in torch.split(w, [64 * f, 64, 4096, 64, 64, 1]))
        w1, w2, w3 = rounded(w1).view(64, f), rounded(w2).view(64, 64), rounded(w3)
        nb = self.mesh.neighbour
        mean, high = c[:, 0, 0], c[:, 0, 1:] / c[:, 0, :1]
        there, j = nb >= 0, nb.clamp(min=0)
        x = [high] + [torch.where(there[:, k, None], high[j[:, k]], 0.0) for k in range(3)]
        x += [torch.where(there, mean[j] / mean[:, None] - 1.0, 0.0)]
        x = rounded(torch.cat(x, 1).clamp(-8.0, 8.0))
        h = rounded(torch.relu(x @ w1[:, :x.shape[1]].T + b1))
        z = torch.relu(h @ w2.T + b2) @ w3 + b3
        p = torch.sigmoid(z)
        return (p >= BAND[1]) | ((p > BAND[0]) & sensor)

    def limit(self, c, relative=0.0, every=False, weights=None):
        troubled = self.sensor(c)
        if weights is not None:
            troubled = self.network(c, weights, troubled)
        e = troubled.nonzero()[:, 0]
        if len(e):
            c = c.index_copy(0, e, self.positive(self.weno(c, e), relative))
        return self.positive(c, relative) if every else c

    def speed(self, c):
        u, v, p = _primitive(c[:, :, 0] / math.sqrt(2.0))
        return torch.hypot(u, v) + torch.sqrt(GAMMA * p / (c[:, 0, 0] / math.sqrt(2.0)))


def _rk3(u, dt, residual, limit):
    e = limit(u + dt * residual(u))
    s = limit(0.75 * u + 0.25 * (e + dt * residual(e)))
    return limit(u / 3.0 + 2.0 / 3.0 * (s + dt * residual(s)))


def _storage_order(mesh):
    """The mixed form's storage order: along a Morton curve of the centroids."""
    v = mesh.v.cpu().numpy()
    x = (v[:, 0, 0] + v[:, 1, 0] + v[:, 2, 0]) / 3.0
    y = (v[:, 0, 1] + v[:, 1, 1] + v[:, 2, 1]) / 3.0
    scale = 65535.0 / max(x.max() - x.min(), y.max() - y.min())
    key = np.zeros(len(x), dtype=np.int64)
    qx, qy = ((x - x.min()) * scale).astype(np.int64), ((y - y.min()) * scale).astype(np.int64)
    for b in range(16):
        key |= ((qx >> b) & 1) << (2 * b) | ((qy >> b) & 1) << (2 * b + 1)
    return np.argsort(key, kind="stable")


def _exact_triangles(case, seed):
    arrays, order, mixed = _mesh(case, seed), case["order"], case["form"] == "mixed"
    mesh = _Triangles(arrays, case["problem"] == "vortex")
    m = _Method(mesh, order, _symmetric(2 * order) if mixed else _collapsed(order + 2))
    floor, every = (MIXED_FLOOR if mixed else 0.0), mixed
    c = _project(arrays, order, _field(case["problem"], seed)).permute(2, 0, 1).contiguous()
    weights = _network(_features(order), seed) if case.get("learned") else None
    limit = lambda x: x
    if case["limited"]:
        c = m.limit(c, floor, every)
        limit = lambda x: m.limit(x, floor, every, weights)
    length, t = mesh.altitude.min(), 0.0
    for _ in range(case["steps"]):
        dt = CFL * length / (m.speed(c).max() * (2 * order + 1))
        c, t = _rk3(c, dt, m.residual, limit), t + float(dt)
    if case.get("host"):
        return {"state": c.permute(1, 2, 0).reshape(-1), "dt": t}
    if mixed:
        return {"state": c[torch.as_tensor(_storage_order(mesh), device=DEVICE)].permute(1, 2, 0).contiguous()}
    return {"state": c.permute(1, 2, 0).contiguous(), "steps": None, "time": t}


def _exact_batch(case, seed):
    inputs = _batch_inputs(case, seed)
    states, times, dts = [], [], []
    for arrays, order, c in inputs:
        m = _Method(_Triangles(arrays, False), order, _collapsed(order))
        limit = lambda x: m.limit(x, MIXED_FLOOR, True)
        c, t, length = limit(c.permute(2, 0, 1).contiguous()), 0.0, m.mesh.altitude.min()
        for _ in range(case["steps"]):
            dt = CFL * length / (m.speed(c).max() * (2 * order + 1))
            c, t = _rk3(c, dt, m.residual, limit), t + dt
        states.append(c.permute(1, 2, 0).reshape(-1))
        times.append(t)
        dts.append(dt)
    return {"states": states, "time": torch.stack(times), "dt": torch.stack(dts)}


def _exact_scalar(case, seed):
    arrays, order = meshgen.jittered_box(case["quads"], jitter=0.15, seed=seed), case["order"]
    mesh = _Triangles(arrays, True)
    m = _Method(mesh, order, _collapsed(order), scalar=True)
    c = _project(arrays, order, _scalar_field).permute(2, 0, 1).contiguous()
    dt = CFL * mesh.altitude.min() / (math.hypot(*VELOCITY) * (2 * order + 1))
    for _ in range(case["steps"]):
        c = _rk3(c, dt, m.residual, lambda x: x)
    return {"state": c.permute(1, 2, 0).contiguous()}


def _exact_line(case, seed):
    (_, x, _), state = _pulse(case, seed)
    order, euler = case["order"], case["equation"] == "euler"
    c, x = _t(state), _t(x)  # [variable][mode][cell]
    h = x[1:] - x[:-1]
    g, w = np.polynomial.legendre.leggauss(order + 1 if euler else max(order, 1))
    phi = _t(_legendre(g, order))
    d = [np.polynomial.legendre.legval(g, np.polynomial.legendre.legder([0] * m + [1]))
         * math.sqrt(m + 0.5) for m in range(order + 1)]
    grad = _t(w[:, None] * np.stack(d, -1))
    lb, rb = _t(_legendre(np.array(-1.0), order)), _t(_legendre(np.array(1.0), order))
    one, zero = torch.ones((), dtype=F64, device=DEVICE), torch.zeros((), dtype=F64, device=DEVICE)

    def residual(c):
        s = torch.einsum("vme,qm->qev", c, phi)
        left, right = torch.einsum("vme,m->ev", c, lb), torch.einsum("vme,m->ev", c, rb)
        if euler:
            f = _flux(s, one, zero)
            face = _hllc(right, left.roll(-1, 0), one, zero)  # at each cell's right end
        else:
            f, face = s, right
        r = torch.einsum("qev,qm->vme", f, grad)
        r = r - torch.einsum("ev,m->vme", face, rb) + torch.einsum("ev,m->vme", face.roll(1, 0), lb)
        return r * (2.0 / h)

    t = 0.0
    length = h.min()
    for _ in range(case["steps"]):
        if euler:
            u, _, p = _primitive(c[:, 0].T / math.sqrt(2.0))
            speed = (u.abs() + torch.sqrt(GAMMA * p / (c[0, 0] / math.sqrt(2.0)))).max()
        else:
            speed = 1.0
        dt = CFL * length / (speed * (2 * order + 1))
        c, t = _rk3(c, dt, residual, lambda x: x), t + dt
    if case["resident"]:
        return {"state": c.contiguous(), "steps": None, "time": float(t)}
    return {"state": c.contiguous()}


def _exact_train(case, seed):
    x, y = _samples(case, seed)
    n, f, batch = len(x), x.shape[1], case["batch"]
    x, y = torch.as_tensor(x, device=DEVICE), _t(y)
    rounded = lambda a: a.float().bfloat16().to(F64)
    x = rounded(x)
    w = torch.as_tensor(_first_weights(case, seed), device=DEVICE).to(F64)
    m1, m2 = torch.zeros_like(w), torch.zeros_like(w)
    sizes = [64 * f, 64, 4096, 64, 64, 1]
    lr, cursor = 2e-3, 0
    for step in range(1, case["steps"] + 1):
        at = (cursor + torch.arange(batch, device=DEVICE)) % n
        cursor = (cursor + batch) % n
        xb, yb = x[at], y[at]
        w1, b1, w2, b2, w3, b3 = torch.split(w, sizes)
        w1, w2, w3 = rounded(w1).view(64, f), rounded(w2).view(64, 64), rounded(w3)
        h1 = rounded(torch.relu(xb @ w1.T + b1))
        h2 = torch.relu(h1 @ w2.T + b2)
        z = h2 @ w3 + b3
        cw = torch.where(yb > 0.0, 8.0, 1.0)
        loss = (cw * (torch.nn.functional.softplus(z) - yb * z)).mean()
        d3 = cw * (torch.sigmoid(z) - yb)
        d2 = (h2 > 0.0) * d3[:, None] * w3
        d1 = (h1 > 0.0) * (d2 @ w2)
        g = torch.cat([(d1.T @ xb).reshape(-1), d1.sum(0), (d2.T @ h1).reshape(-1), d2.sum(0),
                       h2.T @ d3, d3.sum()[None]]) / batch
        m1, m2 = 0.9 * m1 + 0.1 * g, 0.999 * m2 + 0.001 * g * g
        w = w - lr * (m1 / (1 - 0.9 ** step)) / (torch.sqrt(m2 / (1 - 0.999 ** step)) + 1e-8)
    return {"weights": w, "loss": float(loss)}


def exact(case, seed):
    return {"triangles": _exact_triangles, "batch": _exact_batch, "scalar": _exact_scalar,
            "line": _exact_line, "train": _exact_train}[case["kind"]](case, seed)
