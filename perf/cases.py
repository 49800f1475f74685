"""Performance cases of the HAL-CPP compute backend: what its users run, through
the Python binding (halcuda), at the sizes of the repository's benchmark, tests
and examples and over the ranges around them.

A case is a dict with a "kind":

* call     -- one call of a strategy interface on float64 host arrays, as a
              HAL model calls its backend every tick (copies included)
* explicit -- ticks of the resident explicit diffusion, then the field read back
* adi      -- ticks of the resident ADI diffusion, then the field read back; or
              (host) a whole run from and to pinned host memory
* agents   -- a whole run of the moving agents: upload, ticks, state read back
* coupled  -- agents and an ADI field that they feed on, as one call
* wells    -- a plate of independent wells with moving agents
* adjoint  -- loss of a variable-rate model, and its gradient
* pdegrid  -- ticks of the FP64 PDEGrid2D through its own calls

Inputs are made from the seed.  Their distributions are the benchmark's
(halcuda.workloads): uniform or Gaussian-blob fields, uniform sources, 70%
uniform and 30% clustered agents, smooth random rate fields.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hal-cpp_gb300"))
import halcuda as hal  # noqa: E402

N_BLOBS = 60
N_POINTS = 64
UPTAKE = 0.001
SPRING = 0.1
FRICTION = 0.5
MUL = hal.CELL_MUL
ADD = hal.CELL_ADD

# Limits that keep a drawn case within the largest listed one of its kind.
EXPLICIT_CELL_TICKS = 2048 * 2048 * 1000
ADI_CELL_TICKS = 2048 * 2048 * 200
AGENT_TICKS = 1_000_000 * 100
ADJOINT_CELL_STEPS = 512 * 512 * 500
PDEGRID_LINE_TICKS = 2048 * 20


# --------------------------------------------------------------------------
# cases


def listed():
    return [
        # One tick of a small model through IDiffusionBackend2D: the smallest
        # call, where latency counts.
        dict(name="call_diffuse_64", kind="call", op="diffuse", x=64, y=64, wrapX=False, wrapY=False),
        # One implicit tick of a mid-size, uneven grid, wrapped along x.
        dict(name="call_adi_1000x777", kind="call", op="adi", x=1000, y=777, wrapX=True, wrapY=False),
        # One force pass of a dense tissue on a 256^2 grid, bit-exact FP64.
        dict(name="call_forces_50k", kind="call", op="forces", x=256, y=256, agents=50000, radius=1.0,
             wrapX=False, wrapY=False),
        # The reference's small explicit model: fixed inflow on one edge, 64
        # point sources, 1000 ticks between two looks at the field.
        dict(name="explicit_256", kind="explicit", x=256, y=256, ticks=1000, wrapX=False, wrapY=False,
             dirichlet=True, source="points", advect=False),
        # A large explicit model, closed edges, a source in every cell.
        dict(name="explicit_2048", kind="explicit", x=2048, y=2048, ticks=1000, wrapX=False, wrapY=False,
             dirichlet=False, source="dense", advect=False),
        # The headline workload, from and to pinned host memory.
        dict(name="adi_2048_host", kind="adi", x=2048, y=2048, ticks=200, wrapX=False, wrapY=False,
             dirichlet=False, source=True, host=True),
        # A small implicit model on an uneven grid, wrapped along y.
        dict(name="adi_300x517", kind="adi", x=300, y=517, ticks=200, wrapX=False, wrapY=True,
             dirichlet=False, source=True, host=False),
        # A colony of 20000 cells on a torus.
        dict(name="agents_20k", kind="agents", x=256, y=256, agents=20000, ticks=100, radius=1.0, wrapX=True,
             wrapY=True),
        # A million cells that feed on an implicit field.
        dict(name="coupled_1m", kind="coupled", x=2048, y=2048, agents=1_000_000, ticks=100),
        # A 48-well plate, half explicit and half implicit, up to 20000 cells
        # in each well.
        dict(name="wells_48", kind="wells", wells=48, min_side=64, max_side=1024, max_agents=20000, ticks=100),
        # Parameter recovery: the gradient through 500 steps.
        dict(name="adjoint_512", kind="adjoint", x=512, y=512, steps=500, every=22, wrapX=False, wrapY=False,
             grad=True),
        # A model of the reference moved over as it is: FP64 PDEGrid2D calls.
        dict(name="pdegrid_adi_2048", kind="pdegrid", x=2048, y=2048, ticks=20, implicit=True, wrapX=False,
             wrapY=False, dirichlet=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _side(rng, lo, hi):
    """Log-uniform; two thirds of them as drawn (odd ones among them), one
    third rounded to the multiples of 32 that users like."""
    n = _log_int(rng, lo, hi)
    return max(lo, min(hi, (n + 16) // 32 * 32)) if rng.random() < 1.0 / 3.0 else n


def _coin(rng):
    return rng.random() < 0.5


def draw(rng):
    kind = rng.choice(["call", "explicit", "explicit", "adi", "adi", "agents", "coupled", "wells", "adjoint",
                       "pdegrid"])
    if kind == "call":
        op = rng.choice(["diffuse", "adi", "adi_exact", "forces", "diffuse_var", "advect"])
        c = dict(kind=kind, op=op, x=_side(rng, 64, 2048), y=_side(rng, 64, 2048), wrapX=_coin(rng),
                 wrapY=_coin(rng))
        if op == "forces":
            c.update(x=_side(rng, 64, 1024), y=_side(rng, 64, 1024), radius=rng.choice([1.0, 1.0, 2.0]))
            c["agents"] = _log_int(rng, 100, min(200000, 2 * c["x"] * c["y"]))
        return c
    if kind == "explicit":
        x, y = _side(rng, 64, 4096), _side(rng, 64, 4096)
        most = max(1, min(1000, EXPLICIT_CELL_TICKS // (x * y)))
        return dict(kind=kind, x=x, y=y, ticks=_log_int(rng, min(10, most), most), wrapX=_coin(rng),
                    wrapY=_coin(rng), dirichlet=_coin(rng), source=rng.choice(["none", "dense", "points"]),
                    advect=rng.random() < 0.25)
    if kind == "adi":
        x, y = _side(rng, 64, 4096), _side(rng, 64, 4096)
        most = max(1, min(500, ADI_CELL_TICKS // (x * y)))
        return dict(kind=kind, x=x, y=y, ticks=_log_int(rng, min(10, most), most), wrapX=_coin(rng),
                    wrapY=_coin(rng), dirichlet=rng.random() < 0.25, source=_coin(rng), host=_coin(rng))
    if kind == "agents":
        x, y = _side(rng, 64, 2048), _side(rng, 64, 2048)
        n = _log_int(rng, 500, min(1_000_000, x * y))
        return dict(kind=kind, x=x, y=y, agents=n, ticks=_log_int(rng, 10, min(200, AGENT_TICKS // n)),
                    radius=rng.choice([1.0, 1.0, 2.0]), wrapX=_coin(rng), wrapY=_coin(rng))
    if kind == "coupled":
        s = _side(rng, 128, 2048)
        return dict(kind=kind, x=s, y=s, agents=_log_int(rng, 1000, min(1_000_000, s * s)),
                    ticks=_log_int(rng, 10, 100))
    if kind == "wells":
        return dict(kind=kind, wells=rng.randint(4, 48), min_side=64, max_side=_log_int(rng, 128, 1024),
                    max_agents=_log_int(rng, 200, 20000), ticks=_log_int(rng, 10, 100))
    if kind == "adjoint":
        x, y = _side(rng, 64, 1024), _side(rng, 64, 1024)
        most = min(500, ADJOINT_CELL_STEPS // (x * y))
        return dict(kind=kind, x=x, y=y, steps=_log_int(rng, 20, most), every=rng.choice([0, 10, 22]),
                    wrapX=_coin(rng), wrapY=_coin(rng), grad=rng.random() < 0.75)
    x, y = _side(rng, 64, 2048), _side(rng, 64, 2048)
    return dict(kind="pdegrid", x=x, y=y, ticks=_log_int(rng, 2, min(50, PDEGRID_LINE_TICKS // max(x, y))),
                implicit=rng.random() < 0.75, wrapX=_coin(rng), wrapY=_coin(rng), dirichlet=rng.random() < 0.25)


# --------------------------------------------------------------------------
# inputs


def _rng(case, seed):
    return np.random.default_rng([int(seed), case["kind"].encode()[0], case.get("x", 0), case.get("y", 0)])


def _blobs(x, y, rng, count=N_BLOBS):
    """Sum of Gaussian blobs, float32, (x, y)."""
    scale = max(x, y) / 2048.0
    cx, cy = rng.random((count, 1)) * x, rng.random((count, 1)) * y
    sigma = (10.0 + rng.random((count, 1)) * 70.0) * scale
    amp = rng.random((count, 1))
    ex = amp * np.exp(-((np.arange(x) - cx) ** 2) / (2.0 * sigma * sigma))
    ey = np.exp(-((np.arange(y) - cy) ** 2) / (2.0 * sigma * sigma))
    return (ex.T.astype(np.float32) @ ey.astype(np.float32)).ravel()


def _uniform(n, rng, scale=1.0):
    return rng.random(n, dtype=np.float32) * np.float32(scale)


def _ghost(x, y, rng):
    """Boundary values of the four edges: an inflow of 1 on the x = -1 edge
    and small constants on the others."""
    g = np.zeros(2 * (x + y))
    g[:y] = 1.0
    g[y:2 * y] = 0.25 * rng.random()
    g[2 * y + x:] = 0.25 * rng.random()
    return g


def _positions(n, x, y, rng):
    """70% uniform, 30% in a Gaussian cluster, inside the domain; float32."""
    m = int(round(0.3 * n))
    dim = np.array([x, y], dtype=np.float64)
    uni = rng.random((n - m, 2)) * dim
    centre = rng.random(2) * dim
    clu = centre + rng.normal(0.0, 100.0 * max(x, y) / 2048.0, (m, 2))
    pos = np.concatenate([uni, clu]).astype(np.float32)
    hi = np.nextafter(dim.astype(np.float32), np.float32(0))
    pos = np.clip(pos, np.float32(0), hi)
    return np.ascontiguousarray(pos[rng.permutation(n)]).ravel()


def _rates(x, y, rng, lo=0.5, hi=5.0, modes=32):
    """Smooth random rate field in [lo, hi], float32, (x, y)."""
    kx, ky = rng.integers(-4, 5, (modes, 1)), rng.integers(-4, 5, (modes, 1))
    amp, phase = rng.standard_normal((modes, 1)), rng.random((modes, 1)) * 2.0 * np.pi
    ax = np.exp(2j * np.pi * kx * np.arange(x) / x + 1j * phase) * amp
    ay = np.exp(2j * np.pi * ky * np.arange(y) / y)
    acc = (ax.T @ ay).real
    acc = (acc - acc.min()) / max(acc.max() - acc.min(), 1e-12)
    return (lo + (hi - lo) * acc).astype(np.float32).ravel()


def _well_list(case, rng):
    """The plate's wells: sides log-uniform, half explicit and half implicit.
    A plate's sides and agent counts are the case's own; the rest is the
    seed's."""
    plate = np.random.default_rng([case["wells"], case["max_side"], case["max_agents"]])
    wells, fields, counts, pos = [], [], [], []
    ratio = case["max_side"] / case["min_side"]
    for i in range(case["wells"]):
        side = int(round(case["min_side"] * ratio ** plate.random()))
        adi = i % 2 == 1
        n = int(plate.integers(0, case["max_agents"] + 1))
        wells.append(dict(xDim=side, yDim=side, kind="adi" if adi else "explicit",
                          diffRate=float(rng.uniform(1.0, 10.0) if adi else rng.uniform(0.05, 0.24)),
                          decay=float(rng.uniform(0.0, 0.02)), maxAgents=n))
        fields.append(_uniform(side * side, rng))
        counts.append(n)
        hi = np.nextafter(np.float32(side), np.float32(0))
        pos.append(np.minimum(rng.random(2 * n, dtype=np.float32) * np.float32(side), hi))
    return wells, fields, np.array(counts, dtype=np.int32), np.concatenate(pos)


def _inputs(case, seed):
    """Every input of the case, as host arrays."""
    rng = _rng(case, seed)
    kind = case["kind"]
    if kind == "wells":
        wells, fields, counts, pos = _well_list(case, rng)
        return dict(wells=wells, fields=fields, counts=counts, pos=pos,
                    rad=np.full(pos.size // 2, 0.5, dtype=np.float32))
    x, y = case["x"], case["y"]
    n = x * y
    if kind == "call":
        if case["op"] == "forces":
            pos = _positions(case["agents"], x, y, rng).astype(np.float64)
            return dict(pos=pos, rad=np.full(case["agents"], 0.5 * case["radius"]))
        v = dict(field=rng.random(n), rate=5.0 if case["op"].startswith("adi") else 0.2)
        if case["op"] == "diffuse_var":
            v["rx"], v["ry"] = rng.random(n) * 0.25, rng.random(n) * 0.25
        if case["op"] == "advect":
            v["vx"], v["vy"] = 0.5 * rng.random() - 0.25, 0.5 * rng.random() - 0.25
        return v
    if kind == "explicit":
        v = dict(field=_uniform(n, rng), rate=0.2, decay=0.001, vx=0.0, vy=0.0)
        v["ghost"] = _ghost(x, y, rng) if case["dirichlet"] else None
        v["src"] = _uniform(n, rng, 0.001) if case["source"] == "dense" else None
        if case["source"] == "points":
            v["cells"] = rng.choice(n, N_POINTS, replace=False).astype(np.int32)
            v["values"] = np.full(N_POINTS, 0.05, dtype=np.float32)
        if case["advect"]:
            v["rate"], v["vx"], v["vy"] = 0.1, 0.2 * rng.random() - 0.1, 0.2 * rng.random() - 0.1
        return v
    if kind == "adi":
        return dict(field=_blobs(x, y, rng), src=_uniform(n, rng, 0.01) if case["source"] else None,
                    ghost=_ghost(x, y, rng) if case["dirichlet"] else None, rate=5.0, decay=0.01)
    if kind in ("agents", "coupled"):
        v = dict(pos=_positions(case["agents"], x, y, rng),
                 rad=np.full(case["agents"], 0.5 * case.get("radius", 1.0), dtype=np.float32))
        if kind == "coupled":
            v.update(field=_blobs(x, y, rng), src=_uniform(n, rng, 0.01), rate=5.0, decay=0.01)
        return v
    if kind == "adjoint":
        f0 = _blobs(x, y, rng, 40)
        return dict(f0=f0, target=(f0 * np.float32(0.5) + _blobs(x, y, rng, 40) * np.float32(0.5)),
                    D=_rates(x, y, rng), src=_uniform(n, rng, 0.01), decay=0.005)
    return dict(field=rng.random(n), rate=5.0 if case["implicit"] else 0.2, decay=0.01,
                ghost=_ghost(x, y, rng) if case["dirichlet"] else None,
                cells=rng.choice(n, N_POINTS, replace=False).astype(np.int32), values=rng.random(N_POINTS) * 0.05)


# --------------------------------------------------------------------------
# what a program keeps, and one pass of it


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.from_numpy(a).dtype, pin_memory=True)
    out = t.numpy()
    out[...] = a
    return t, out


def prepare(case, seed):
    v = _inputs(case, seed)
    kind = case["kind"]
    st = dict(case=case, v=v)
    if kind == "wells":
        st["h"] = h = hal.Wells(v["wells"])
        for i, f in enumerate(v["fields"]):
            h.set_field(i, f)
        h.set_agents(v["counts"], v["pos"], v["rad"])
        h.set_motion(True, FRICTION)
        return st
    x, y = case["x"], case["y"]
    if kind == "call":
        if case["op"] == "forces":
            st["h"] = hal.Agents(x, y, case["agents"])
        elif case["op"].startswith("adi"):
            st["h"] = hal.Adi(x, y)
            st["h"].set_exact(case["op"] == "adi_exact")
        else:
            st["h"] = hal.Diffusion(x, y)
        st["deltas"] = np.zeros(x * y)
    elif kind == "explicit":
        st["h"] = h = hal.Diffusion(x, y)
        h.set_field(v["field"])
        if v["src"] is not None:
            h.set_source(v["src"])
        if "cells" in v:
            h.set_point_sources(v["cells"], v["values"])
        if v["ghost"] is not None:
            h.set_dirichlet(v["ghost"])
        if case["advect"]:
            h.set_velocity(v["vx"], v["vy"])
    elif kind == "adi":
        st["h"] = h = hal.Adi(x, y)
        if v["ghost"] is not None:
            h.set_dirichlet(v["ghost"])
        if case["host"]:
            st["keep"], st["field"] = _pinned(v["field"])
            st["keep_src"], st["src"] = _pinned(v["src"]) if v["src"] is not None else (None, None)
        else:
            h.set_field(v["field"])
            if v["src"] is not None:
                h.set_source(v["src"])
    elif kind in ("agents", "coupled"):
        st["h"] = hal.Agents(x, y, case["agents"])
        if kind == "coupled":
            st["adi"] = a = hal.Adi(x, y)
            a.set_source(v["src"])
            a.set_uptake(st["h"], UPTAKE)
    elif kind == "adjoint":
        st["h"] = hal.Adjoint(x, y, case["wrapX"], case["wrapY"])
        st["h"].set_problem(v["f0"], v["target"], case["steps"], case["every"])
    else:
        st["h"] = hal.PDEGrid(x, y, case["wrapX"], case["wrapY"])
        st["h"].set_state(v["field"])
    return st


def run(st):
    case, v, h = st["case"], st["v"], st["h"]
    kind = case["kind"]
    if kind == "call":
        op, x, y, wx, wy = case["op"], case["x"], case["y"], case["wrapX"], case["wrapY"]
        if op == "forces":
            return h.accumulate_forces(v["pos"], v["rad"], case["radius"], SPRING, x, y, wx, wy)
        if op == "diffuse":
            return h.diffuse(v["field"], st["deltas"], v["rate"], x, y, wx, wy)
        if op == "diffuse_var":
            return h.diffuse_var(v["field"], st["deltas"], v["rx"], v["ry"], wx, wy)
        if op == "advect":
            return h.advect(v["field"], st["deltas"], v["vx"], v["vy"], wx, wy)
        return h.diffuse_adi(v["field"], st["deltas"], v["rate"], x, y, wx, wy)
    if kind == "explicit":
        h.run_ticks(case["ticks"], v["rate"], v["decay"], case["wrapX"], case["wrapY"])
        return h.get_field()
    if kind == "adi":
        args = (case["ticks"], v["rate"], v["decay"], case["wrapX"], case["wrapY"])
        if case["host"]:
            return h.run_ticks_host(st["field"], st["src"], *args)
        h.run_ticks(*args)
        return h.get_field()
    if kind == "agents":
        h.upload(v["pos"], v["rad"])
        h.set_velocities()
        h.step(case["ticks"], case["radius"], SPRING, case["wrapX"], case["wrapY"], friction=FRICTION)
        return h.get_state()
    if kind == "coupled":
        a = st["adi"]
        h.upload(v["pos"], v["rad"])
        h.set_velocities()
        a.set_field(v["field"])
        a.run_coupled(h, case["ticks"], v["rate"], v["decay"], False, False, 1.0, SPRING, FRICTION, -1.0)
        return a.get_field(), h.get_state()
    if kind == "wells":
        h.set_agents(v["counts"], v["pos"], v["rad"])
        h.set_velocities()
        h.run_ticks(case["ticks"], 1.0, SPRING)
        return [h.get_field(i) for i in range(case["wells"])], h.get_agents()
    if kind == "adjoint":
        if case["grad"]:
            return h.gradient(v["D"], v["decay"], v["src"])
        return h.forward(v["D"], v["decay"], v["src"], want_field=True)
    for _ in range(case["ticks"]):
        if case["implicit"]:
            h.diffusion_adi(v["rate"], v["ghost"])
        else:
            h.diffusion(v["rate"], v["ghost"])
        h.apply(v["cells"], v["values"], op=ADD)
        h.apply_all(MUL, -v["decay"])
        h.update()
    return h.get_state()


def work(case):
    """Bytes: every input read once and every output written once.  Operations:
    9 per cell of an explicit tick (4 differences, 3 sums, the rate and the
    commit) and 2 for the decay; 26 per cell of an ADI tick (two right-hand
    sides of 5, two eliminations and substitutions of 7, and the commit);
    about 20 per pair of agents within reach of each other, and 10 per move."""
    kind = case["kind"]
    if kind == "wells":
        ratio = case["max_side"] / case["min_side"]
        mean = case["min_side"] ** 2 * ((ratio ** 2 - 1.0) / (2.0 * math.log(ratio)) if ratio > 1 else 1.0)
        cells, agents = case["wells"] * mean, case["wells"] * case["max_agents"] / 2
        return {"bytes": 8.0 * cells + 28.0 * agents, "flops": case["ticks"] * (cells * 18.5 + agents * 50.0)}
    n = case["x"] * case["y"]
    if kind == "call":
        if case["op"] == "forces":
            m = case["agents"]
            near = m / n * math.pi * case["radius"] ** 2
            return {"bytes": 40.0 * m, "flops": m * (10.0 + 20.0 * near)}
        arrays = 5 if case["op"] == "diffuse_var" else 3
        return {"bytes": 8.0 * arrays * n, "flops": (26.0 if case["op"].startswith("adi") else 9.0) * n}
    if kind == "explicit":
        return {"bytes": 4.0 * n * (3 if case["source"] == "dense" else 2), "flops": 11.0 * n * case["ticks"]}
    if kind == "adi":
        return {"bytes": 4.0 * n * (3 if case["source"] else 2), "flops": 26.0 * n * case["ticks"]}
    if kind == "agents":
        m = case["agents"]
        near = m / n * math.pi * case["radius"] ** 2
        return {"bytes": 28.0 * m, "flops": case["ticks"] * m * (10.0 + 20.0 * near)}
    if kind == "coupled":
        m = case["agents"]
        return {"bytes": 12.0 * n + 28.0 * m,
                "flops": case["ticks"] * (26.0 * n + m * (10.0 + 20.0 * math.pi * m / n))}
    if kind == "adjoint":
        return {"bytes": 4.0 * n * (6 if case["grad"] else 4), "flops": (100.0 if case["grad"] else 30.0) * n * case["steps"]}
    return {"bytes": 8.0 * 3 * n, "flops": (26.0 if case["implicit"] else 11.0) * n * case["ticks"]}


# --------------------------------------------------------------------------
# the same in plain 64-bit torch


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a), device="cuda").to(torch.float64)


def _edges(g, x, y):
    """(x = -1, x = xDim, y = -1, y = yDim) boundary values, or four None."""
    if g is None:
        return None, None, None, None
    g = _dev(g)
    return g[:y], g[y:2 * y], g[2 * y:2 * y + x], g[2 * y + x:]


def _diffs(f, dim, wrap, lo, hi):
    """f[+1] - f and f[-1] - f along an axis; past a closed edge 0, or twice the
    difference to the boundary value."""
    up, dn = torch.roll(f, -1, dim) - f, torch.roll(f, 1, dim) - f
    if not wrap:
        n = f.shape[dim]
        up.select(dim, n - 1).copy_(2 * (hi - f.select(dim, n - 1)) if hi is not None else torch.zeros_like(f.select(dim, 0)))
        dn.select(dim, 0).copy_(2 * (lo - f.select(dim, 0)) if lo is not None else torch.zeros_like(f.select(dim, 0)))
    return up, dn


def _line_inverse(n, rate, wrap, dirichlet):
    """Inverse of I - rate/2 L for one line, L the 3-point Laplacian."""
    L = torch.zeros(n, n, dtype=torch.float64, device="cuda")
    i = torch.arange(n, device="cuda")
    for s in (1, -1):
        j = (i + s) % n
        ok = torch.ones(n, dtype=torch.bool, device="cuda") if wrap else (i + s >= 0) & (i + s < n)
        L.index_put_((i[ok], j[ok]), torch.ones(int(ok.sum()), dtype=torch.float64, device="cuda"), accumulate=True)
        L.index_put_((i[ok], i[ok]), -torch.ones(int(ok.sum()), dtype=torch.float64, device="cuda"), accumulate=True)
    if dirichlet and not wrap:
        L[0, 0] -= 2.0
        L[n - 1, n - 1] -= 2.0
    return torch.linalg.inv(torch.eye(n, dtype=torch.float64, device="cuda") - 0.5 * rate * L)


class _AdiStep:
    """v of one ADI step: (I - Ly/2) v = (I + Lx/2) w, (I - Lx/2) w = (I + Ly/2) f."""

    def __init__(self, x, y, rate, wrapX, wrapY, ghost=None):
        self.rate, self.wx, self.wy = rate, wrapX, wrapY
        self.g = _edges(ghost, x, y)
        self.ix = _line_inverse(x, rate, wrapX, ghost is not None)
        self.iy = _line_inverse(y, rate, wrapY, ghost is not None)

    def __call__(self, f):
        h = 0.5 * self.rate
        xl, xh, yl, yh = self.g
        a, b = _diffs(f, 1, self.wy, yl, yh)
        d = f + h * (a + b)
        if xl is not None and not self.wx:
            d[0] += 2 * h * xl
            d[-1] += 2 * h * xh
        w = self.ix @ d
        a, b = _diffs(w, 0, self.wx, xl, xh)
        d = w + h * (a + b)
        if yl is not None and not self.wy:
            d[:, 0] += 2 * h * yl
            d[:, -1] += 2 * h * yh
        return d @ self.iy.T


def _pair_forces(p, rad, xd, yd, base, wrapX, wrapY, reach, spring):
    """Force on each agent from those of its domain within `reach`: p (n, 2);
    xd, yd, base: per-agent sides and first cell of its domain."""
    cx = torch.minimum(p[:, 0].floor().long().clamp_min(0), xd - 1)
    cy = torch.minimum(p[:, 1].floor().long().clamp_min(0), yd - 1)
    cell = base + cx * yd + cy
    order = torch.argsort(cell, stable=True)
    sp, sr, sc = p[order], rad[order], cell[order]
    cells = int((base + xd * yd).max())
    count = torch.bincount(sc, minlength=cells)
    start = torch.cumsum(count, 0) - count
    out = torch.zeros_like(p)
    fx, fy = xd.to(p.dtype), yd.to(p.dtype)
    k = int(math.ceil(reach))
    for dx in range(-k, k + 1):
        for dy in range(-k, k + 1):
            qx, qy = cx + dx, cy + dy
            ok = torch.ones_like(qx, dtype=torch.bool)
            if wrapX:
                qx = qx % xd
            else:
                ok &= (qx >= 0) & (qx < xd)
            if wrapY:
                qy = qy % yd
            else:
                ok &= (qy >= 0) & (qy < yd)
            q = torch.where(ok, base + qx * yd + qy, base)
            n = torch.where(ok, count[q], 0)
            me, s = torch.nonzero(n, as_tuple=True)[0], 0
            while me.numel():
                j = start[q[me]] + s
                a, b = p[me], sp[j]
                d = b - a
                if wrapX:
                    w = fx[me]
                    d[:, 0] = torch.where(d[:, 0].abs() > 0.5 * w, d[:, 0] - torch.sign(d[:, 0]) * w, d[:, 0])
                if wrapY:
                    w = fy[me]
                    d[:, 1] = torch.where(d[:, 1].abs() > 0.5 * w, d[:, 1] - torch.sign(d[:, 1]) * w, d[:, 1])
                r = d.square().sum(1).sqrt()
                near = (r < reach) & (r > 0) & (order[j] != me)
                f = torch.where(near, spring * (rad[me] + sr[j] - r) / torch.where(near, r, 1.0), 0.0)
                out.index_add_(0, me, -d * f[:, None])
                s += 1
                me = me[n[me] > s]
    return out, cell


def _move(p, v, dv, xd, yd, wrapX, wrapY, friction):
    v = v + dv
    q = p + v
    for k, (dim, wrap) in enumerate(((xd.to(p.dtype), wrapX), (yd.to(p.dtype), wrapY))):
        c = q[:, k]
        inside = (c >= 0) & (c < dim)
        q[:, k] = torch.where(inside, c, torch.remainder(c, dim) if wrap else p[:, k])
    return q, v * friction


def _ones(n, value):
    return torch.full((n,), int(value), dtype=torch.long, device="cuda")


def _explicit_tick(f, rate, decay, wx, wy, g, src, vx=0.0, vy=0.0):
    xl, xh, yl, yh = g
    px, mx = _diffs(f, 0, wx, xl, xh)
    py, my = _diffs(f, 1, wy, yl, yh)
    d = (rate + max(-vx, 0.0)) * px + (rate + max(vx, 0.0)) * mx + (rate + max(-vy, 0.0)) * py
    d += (rate + max(vy, 0.0)) * my
    d -= decay * f
    return f + (d if src is None else d + src)


class _VarLines:
    """(I + L/2) and the inverse of (I - L/2) along one axis of a field of
    rates, each face carrying the rate of the cell before it."""

    def __init__(self, e, wrap):
        # e (lines, n): face (j, j+1); the last one only when wrapped
        self.e = e.clone()
        if not wrap:
            self.e[:, -1] = 0.0
        m, n = e.shape
        lo = torch.roll(self.e, 1, 1)
        b = 1.0 + 0.5 * (self.e + lo)
        a = -0.5 * lo
        c = -0.5 * self.e
        if wrap:  # rank-one split of the corners
            gamma = -b[:, 0].clone()
            a0, cn = a[:, 0].clone(), c[:, -1].clone()
            b[:, 0] -= gamma
            b[:, -1] -= a0 * cn / gamma
        inv = torch.eye(n, dtype=torch.float64, device="cuda").repeat(m, 1, 1).permute(1, 0, 2).contiguous()
        cp = torch.empty(n, m, dtype=torch.float64, device="cuda")
        inv[0] /= b[:, :1]
        cp[0] = c[:, 0] / b[:, 0]
        for j in range(1, n):
            den = b[:, j] - a[:, j] * cp[j - 1]
            cp[j] = c[:, j] / den
            inv[j] = (inv[j] - a[:, j, None] * inv[j - 1]) / den[:, None]
        for j in range(n - 2, -1, -1):
            inv[j] -= cp[j][:, None] * inv[j + 1]
        inv = inv.permute(1, 0, 2).contiguous()
        if wrap:
            u = inv[:, :, 0] * gamma[:, None] + inv[:, :, -1] * cn[:, None]
            r = a0 / gamma
            vt = inv[:, 0, :] + r[:, None] * inv[:, -1, :]
            s = 1.0 + u[:, 0] + r * u[:, -1]
            inv -= u[:, :, None] * (vt / s[:, None])[:, None, :]
        self.inv = inv

    def apply(self, u):
        d = self.e * (torch.roll(u, -1, 1) - u)
        return u + 0.5 * (d - torch.roll(d, 1, 1))

    def solve(self, d):
        return torch.bmm(self.inv, d[:, :, None])[:, :, 0]

    def face(self, p, q):
        g = -0.5 * (torch.roll(p, -1, 1) - p) * (torch.roll(q, -1, 1) - q)
        return g * (self.e != 0)


def _adjoint(case, v):
    x, y, steps = case["x"], case["y"], case["steps"]
    D, f, target, src = (_dev(v[k]).view(x, y) for k in ("D", "f0", "target", "src"))
    decay = float(v["decay"])
    lx, ly = _VarLines(D.T.contiguous(), case["wrapX"]), _VarLines(D, case["wrapY"])
    kept = []
    for _ in range(steps):
        w = lx.solve(ly.apply(f).T.contiguous())
        t = ly.solve(lx.apply(w).T.contiguous())
        if case["grad"]:
            kept.append((f, w, t))
        f = f + ((t - f) - decay * f + src)
    r = f - target
    loss = 0.5 * float(r.square().sum())
    if not case["grad"]:
        return loss, f.reshape(-1)
    g, gD, gS, gK = r, torch.zeros_like(r), torch.zeros_like(r), 0.0
    for ft, w, t in reversed(kept):
        gS = gS + g
        gK = gK - (g * ft).sum()
        b2 = ly.solve(g)
        gD += ly.face(b2, t)
        b2x = b2.T.contiguous()
        gx = lx.face(b2x, w)
        b1 = lx.solve(lx.apply(b2x))
        gx += lx.face(b1, w)
        gD += gx.T
        b1 = b1.T.contiguous()
        gD += ly.face(b1, ft)
        g = ly.apply(b1) - decay * g
    return loss, gD.reshape(-1), float(gK), gS.reshape(-1)


def exact(case, seed):
    v = _inputs(case, seed)
    kind = case["kind"]
    if kind == "wells":
        return _exact_wells(case, v)
    x, y = case["x"], case["y"]
    wx, wy = case.get("wrapX", False), case.get("wrapY", False)
    if kind in ("agents", "coupled") or case.get("op") == "forces":
        n = case["agents"]
        p, rad = _dev(v["pos"]).view(-1, 2), _dev(v["rad"])
        where = (_ones(n, x), _ones(n, y), _ones(n, 0))
        reach = case.get("radius", 1.0)
        if kind == "call":
            return _pair_forces(p, rad, *where, wx, wy, reach, SPRING)[0].reshape(-1)
        if kind == "agents":
            # The trajectory has no such value: which of two nearly coincident
            # agents goes where, and on which side of a wrapped edge one ends,
            # is decided by rounding and grows over the ticks.
            return None
        vel = torch.zeros_like(p)
        f, src = _dev(v["field"]).view(x, y), _dev(v["src"]).view(x, y)
        step = _AdiStep(x, y, v["rate"], False, False)
        for _ in range(case["ticks"]):
            dv, cell = _pair_forces(p, rad, *where, wx, wy, reach, SPRING)
            p, vel = _move(p, vel, dv, where[0], where[1], wx, wy, FRICTION)
            count = torch.bincount(cell, minlength=x * y).view(x, y)
            f = f + ((step(f) - f) - v["decay"] * f + src - UPTAKE * count * f)
        return f.reshape(-1), (None, None)
    if kind == "adjoint":
        return _adjoint(case, v)
    f = _dev(v["field"]).view(x, y)
    if kind == "call":
        none = (None,) * 4
        if case["op"] == "diffuse":
            out = _explicit_tick(f, v["rate"], 0.0, wx, wy, none, None) - f
        elif case["op"] == "diffuse_var":
            rx, ry = _dev(v["rx"]).view(x, y), _dev(v["ry"]).view(x, y)
            px, mx = _diffs(f, 0, wx, None, None)
            py, my = _diffs(f, 1, wy, None, None)
            out = px * rx + mx * torch.roll(rx, 1, 0) + py * ry + my * torch.roll(ry, 1, 1)
        elif case["op"] == "advect":
            out = _explicit_tick(f, 0.0, 0.0, wx, wy, none, None, v["vx"], v["vy"]) - f
        else:
            out = _AdiStep(x, y, v["rate"], wx, wy)(f) - f
        return out.reshape(-1)
    if kind == "pdegrid":
        step = _AdiStep(x, y, v["rate"], wx, wy, v["ghost"]) if case["implicit"] else None
        g = _edges(v["ghost"], x, y)
        src = torch.zeros(x * y, dtype=torch.float64, device="cuda")
        src[torch.as_tensor(v["cells"], device="cuda").long()] = _dev(v["values"])
        src = src.view(x, y)
        for _ in range(case["ticks"]):
            if step is None:
                f = _explicit_tick(f, v["rate"], v["decay"], wx, wy, g, src)
            else:
                f = f + ((step(f) - f) + src - v["decay"] * f)
        return f.reshape(-1), torch.zeros_like(f).reshape(-1), None
    src = None if v.get("src") is None else _dev(v["src"]).view(x, y)
    if kind == "adi":
        step = _AdiStep(x, y, v["rate"], wx, wy, v["ghost"])
        for _ in range(case["ticks"]):
            d = (step(f) - f) - v["decay"] * f
            f = f + (d if src is None else d + src)
        return f.reshape(-1)
    if "cells" in v:
        src = torch.zeros(x * y, dtype=torch.float64, device="cuda")
        src[torch.as_tensor(v["cells"], device="cuda").long()] = _dev(v["values"])
        src = src.view(x, y)
    g = _edges(v["ghost"], x, y)
    for _ in range(case["ticks"]):
        f = _explicit_tick(f, v["rate"], v["decay"], wx, wy, g, src, v["vx"], v["vy"])
    return f.reshape(-1)


def _exact_wells(case, v):
    fields = []
    for w, f in zip(v["wells"], v["fields"]):
        s = w["xDim"]
        f = _dev(f).view(s, s)
        step = _AdiStep(s, s, w["diffRate"], False, False) if w["kind"] == "adi" else None
        for _ in range(case["ticks"]):
            if step is None:
                f = _explicit_tick(f, w["diffRate"], w["decay"], False, False, (None,) * 4, None)
            else:
                f = f + ((step(f) - f) - w["decay"] * f)
        fields.append(f.reshape(-1))
    return fields, (None, None)
