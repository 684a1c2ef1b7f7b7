"""The calls this library's users wait for, as measurable cases.

A case is one pass through the public entry points: the initial fields go in
from pinned host memory, the solver steps, and the fields (or the gradients,
or the output arrays) come back, as the benchmark's end-to-end leg does it.
Meshes, orders, step sizes and boundary kinds are those of the repository's
configurations, benchmark legs and tests; the fields are seeded pulses and
plane waves of the widths used there.

`kind` of a case:
  uniform  one order on every element (periodic, walled, outflow or inflow
           square), one or many instances, FP64, FP64_STRICT or FP32
  mixed    a periodic mesh whose orders differ after p-adaptation (mortars
           on most faces)
  hp       a walled mesh after p-adaptation and element splitting (2:1 faces)
  solve    the adaptive configuration as it is configured: steps to an end
           time, the error estimated and the adaptation decided every 20
           steps (at its threshold nothing refines)
  adapt    mesh load, steps, an adaptation that splits elements and raises
           orders, steps on the new mesh
  adjoint  forward solve with receivers and its gradient
  output   output interpolation and analytic errors of a mesh's fields
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch
import torch.utils.checkpoint

import ndg_cuda_b200 as ndg
from ndg_cuda_b200 import meshgen, workloads

_PRECISION = {"fp64": ndg.FP64, "strict": ndg.FP64_STRICT, "fp32": ndg.FP32}
_BOUNDARY = {"wall": meshgen.WALL, "outflow": meshgen.OUTFLOW, "inflow": meshgen.INFLOW, "periodic": meshgen.WALL}
_RK_A, _RK_B, _RK_G = (0.0, -5.0 / 9.0, -153.0 / 128.0), (0.0, 1.0 / 3.0, 0.75), (1.0 / 3.0, 15.0 / 16.0, 8.0 / 15.0)
_CFL = 0.5


def listed():
    return [
        # A first or a coarse run: the small periodic configuration, 200
        # steps of launches on 256 elements.
        {"name": "small_16_n4", "kind": "uniform", "res": 16, "order": 4, "boundary": "periodic", "instances": 1, "precision": "fp64",
         "jitter": 0.0, "steps": 200, "tune": False},
        # The flagship configuration, with the autotuned tile as the
        # benchmark runs it.
        {"name": "plane_256_n8", "kind": "uniform", "res": 256, "order": 8, "boundary": "periodic", "instances": 1, "precision": "fp64",
         "jitter": 0.0, "steps": 200, "tune": True},
        # The same in the FP32 form.
        {"name": "plane_256_n8_fp32", "kind": "uniform", "res": 256, "order": 8, "boundary": "periodic", "instances": 1, "precision": "fp32",
         "jitter": 0.0, "steps": 200, "tune": True},
        # The highest order of the published order sweep, boundaries held to
        # the analytic wave, default tile.
        {"name": "inflow_64_n16", "kind": "uniform", "res": 64, "order": 16, "boundary": "inflow", "instances": 1, "precision": "fp64",
         "jitter": 0.0, "steps": 100, "tune": False},
        # An ordinary odd-sized distorted mesh of odd order, default tile.
        {"name": "walls_91_n5", "kind": "uniform", "res": 91, "order": 5, "boundary": "wall", "instances": 1, "precision": "fp64",
         "jitter": 0.1, "steps": 200, "tune": False},
        # Many sources on one mesh: the batched configuration, FP32 form.
        {"name": "batch_64x64_n6_fp32", "kind": "uniform", "res": 64, "order": 6, "boundary": "wall", "instances": 64, "precision": "fp32",
         "jitter": 0.0, "steps": 100, "tune": True},
        # Stepping on a p-adapted mesh, orders 4 to 10 scattered.
        {"name": "mixed_128", "kind": "mixed", "res": 128, "order": 4, "rounds": 3, "precision": "fp64", "steps": 100},
        # Stepping on an hp-adapted mesh with two split levels, FP32 form.
        {"name": "hp_128_fp32", "kind": "hp", "res": 128, "order": 4, "rounds": 2, "precision": "fp32", "steps": 100},
        # The adaptive configuration, estimates and decisions included.
        {"name": "solve_128", "kind": "solve", "res": 128, "order": 4, "interval": 20, "steps": 60, "precision": "fp64"},
        # A driver that loads a mesh, steps, adapts once and steps on.
        {"name": "adapt_64", "kind": "adapt", "res": 64, "order": 4, "rounds": 1, "steps": 40, "precision": "fp64"},
        # The adjoint configuration at a fifth of its steps.
        {"name": "adjoint_96_n7", "kind": "adjoint", "res": 96, "order": 7, "steps": 200, "interval": 50, "receivers": 16, "precision": "fp64"},
        # The output a run writes at an output time.
        {"name": "output_64_n8", "kind": "output", "res": 64, "order": 8, "points": 10, "jitter": 0.1},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# DOF-stages of the largest listed case (256 x 256 elements of order 8, 200 steps)
_MOST = 3 * 256 * 256 * 81 * 3 * 200


def draw(rng):
    kind = rng.choice(["uniform"] * 6 + ["mixed"] * 2 + ["hp", "solve", "adapt", "adjoint", "adjoint", "output"])
    if kind == "uniform":
        order, res = rng.randint(2, 16), _log(rng, 8, 256)
        res = min(res, int(math.sqrt(3.6e7 / (3 * (order + 1) ** 2))))
        most = max(1, min(64, int(2.0e7 / (3 * res * res * (order + 1) ** 2))))
        instances = rng.choice([1, 1, _log(rng, 1, most)])
        steps = _log(rng, 50, 400)
        steps = max(20, min(steps, int(0.8 * _MOST / (9 * instances * res * res * (order + 1) ** 2))))
        precision = rng.choice(["fp64"] * 6 + ["fp32"] * 5 + ["strict"])
        if precision == "fp32" and order < 3:
            precision = "fp64"  # the scheme is unstable at N = 2 and CFL 0.5, which magnifies FP32 rounding
        steps = min(steps, 60) if order < 3 else steps
        return {"kind": kind, "res": res, "order": order, "boundary": rng.choice(["periodic", "wall", "outflow", "inflow"]),
                "instances": instances, "precision": precision, "jitter": rng.choice([0.0, 0.1]), "steps": steps,
                "tune": precision != "strict" and rng.random() < 0.4}
    if kind == "mixed":
        return {"kind": kind, "res": _log(rng, 12, 128), "order": rng.randint(3, 5), "rounds": rng.randint(1, 3),
                "precision": rng.choice(["fp64", "fp32"]), "steps": _log(rng, 20, 100)}
    if kind == "hp":
        return {"kind": kind, "res": _log(rng, 16, 128), "order": rng.randint(3, 5), "rounds": rng.randint(1, 2),
                "precision": rng.choice(["fp64", "fp32"]), "steps": _log(rng, 20, 100)}
    if kind == "solve":
        return {"kind": kind, "res": rng.randint(64, 160), "order": rng.randint(4, 8), "interval": rng.choice([10, 20, 50]),
                "steps": rng.randint(20, 100), "precision": rng.choice(["fp64", "fp32"])}
    if kind == "adapt":
        return {"kind": kind, "res": _log(rng, 16, 64), "order": rng.randint(3, 6), "rounds": 1, "steps": rng.randint(10, 60),
                "precision": rng.choice(["fp64", "fp32"])}
    if kind == "adjoint":
        return {"kind": kind, "res": _log(rng, 10, 96), "order": rng.randint(3, 9), "steps": _log(rng, 20, 120),
                "interval": rng.choice([0, 10, 25, 50]), "receivers": rng.randint(1, 24), "precision": rng.choice(["fp64", "fp32"])}
    return {"kind": kind, "res": _log(rng, 8, 64), "order": rng.randint(3, 10), "points": rng.randint(4, 12), "jitter": rng.choice([0.0, 0.1])}


# ---------------------------------------------------------------------------
# Inputs.


@functools.lru_cache(maxsize=24)
def _zone(res, boundary, jitter, seed):
    order = "hilbert" if not (res & (res - 1)) else "rowmajor"
    box = dict(x_min=0.0, x_max=1.0, y_min=0.0, y_max=1.0) if boundary == "inflow" else {}
    periodic = boundary == "periodic"
    return meshgen.uniform_zone(res, order=order, boundary=_BOUNDARY[boundary], x_periodic=periodic, y_periodic=periodic, jitter=jitter,
                                seed=seed, **box)


def _case_zone(case, seed):
    kind = case["kind"]
    if kind == "uniform":
        return _zone(case["res"], case["boundary"], case["jitter"], seed if case["jitter"] else 0)
    if kind == "mixed":
        return _zone(case["res"], "periodic", 0.1, seed)
    if kind == "output":
        return _zone(case["res"], "wall", case["jitter"], seed if case["jitter"] else 0)
    if kind == "adjoint":
        return _zone(case["res"], "wall", 0.0, 0)
    # hp, adapt: the refined region follows the element centres, so one mesh
    # for every seed; solve: the configuration's one jittered mesh
    return _zone(case["res"], "wall", 0.1, 7)


def _corners(zone):
    """(K, 4, 2) corner coordinates of the zone's quads."""
    conn = zone["sections"][0][4].reshape(-1, 4) - 1
    return np.stack([zone["x"][conn], zone["y"][conn]], axis=-1)


def _plane_wave(x, y, t):
    a = 0.707106781186548 * (x + 0.2) + 0.707106781186548 * (y + 0.2) - t
    return np.exp(-a * a / 0.120112240878645 ** 2)


def _node_positions(zone, orders):
    """x, y of every node, element after element, node i (N + 1) + j."""
    corners = _corners(zone)
    start = np.concatenate([[0], np.cumsum((orders + 1) ** 2)])
    X, Y = np.empty(start[-1]), np.empty(start[-1])
    for N in np.unique(orders):
        n = int(N) + 1
        x = np.polynomial.legendre.leggauss(n)[0]
        xi, eta = (v.ravel() for v in np.meshgrid(x, x, indexing="ij"))
        w = np.stack([(1 - xi) * (1 - eta), (1 + xi) * (1 - eta), (1 + xi) * (1 + eta), (1 - xi) * (1 + eta)]) / 4
        ids = np.flatnonzero(orders == N)
        at = start[ids][:, None] + np.arange(n * n)[None, :]
        X[at], Y[at] = corners[ids, :, 0] @ w, corners[ids, :, 1] @ w
    return X, Y


def _fields(case, seed, zone, orders):
    """p, u, v: per instance a travelling pulse and a standing one, seeded;
    the inflow square starts from the plane wave its boundary carries."""
    rng = np.random.default_rng(seed)
    X, Y = _node_positions(zone, orders)
    instances = case.get("instances", 1)
    lo, size = (0.0, 1.0) if case.get("boundary") == "inflow" else (-1.0, 2.0)
    out = np.empty((3, instances, X.size))
    for i in range(instances):
        (ax, ay), (bx, by) = lo + size * rng.uniform(0.1, 0.9, 2), lo + size * rng.uniform(0.1, 0.9, 2)
        sa, sb, th = size * rng.uniform(0.025, 0.05), size * rng.uniform(0.04, 0.08), rng.uniform(0.0, 2 * np.pi)
        if case["kind"] == "solve":
            # the configuration's width, off the walls: resolved, nothing refines
            ax, ay, bx, by, sa, sb = 0.5 * ax, 0.5 * ay, 0.5 * bx, 0.5 * by, 0.1, 0.1
        a = np.exp(-((X - ax) ** 2 + (Y - ay) ** 2) / (2 * sa * sa))
        b = 0.5 * np.exp(-((X - bx) ** 2 + (Y - by) ** 2) / (2 * sb * sb))
        out[0, i], out[1, i], out[2, i] = a + b, np.cos(th) * a, np.sin(th) * a
        if case.get("boundary") == "inflow":
            w = _plane_wave(X, Y, 0.0)
            out[0, i] = w + 0.1 * out[0, i]
            out[1, i], out[2, i] = 0.707106781186548 * w + 0.1 * out[1, i], 0.707106781186548 * w + 0.1 * out[2, i]
    return out


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=torch.cuda.is_available())
    t.numpy()[...] = a
    return t


def _p_flags(case, seed, K):
    """Elements whose order rises by 2, per round: each element's number of
    rises binomial (0.4 a round), scattered by the seed."""
    share = _rise_shares(case)
    counts = np.floor(np.cumsum(share) * K + 0.5).astype(int)
    rises = np.searchsorted(counts, np.arange(K), side="right")
    rises = np.random.default_rng(seed + 1).permutation(np.minimum(rises, case["rounds"]))
    return [rises > r for r in range(case["rounds"])]


def _rise_shares(case):
    share = [1.0]
    for _ in range(case["rounds"]):
        share = [0.6 * a + 0.4 * b for a, b in zip(share + [0.0], [0.0] + share)]
    return share


def _hp_flags(corners, r):
    """A ring around the centre, narrower every round r: refine flags and
    decay rates (its crest splits, its flanks gain order)."""
    c = corners.mean(axis=1)
    d = np.abs(np.hypot(c[:, 0] - 0.1, c[:, 1] + 0.05) - 0.45)
    return (d < 0.2 / (r + 1)).astype(np.int32), np.where(d < 0.05 / (r + 1), 0.5, 2.0)


def _adjoint_inputs(case, seed, zone, dt):
    """Initial pressure, wave speed, receivers and recorded traces."""
    rng = np.random.default_rng(seed + 3)
    orders = np.full(case["res"] ** 2, case["order"])
    X, Y = _node_positions(zone, orders)
    th = rng.uniform(0, 2 * np.pi)
    p0 = np.exp(-((X - 0.45 * np.cos(th)) ** 2 + (Y - 0.45 * np.sin(th)) ** 2) / (2 * 0.1 ** 2))
    R = case["receivers"]
    ang = 2 * np.pi * (np.arange(R) + 0.5) / R + 0.01 * th
    xy = 0.7 * np.stack([np.cos(ang), np.sin(ang)], axis=1)
    t = dt * np.arange(case["steps"] + 1)[:, None] / (dt * case["steps"])
    targets = rng.uniform(0.1, 0.4, R) * np.exp(-((t - rng.uniform(0.2, 0.8, R)) / 0.2) ** 2)
    return p0, xy, targets


def _dt(corners, N, c=None):
    """CFL step: the least corner distance of each element, over N^2 c."""
    p = [corners[:, k] for k in range(4)]
    d = np.min([np.linalg.norm(p[a] - p[b], axis=1) for a in range(4) for b in range(a)], axis=0)
    return float(np.min(_CFL * d / (np.asarray(N, float) ** 2 * (1.0 if c is None else c))))


def prepare(case, seed):
    kind = case["kind"]
    zone = _case_zone(case, seed)
    K = case["res"] ** 2
    s = {"case": case}
    if kind == "adapt":
        # the run itself loads the mesh, as a driver does
        s["zone"] = ndg.Zone.from_dict(zone)
        s["in"] = [f.copy() for f in _fields(case, seed, zone, np.full(K, case["order"]))[:, 0]]
        s["flags"] = _hp_flags(_corners(zone), 0)
        return s
    if kind == "adjoint":
        c = workloads.speed_field(zone, seed=seed)
        dt = _dt(_corners(zone), case["order"], c)
        p0, xy, targets = _adjoint_inputs(case, seed, zone, dt)
        mesh = ndg.Mesh2D_t(zone, case["order"])
        s.update(mesh=mesh, adj=ndg.Adjoint2D_t(mesh, xy, speed=c, precision=_PRECISION[case["precision"]]), p0=p0, dt=dt, targets=targets)
        return s
    if kind == "output":
        mesh = ndg.Mesh2D_t(zone, case["order"], n_interpolation_points=case["points"])
        f = _fields(case, seed, zone, np.full(K, case["order"]))
        for i, name in enumerate(("p", "u", "v")):
            mesh.set_field(name, f[i])
        mesh.synchronize()
        s.update(mesh=mesh, time=0.1 + 0.01 * (seed % 10))
        return s
    if kind == "uniform":
        mesh = ndg.Mesh2D_t(zone, case["order"], n_instances=case["instances"], precision=_PRECISION[case["precision"]])
    elif kind == "solve":
        mesh = ndg.Mesh2D_t(zone, case["order"], maximum_N=12, max_split_level=2, adaptivity_interval=case["interval"], tolerance_min=1e-3,
                            tolerance_max=1e-14, cfl=_CFL, precision=_PRECISION[case["precision"]])
        s["solver"] = ndg.Solver2D_t(_CFL, [(case["steps"] - 0.5) * _dt(_corners(zone), case["order"])])
    else:
        mesh = ndg.Mesh2D_t(zone, case["order"], maximum_N=case["order"] + 2 * case["rounds"], max_split_level=2 if kind == "hp" else 0,
                            precision=_PRECISION[case["precision"]])
        if kind == "mixed":
            for flags in _p_flags(case, seed, K):
                mesh.adapt(flags.astype(np.int32), np.full(K, 2.0))
        else:
            for r in range(case["rounds"]):
                nodes = mesh.elements()["nodes"][:4 * mesh.n_elements_].reshape(-1, 4)
                mesh.adapt(*_hp_flags(mesh.nodes()[nodes], r))
    if kind == "hp":
        # fields at the adapted mesh's nodes: the refined topology's own corners
        nodes = mesh.elements()["nodes"][:4 * mesh.n_elements_].reshape(-1, 4)
        xy = mesh.nodes()
        refined = {"x": xy[:, 0], "y": xy[:, 1], "sections": [("Elements", 0, 1, len(nodes), nodes.ravel() + 1)]}
        f = _fields(case, seed, refined, mesh.elements()["N"][:mesh.n_elements_])
    else:
        f = _fields(case, seed, zone, _orders(case, seed))
    if case.get("tune"):
        for i, name in enumerate(("p", "u", "v")):
            mesh.set_field(name, f[i])
        mesh.autotune()
    s["mesh"] = mesh
    s["in"] = [_pinned(f[i]) for i in range(3)]
    s["out"] = [_pinned(np.zeros_like(f[i])) for i in range(3)]
    return s


def _orders(case, seed):
    """The element orders of a uniform or mixed case, from its inputs."""
    orders = np.full(case["res"] ** 2, case["order"])
    if case["kind"] == "mixed":
        for flags in _p_flags(case, seed, orders.size):
            orders = orders + 2 * flags
    return orders


# ---------------------------------------------------------------------------
# One pass.


def _ok(status):
    if status != 0:
        raise ndg.NdgError(status, ndg.lib().ndg_last_error().decode())


def run(state):
    case = state["case"]
    if case["kind"] == "adapt":
        mesh = ndg.Mesh2D_t(state["zone"], case["order"], maximum_N=12, max_split_level=2, cfl=_CFL, precision=_PRECISION[case["precision"]])
        for i, name in enumerate(("p", "u", "v")):
            mesh.set_field(name, state["in"][i])
        time = ndg.Solver2D_t.run(mesh, case["steps"] // 2)
        mesh.adapt(*state["flags"])
        ndg.Solver2D_t.run(mesh, case["steps"] - case["steps"] // 2, time)
        out = {"N": mesh.elements()["N"]}
        for name in ("p", "u", "v"):
            out[name] = mesh.get_field(name)
        mesh.close()
        return out
    if case["kind"] == "adjoint":
        adj = state["adj"]
        J, samples = adj.forward(state["p0"], state["dt"], case["steps"], targets=state["targets"], checkpoint_interval=case["interval"])
        return {"J": J, "samples": samples, **adj.backward()}
    mesh = state["mesh"]
    if case["kind"] == "output":
        return mesh.get_solution(state["time"], complete=True)
    L = ndg.lib()
    for i in range(3):
        _ok(L.ndg_set_field(mesh.handle, -1, i, state["in"][i].data_ptr()))
    if case["kind"] == "solve":
        state["solver"].solve(mesh)
        if mesh.field_size != state["out"][0].numel():
            raise RuntimeError("the mesh refined: the outputs no longer fit")
    else:
        ndg.Solver2D_t.run(mesh, case["steps"])
    for i in range(3):
        _ok(L.ndg_get_field(mesh.handle, -1, i, state["out"][i].data_ptr()))
    return {"p": state["out"][0], "u": state["out"][1], "v": state["out"][2]}


# ---------------------------------------------------------------------------
# What a pass cannot do without.


def _nodes_of(case):
    """Nodes of a case's mesh (its expectation where the seed decides)."""
    K = case["res"] ** 2
    if case["kind"] == "mixed":
        return K * sum(w * (case["order"] + 2 * i + 1) ** 2 for i, w in enumerate(_rise_shares(case)))
    return K * (case["order"] + 1) ** 2


def work(case):
    """Stepping: q and k read and written once per RK3 stage in FP64 (the
    first stage reads no k: 88 B per degree of freedom and step), and per
    node, field and direction one row of the (N + 1)^2 contraction, the
    flux line and the lift (2 (N + 1) + 7 operations), the RK update 4."""
    n = case["order"] + 1
    nodes = _nodes_of(case)
    if case["kind"] == "output":
        P2, K = case["points"] ** 2, case["res"] ** 2
        return {"bytes": 8.0 * (3 * nodes + 8 * K * P2), "flops": float(6 * K * 2 * (case["points"] * n * n + P2 * n))}
    dof = 3.0 * nodes * case.get("instances", 1)
    per_stage = 2 * (2 * n + 7) + 4
    steps = case["steps"]
    if case["kind"] == "adjoint":
        # forward, recomputation of all but the last interval (keeping its
        # stage inputs), adjoint stages at 40 B
        kept = 1.0 if case["interval"] == 0 else min(1.0, case["interval"] / steps)
        return {"bytes": dof * steps * (88.0 + (1 - kept) * 88.0 + 24.0 + 120.0), "flops": dof * 3 * steps * per_stage * (3.0 - kept)}
    return {"bytes": dof * 88.0 * steps + 48.0 * nodes * case.get("instances", 1), "flops": dof * 3 * steps * per_stage}


def tolerance(case):
    kind, precision = case["kind"], case.get("precision", "fp64")
    if precision == "strict" and case.get("boundary") != "inflow":
        return "exact"
    # measured against exact(): FP64 up to 3.5e-14 (order 16), FP32 up to 1.1e-6
    return {"rel": 4e-6} if precision == "fp32" else {"rel": 2e-13}


# ---------------------------------------------------------------------------
# The results in 64 bits with plain torch: the conforming spectral-element
# operator on a square of quads, element orders free.


class _Exact:
    def __init__(self, zone, orders, boundary):
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=self.dev)  # noqa: E731
        conn = zone["sections"][0][4].reshape(-1, 4) - 1
        K = len(conn)
        cr = _corners(zone)
        nb, nbs = np.zeros((K, 4), np.int64), np.zeros((K, 4), np.int64)
        ghost = np.zeros((K, 4), bool)
        sides = {}
        for s in range(4):
            for e, (a, b) in enumerate(zip(conn[:, s].tolist(), conn[:, (s + 1) % 4].tolist())):
                sides.setdefault((min(a, b), max(a, b)), []).append((e, s))
        bars = {}
        for sec in zone["sections"][1:]:
            for i, (a, b) in enumerate((sec[4].reshape(-1, 2) - 1).tolist()):
                bars[sec[2] + i] = sides[(min(a, b), max(a, b))][0]
        for pair in sides.values():
            if len(pair) == 2:
                (e, s), (g, h) = pair
                nb[e, s], nbs[e, s], nb[g, h], nbs[g, h] = g, h, e, s
            else:
                ghost[pair[0]] = True
        for _, points, donors in zone["conns"]:
            for a, b in zip(points.tolist(), donors.tolist()):
                (e, s), (g, h) = bars[a], bars[b]
                nb[e, s], nbs[e, s], ghost[e, s] = g, h, False
        edge = np.roll(cr, -1, axis=1) - cr
        length = np.linalg.norm(edge, axis=2)
        self.boundary, self.K = boundary, K
        self.orders = [int(N) for N in np.unique(orders)]
        start = np.concatenate([[0], np.cumsum((orders + 1) ** 2)])
        local = np.zeros(K, np.int64)
        self.g = {}
        for N in self.orders:
            ids = np.flatnonzero(orders == N)
            local[ids] = np.arange(ids.size)
        for N in self.orders:
            n = N + 1
            ids = np.flatnonzero(orders == N)
            x, w = np.polynomial.legendre.leggauss(n)
            diff = x[:, None] - x[None, :]
            np.fill_diagonal(diff, 1.0)
            wb = 1.0 / diff.prod(axis=1)
            D = (wb[None, :] / wb[:, None]) / diff
            np.fill_diagonal(D, 0.0)
            np.fill_diagonal(D, -D.sum(axis=1))
            p = cr[ids]
            lin = lambda a, b: ((1 - x) * a[:, None] + (1 + x) * b[:, None]) / 4  # noqa: E731
            x_xi, y_xi = (lin(p[:, 1, d] - p[:, 0, d], p[:, 2, d] - p[:, 3, d]) for d in range(2))   # functions of eta
            x_eta, y_eta = (lin(p[:, 3, d] - p[:, 0, d], p[:, 2, d] - p[:, 1, d]) for d in range(2))  # functions of xi
            J = x_xi[:, None, :] * y_eta[:, :, None] - x_eta[:, :, None] * y_xi[:, None, :]
            end = lambda at: _lagrange(x, np.array([at]))[0]  # noqa: E731
            lm, lp = end(-1.0), end(1.0)
            pairs = []
            for M in self.orders:
                at = np.argwhere((orders[nb[ids]] == M) & ~ghost[ids])
                if len(at):
                    xf = x if N >= M else np.polynomial.legendre.leggauss(M + 1)[0]
                    xm = np.polynomial.legendre.leggauss(M + 1)[0]
                    wf = w if N >= M else np.polynomial.legendre.leggauss(M + 1)[1]
                    e_, s_ = at[:, 0], at[:, 1]
                    to_own = None if N >= M else t((_lagrange(x, xf) * wf[:, None] / w[None, :]))
                    pairs.append((M, t(e_), t(s_), t(local[nb[ids][e_, s_]]), t(nbs[ids][e_, s_]),
                                  None if N >= M else t(_lagrange(x, xf).T), None if M >= N else t(_lagrange(xm, xf).T), to_own))
            bnd = np.argwhere(ghost[ids])
            normal = np.stack([edge[ids][..., 1], -edge[ids][..., 0]], -1) / length[ids][..., None]
            mid = cr[ids][:, :, None, :] * ((1 - x) / 2)[None, None, :, None] + np.roll(cr[ids], -1, axis=1)[:, :, None, :] * ((1 + x) / 2)[None, None, :, None]
            self.g[N] = dict(at=t(start[ids][:, None] + np.arange(n * n)[None, :]), n=n, Dt=t((-(D.T * w[None, :]) / w[:, None]).T),
                             lm=t(lm), lp=t(lp), lmw=t(lm / w), lpw=t(lp / w), x_xi=t(x_xi)[:, None, :], y_xi=t(y_xi)[:, None, :],
                             x_eta=t(x_eta)[:, :, None], y_eta=t(y_eta)[:, :, None], iJ=t(1.0 / J), pairs=pairs, be=t(bnd[:, 0]), bs=t(bnd[:, 1]),
                             normal=t(normal), scale=t(length[ids] / 2), sidexy=t(mid))
        self.nb, self.ghost = t(nb), t(ghost)

    def traces(self, N, Q):
        g = self.g[N]
        return torch.stack([Q @ g["lm"], torch.einsum("bfkij,i->bfkj", Q, g["lp"]), (Q @ g["lp"]).flip(-1),
                            torch.einsum("bfkij,i->bfkj", Q, g["lm"]).flip(-1)], dim=3)

    @staticmethod
    def upwind(own, far, nx, ny):
        wl = own[:, 0] + own[:, 1] * nx + own[:, 2] * ny
        wr = far[:, 0] - far[:, 1] * nx - far[:, 2] * ny
        return torch.stack([(wl - wr) / 2, nx * (wl + wr) / 2, ny * (wl + wr) / 2], dim=1)

    def rate(self, q, time, c=None):
        """dq/dt of q, shape (instances, 3, nodes)."""
        Q = {N: q[:, :, g["at"]].unflatten(-1, (g["n"], g["n"])) for N, g in self.g.items()}
        T = {N: self.traces(N, Q[N]) for N in self.orders}
        out = torch.empty_like(q) if len(self.orders) > 1 else None
        for N, g in self.g.items():
            F = torch.zeros_like(T[N])
            for M, e, s, fe, fs, up_own, up_far, to_own in g["pairs"]:
                own, far = T[N][:, :, e, s], T[M][:, :, fe, fs].flip(-1)
                own = own if up_own is None else own @ up_own
                far = far if up_far is None else far @ up_far
                f = self.upwind(own, far, g["normal"][e, s, 0, None], g["normal"][e, s, 1, None])
                F = F.index_put((_all(F, 0), _all(F, 1), e[None, None, :], s[None, None, :]), f if to_own is None else f @ to_own)
            e, s = g["be"], g["bs"]
            if e.numel():
                own = T[N][:, :, e, s]
                nx, ny, sc = g["normal"][e, s, 0, None], g["normal"][e, s, 1, None], g["scale"][e, s, None]
                if self.boundary == "inflow":
                    xy = g["sidexy"][e, s]
                    a = 0.707106781186548 * (xy[..., 0] + 0.2) + 0.707106781186548 * (xy[..., 1] + 0.2) - time
                    p = torch.exp(-a * a / 0.120112240878645 ** 2)
                    far = torch.stack([p, 0.707106781186548 * p, 0.707106781186548 * p])[None].expand_as(own)
                else:
                    far = own * sc  # the ghost's trace carries its edge metric
                    if self.boundary == "wall":
                        l0, l1 = -(far[:, 1] * nx + far[:, 2] * ny), -far[:, 1] * ny + far[:, 2] * nx
                        far = torch.stack([far[:, 0], nx * l0 - ny * l1, ny * l0 + nx * l1], dim=1)
                F = F.index_put((_all(F, 0), _all(F, 1), e[None, None, :], s[None, None, :]), self.upwind(own, far, nx, ny))
            F = F * g["scale"][None, None, :, :, None]
            if c is not None:
                F = F * torch.where(self.ghost, c[:, None], 0.5 * (c[:, None] + c[self.nb]))[None, None, :, :, None]
            P, U, V = Q[N][:, 0], Q[N][:, 1], Q[N][:, 2]
            ce = 1.0 if c is None else c[None, None, :, None, None]
            line = torch.stack([g["y_eta"] * U - g["x_eta"] * V, g["y_eta"] * P, -g["x_eta"] * P], dim=1) * ce
            G = torch.matmul(line.transpose(-1, -2), g["Dt"]).transpose(-1, -2)
            G = G + g["lpw"][:, None] * F[:, :, :, 1, None, :] + g["lmw"][:, None] * F[:, :, :, 3, None, :].flip(-1)
            line = torch.stack([g["x_xi"] * V - g["y_xi"] * U, -g["y_xi"] * P, g["x_xi"] * P], dim=1) * ce
            G = G + torch.matmul(line, g["Dt"])
            G = G + F[:, :, :, 2, :, None].flip(-2) * g["lpw"] + F[:, :, :, 0, :, None] * g["lmw"]
            G = -G * g["iJ"]
            if out is None:
                return G.flatten(-3)
            out[:, :, g["at"].flatten()] = G.flatten(-3)
        return out

    def step(self, q, time, dt, c=None):
        k = None
        for m in range(3):
            G = self.rate(q, time + _RK_B[m] * dt, c)
            k = G if m == 0 else _RK_A[m] * k + G
            q = q + _RK_G[m] * dt * k
        return q


def _all(F, d):
    return torch.arange(F.shape[d], device=F.device).reshape([-1 if i == d else 1 for i in range(3)])


def _lagrange(x, at):
    """Lagrange basis over nodes x at the points `at`: (len(at), len(x))."""
    n = len(x)
    out = np.ones((len(at), n))
    for j in range(n):
        for m in range(n):
            if m != j:
                out[:, j] *= (at - x[m]) / (x[j] - x[m])
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("hp", "adapt"):
        return None  # split meshes: no short plain form
    zone = _case_zone(case, seed)
    if kind == "output":
        return _exact_output(case, seed, zone)
    if kind == "adjoint":
        return _exact_adjoint(case, seed, zone)
    orders = _orders(case, seed)
    E = _Exact(zone, orders, case.get("boundary", "wall" if kind == "solve" else "periodic"))
    q = torch.as_tensor(_fields(case, seed, zone, orders).transpose(1, 0, 2).copy(), device=E.dev)
    dt, time = _dt(_corners(zone), orders), 0.0
    with torch.no_grad():
        for i in range(case["steps"]):
            # an end time half a step short of the last full step's
            last = case["kind"] == "solve" and i == case["steps"] - 1
            q = E.step(q, time, 0.5 * dt if last else dt)
            time += dt
    return {"p": q[:, 0].contiguous().cpu(), "u": q[:, 1].contiguous().cpu(), "v": q[:, 2].contiguous().cpu()}


def _exact_output(case, seed, zone):
    n, P, time = case["order"] + 1, case["points"], 0.1 + 0.01 * (seed % 10)
    f = _fields(case, seed, zone, np.full(case["res"] ** 2, case["order"]))[:, 0].reshape(3, -1, n, n)
    x = np.polynomial.legendre.leggauss(n)[0]
    xi = np.arange(P) / (P - 1) * 2 - 1
    I = _lagrange(x, xi)
    up = lambda a: np.einsum("pi,kij,qj->kpq", I, a, I, optimize=True).ravel()  # noqa: E731
    a, b = (v.ravel() for v in np.meshgrid(xi, xi, indexing="ij"))
    w = np.stack([(1 - a) * (1 - b), (1 + a) * (1 - b), (1 + a) * (1 + b), (1 - a) * (1 + b)]) / 4
    cr = _corners(zone)
    out = {"x": (cr[..., 0] @ w).ravel(), "y": (cr[..., 1] @ w).ravel(), "p": up(f[0]), "u": up(f[1]), "v": up(f[2])}
    X, Y = _node_positions(zone, np.full(case["res"] ** 2, case["order"]))
    wave = _plane_wave(X, Y, time).reshape(-1, n, n)
    for i, name in enumerate(("p", "u", "v")):
        out[name + "_analytical_error"] = up(np.abs((1.0 if i == 0 else 0.707106781186548) * wave - f[i]))
    return out


def _exact_adjoint(case, seed, zone):
    N, steps = case["order"], case["steps"]
    n, K = N + 1, case["res"] ** 2
    cr = _corners(zone)
    c_np = workloads.speed_field(zone, seed=seed)
    dt = _dt(cr, N, c_np)
    p0, xy, targets = _adjoint_inputs(case, seed, zone, dt)
    E = _Exact(zone, np.full(K, N), "wall")
    t = lambda a: torch.as_tensor(a, device=E.dev)  # noqa: E731
    lo, hi = cr.min(axis=1), cr.max(axis=1)  # undistorted squares
    x = np.polynomial.legendre.leggauss(n)[0]
    el, wr = [], []
    for r in xy:
        e = int(np.flatnonzero(np.all((lo <= r) & (r < hi), axis=1))[0])
        p = cr[e]
        A = np.stack([p[1] - p[0], p[3] - p[0]], axis=1)
        xi, eta = 2 * np.linalg.solve(A, r - p[0]) - 1
        el.append(e)
        wr.append(np.outer(_lagrange(x, np.array([xi]))[0], _lagrange(x, np.array([eta]))[0]).ravel())
    at = t(np.array(el)[:, None] * n * n + np.arange(n * n)[None, :])
    wr, d = t(np.array(wr)), t(targets)
    q0 = t(np.stack([p0, np.zeros_like(p0), np.zeros_like(p0)])[None]).requires_grad_(True)
    c = t(c_np).requires_grad_(True)

    def step(q, c):
        q = E.step(q, 0.0, dt, c)
        return q, (q[0, 0][at] * wr).sum(1)

    q, J, samples = q0, 0.0, [(q0[0, 0][at] * wr).sum(1)]
    for i in range(steps):
        q, s = torch.utils.checkpoint.checkpoint(step, q, c, use_reentrant=False)
        samples.append(s)
        J = J + dt / 2 * ((s - d[i + 1]) ** 2).sum()
    J.backward()
    gq = q0.grad[0].cpu()
    return {"J": float(J.detach()), "samples": torch.stack(samples).detach().cpu(), "p0": gq[0].contiguous(), "u0": gq[1].contiguous(),
            "v0": gq[2].contiguous(), "c": c.grad.cpu()}
