"""Performance cases: what users of the engine have it do, through its public
Python entry points (klampt_gb300.engine, klampt_gb300.autodiff).

A case is a dict of plain values; `prepare` makes its state (a world that a
program keeps, and the query batch made from the seed), `run` is one pass,
`work` the bytes and operations of a pass that cannot be done without, and
`exact` the result in 64-bit torch, without the engine, where that is quick.

Scenes are the ones of klampt_gb300.scenes: arms of 6 and 7 joints, a dual
arm and a 30-DOF humanoid among icospheres, boxes or a heightfield terrain.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from klampt_gb300 import scenes as sc
from klampt_gb300.autodiff import MinDistance, SelfMinDistance, SoftMinDistance
from klampt_gb300.engine import Geometry, World

DEVICE = "cuda"


def listed():
    return [
        # a lazy planner checks the unverified edges of its current path: the
        # smallest calls, where latency and launches count
        {"name": "path_edges", "kind": "edges", "spheres": 2000, "edges": 24, "max_steps": 400, "plan": False},
        # a roadmap's edges in bulk: the engine's headline batch, replayed as
        # an edge plan with the launch options its autotuner settles on
        {"name": "roadmap_edges", "kind": "edges", "spheres": 2000, "edges": 16384, "max_steps": 400, "plan": True},
        # a planner round's new milestones: joint limits, environment and
        # self collision in one verdict
        {"name": "milestones", "kind": "feasible", "robot": "arm7", "spheres": 2000, "boxes": 0, "configs": 500},
        # sampled configurations in bulk, environment and self verdicts apart
        {"name": "configs", "kind": "configs", "robot": "arm7", "spheres": 2000, "boxes": 0, "configs": 262144},
        # a mixed fleet (6/7/12/30 joints) in one call, 1.0 M triangles
        {"name": "fleet_configs", "kind": "multi", "spheres": 700, "boxes": 8700, "configs": 65536},
        # clearance and its gradient over a terrain with boxes, clamped
        {"name": "terrain_clearance", "kind": "clearance", "nx": 512, "ny": 1024, "boxes": 500, "configs": 32768,
         "cutoff": 0.2},
        # one trajectory of an optimiser: soft-min clearance, forward and backward
        {"name": "trajectory_softmin", "kind": "softmin", "spheres": 2000, "trajectories": 1, "waypoints": 32,
         "path": True},
        # a batch of trajectories optimised together
        {"name": "softmin_batch", "kind": "softmin", "spheres": 2000, "trajectories": 200, "waypoints": 32,
         "path": False},
        # a humanoid's distance to itself and its gradient (posture costs)
        {"name": "self_clearance", "kind": "self", "configs": 8192, "cutoff": 1.0},
        # distance of two free meshes over a batch of placements
        {"name": "mesh_distance", "kind": "geom", "op": "distance", "rings": 32, "subdiv": 2, "queries": 16384,
         "spread": 0.5},
        # a depth camera's frame
        {"name": "camera_rays", "kind": "rays", "spheres": 2000, "width": 640, "height": 480},
        # point and orientation targets of an arm, solved as a batch
        {"name": "ik_batch", "kind": "ik", "robot": "arm7", "problems": 65536, "rotation": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges."""
    kind = rng.choice(["edges", "edges", "feasible", "configs", "multi", "clearance", "softmin", "softmin", "self",
                       "geom", "rays", "ik"])
    if kind == "edges":
        return {"kind": kind, "spheres": _log(rng, 60, 2000), "edges": _log(rng, 8, 16384),
                "max_steps": _log(rng, 30, 400), "plan": rng.random() < 0.5}
    if kind in ("feasible", "configs"):
        boxes = rng.choice([0, 20])
        return {"kind": kind, "robot": rng.choice(["arm6", "arm7", "dual", "humanoid"]),
                "spheres": 0 if boxes else _log(rng, 60, 2000), "boxes": boxes, "configs": _log(rng, 64, 65536)}
    if kind == "multi":
        return {"kind": kind, "spheres": _log(rng, 20, 700), "boxes": _log(rng, 100, 8700),
                "configs": _log(rng, 512, 65536)}
    if kind == "clearance":
        return {"kind": kind, "nx": _log(rng, 64, 512), "ny": _log(rng, 64, 1024), "boxes": _log(rng, 20, 500),
                "configs": _log(rng, 64, 32768), "cutoff": round(rng.uniform(0.05, 1.0), 3)}
    if kind == "softmin":
        return {"kind": kind, "spheres": _log(rng, 100, 2000), "trajectories": _log(rng, 1, 100),
                "waypoints": rng.randint(8, 64), "path": rng.random() < 0.5}
    if kind == "self":
        return {"kind": kind, "configs": _log(rng, 32, 8192), "cutoff": round(rng.uniform(0.2, 2.0), 3)}
    if kind == "geom":
        return {"kind": kind, "op": rng.choice(["distance", "distance", "collide", "within"]),
                "rings": rng.randint(4, 40), "subdiv": rng.randint(1, 4), "queries": _log(rng, 32, 16384),
                "spread": round(rng.uniform(0.15, 0.8), 3)}
    if kind == "rays":
        return {"kind": kind, "spheres": _log(rng, 60, 2000), "width": rng.randint(40, 640),
                "height": rng.randint(30, 480)}
    return {"kind": kind, "robot": rng.choice(["arm6", "arm7", "dual"]), "problems": _log(rng, 16, 65536),
            "rotation": rng.random() < 0.7}


# ---- scenes ------------------------------------------------------------------

TAU = 0.01  # soft-min temperature (m)
IK_TOL = 1e-4
WITHIN = 0.05  # tolerance of the within-distance queries (m)
_WORLDS = {}  # a program keeps its worlds; states of one scene share one


def _robot(name):
    return {"arm6": lambda: sc.arm(6, rings=16), "arm7": lambda: sc.arm(7, rings=32), "dual": sc.dual_arm,
            "humanoid": sc.humanoid}[name]()


def _fleet():
    return [sc.arm(6, rings=16, segments=16), sc.arm(7, rings=32), sc.dual_arm(), sc.humanoid()]


def _scene(case):
    """(environment, robots) of a case."""
    kind = case["kind"]
    if kind in ("edges", "softmin", "rays"):
        return sc.sphere_field(np.random.default_rng(1001), n=case["spheres"]), [sc.arm(7, rings=32)]
    if kind in ("feasible", "configs"):
        rng = np.random.default_rng(1000)
        if case["boxes"]:
            env = sc.env_from_objects("boxes", sc.random_boxes(case["boxes"], rng))
        else:
            env = sc.sphere_field(np.random.default_rng(1001), n=case["spheres"])
        return env, [_robot(case["robot"])]
    if kind == "multi":
        rng = np.random.default_rng(1003)
        meshes = sc.random_icospheres(case["spheres"], rng, sc.SPHERE_FIELD_CENTER, 2.0, subdiv=3)
        meshes += sc.random_boxes(case["boxes"], rng, lo=-1.0, hi=1.0, half_lo=0.01, half_hi=0.04)
        return sc.env_from_objects("boxes_spheres", meshes), _fleet()
    if kind == "clearance":
        rng = np.random.default_rng(1004)
        nx, ny, spacing = case["nx"], case["ny"], 0.004 * 512 / case["nx"]
        heights = sc.terrain_heights(nx, ny, spacing, rng)
        terrain = sc.heightfield_mesh(nx, ny, spacing, heights,
                                      (-spacing * (nx - 1) / 2, -spacing * (ny - 1) / 2, -1.0))
        boxes = sc.random_boxes(case["boxes"], rng)
        return sc.env_from_objects("terrain_boxes", [terrain] + boxes, [1] + [0] * len(boxes),
                                   [0] + [1] * len(boxes)), [sc.arm(7, rings=32)]
    if kind == "self":
        return sc.env_from_objects("far", [sc.box_mesh((9, 9, 9), (0.1, 0.1, 0.1))]), [sc.humanoid()]
    return sc.env_from_objects("far", [sc.box_mesh((9, 9, 9), (0.1, 0.1, 0.1))]), [_robot(case["robot"])]  # ik


def _world(case):
    kind = case["kind"]
    keys = {"edges": ("spheres", "plan"), "softmin": ("spheres",), "rays": ("spheres",),
            "feasible": ("robot", "spheres", "boxes"), "configs": ("robot", "spheres", "boxes"),
            "multi": ("spheres", "boxes"), "clearance": ("nx", "ny", "boxes"), "self": (), "ik": ("robot",)}[kind]
    key = (kind,) + tuple(case[k] for k in keys)
    if key not in _WORLDS:
        env, robots = _scene(case)
        world = World(env, robots)
        if kind == "edges" and case["plan"]:
            for name, value in (("blocks_per_sm", 2), ("grab", 1), ("job_flush", 32), ("edge_chunk", 32)):
                world.set_option(name, value)
        _WORLDS[key] = (env, robots, world)
    return _WORLDS[key]


def _cuda(x):
    return torch.as_tensor(np.ascontiguousarray(x)).to(DEVICE)


def _placements(rng, n, spread):
    """Random rigid transforms [n, 12] (rotation row-major, translation)."""
    q = rng.normal(size=(n, 4))
    w, x, y, z = (q / np.linalg.norm(q, axis=1, keepdims=True)).T
    R = np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                  2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                  2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], 1)
    return np.concatenate([R, rng.uniform(-spread, spread, (n, 3))], 1)


def _fk64(robot, q):
    """World transforms (R [n, L, 3, 3], t [n, L, 3]) in 64 bits."""
    n, L = q.shape
    R = torch.zeros(n, L, 3, 3, dtype=torch.float64, device=q.device)
    t = torch.zeros(n, L, 3, dtype=torch.float64, device=q.device)
    for i in range(L):
        T0 = torch.as_tensor(robot.T0_parent[i], dtype=torch.float64, device=q.device)
        R0, t0 = T0[:9].reshape(3, 3), T0[9:]
        a = torch.as_tensor(np.asarray(robot.axes[i], np.float64), device=q.device)
        K = torch.zeros(3, 3, dtype=torch.float64, device=q.device)
        K[0, 1], K[0, 2], K[1, 0], K[1, 2], K[2, 0], K[2, 1] = -a[2], a[1], a[2], -a[0], -a[1], a[0]
        I = torch.eye(3, dtype=torch.float64, device=q.device)
        s, c = torch.sin(q[:, i])[:, None, None], torch.cos(q[:, i])[:, None, None]
        J = I + s * K + (1 - c) * (K @ K) if robot.joint_types[i] == 0 else I.expand(n, 3, 3)
        p = int(robot.parents[i])
        Rl, tl = R0 @ J, t0.expand(n, 3)
        R[:, i] = Rl if p < 0 else R[:, p] @ Rl
        t[:, i] = tl if p < 0 else t[:, p] + (R[:, p] @ tl[..., None])[..., 0]
    return R, t


def _host_inputs(case, seed):
    """The query batch of a case as host arrays, from the seed alone."""
    rng = np.random.default_rng([seed, 77])
    kind = case["kind"]
    if kind == "edges":
        qa, qb, n = sc.random_edges(sc.arm(7, rings=1), case["edges"], rng, max_steps=case["max_steps"])
        return {"qa": qa, "qb": qb, "n": n}
    if kind in ("feasible", "configs"):
        return {"q": sc.uniform_configs(_robot(case["robot"]), case["configs"], rng)}
    if kind == "multi":
        robots = _fleet()
        total = case["configs"]
        ids = rng.choice(4, size=total, p=(0.4, 0.3, 0.2, 0.1)).astype(np.int32)
        q = np.zeros((total, max(r.num_links for r in robots)), np.float32)
        for i, r in enumerate(robots):
            at = np.flatnonzero(ids == i)
            q[at, :r.num_links] = sc.uniform_configs(r, len(at), rng)
        return {"ids": ids, "q": q}
    if kind == "clearance":
        return {"q": sc.uniform_configs(sc.arm(7, rings=1), case["configs"], rng)}
    if kind == "softmin":
        robot = sc.arm(7, rings=1)
        T, W = case["trajectories"], case["waypoints"]
        if case["path"]:  # a straight path between two configurations, disturbed
            a, b = rng.uniform(robot.qmin, robot.qmax, (2, T, 1, 7))
            q = a + (b - a) * np.linspace(0, 1, W)[None, :, None] + rng.normal(0, 0.05, (T, W, 7))
            return {"q": np.clip(q, robot.qmin, robot.qmax).astype(np.float32)}
        return {"q": sc.noisy_trajectories(robot, T, W, rng)}
    if kind == "self":  # from folded to widely spread postures
        q = sc.uniform_configs(sc.humanoid(), case["configs"], rng)
        return {"q": (q * rng.uniform(0, 1, (case["configs"], 1))).astype(np.float32)}
    if kind == "geom":
        return {"Ta": _placements(rng, case["queries"], case["spread"]),
                "Tb": _placements(rng, case["queries"], case["spread"])}
    if kind == "rays":
        eye = np.asarray(sc.CAMERA_EYES[seed % 4]) + rng.uniform(-0.2, 0.2, 3)
        s, d = sc.camera_rays(eye, sc.SPHERE_FIELD_CENTER, case["width"], case["height"])
        return {"s": s, "d": d}
    robot = _robot(case["robot"])  # ik: reachable targets, starts near a solution
    link = min(robot.num_links, 7) - 1 if case["robot"] != "dual" else 5
    qt = rng.uniform(-2.5, 2.5, (case["problems"], robot.num_links)).astype(np.float32)
    R, t = _fk64(robot, torch.as_tensor(qt, dtype=torch.float64))
    tip = (R[:, link] @ torch.tensor([0.0, 0.0, 0.3], dtype=torch.float64) + t[:, link]).numpy()
    q0 = np.clip(qt + rng.normal(0, 0.3, qt.shape), -np.pi, np.pi)
    return {"q0": q0.astype(np.float32), "link": link, "tip": tip.astype(np.float32),
            "R": R[:, link].reshape(-1, 9).numpy().astype(np.float32)}


# ---- the state and one pass -----------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    x = _host_inputs(case, seed)
    state = {"case": case}
    state.update((k, _cuda(v) if isinstance(v, np.ndarray) else v) for k, v in x.items())
    if kind == "geom":
        key = ("geom", case["rings"], case["subdiv"])
        if key not in _WORLDS:
            _WORLDS[key] = (Geometry(*sc.cylinder_mesh(0.05, 0.3, 32, case["rings"])),
                            Geometry(*sc.icosphere_mesh((0, 0, 0), 0.1, case["subdiv"])))
        state["a"], state["b"] = _WORLDS[key]
        return state
    _, _, state["world"] = _world(case)
    if kind == "edges" and case["plan"]:
        state["out"] = torch.empty(case["edges"], dtype=torch.int32, device=DEVICE)
        state["edge_plan"] = state["world"].edge_plan(state["qa"], state["qb"], state["n"], state["out"])
    if kind in ("clearance", "softmin", "self"):
        state["q"].requires_grad_(True)
    if kind == "ik":
        state["plocal"] = torch.tensor([[0.0, 0.0, 0.3]], device=DEVICE)
    return state


def run(state):
    case, world = state["case"], state.get("world")
    kind = case["kind"]
    if kind == "edges":
        if case["plan"]:
            state["edge_plan"].launch()
            return state["out"]
        return world.check_edges(state["qa"], state["qb"], state["n"])
    if kind == "feasible":
        return world.is_feasible(state["q"])
    if kind == "configs":
        return world.check_configs(state["q"])
    if kind == "multi":
        return world.check_configs_multi(state["ids"], state["q"])
    if kind in ("clearance", "softmin", "self"):
        q = state["q"]
        q.grad = None
        if kind == "softmin":
            value = SoftMinDistance.apply(q, world, TAU)
        elif kind == "clearance":
            value = MinDistance.apply(q, world, case["cutoff"])
        else:
            value = SelfMinDistance.apply(q, world, case["cutoff"])
        value.sum().backward()
        return {"value": value.detach(), "grad": q.grad}
    if kind == "geom":
        if case["op"] == "distance":
            d, cp, elem, direction = state["a"].distance(state["b"], state["Ta"], state["Tb"])
            return {"d": d, "cp": cp, "elem": elem, "dir": direction}
        return state["a"].collide(state["b"], state["Ta"], state["Tb"], WITHIN if case["op"] == "within" else 0.0)
    if kind == "rays":
        obj, tri, t, point = world.raycast(state["s"], state["d"])
        return {"obj": obj, "tri": tri, "t": t, "point": point}
    q, ok, residual, iters = world.ik_solve(state["q0"], state["link"], state["plocal"], state["tip"],
                                            Rtarget=state["R"] if case["rotation"] else None, tol=IK_TOL)
    return {"q": q, "ok": ok, "residual": residual, "iters": iters}


def work(case):
    """Query inputs read once, results written once, and the operations of one
    forward kinematics per configuration (35 for the joint rotation, 63 per
    composition, per link) or one placement per query."""
    kind = case["kind"]
    links = {"arm6": 6, "arm7": 7, "dual": 12, "humanoid": 31}
    fk = 98
    if kind == "edges":  # at least the first configuration of every edge
        E = case["edges"]
        return {"bytes": E * (2 * 7 * 4 + 4 + 4), "flops": E * 7 * fk}
    if kind in ("feasible", "configs"):
        L, B = links[case["robot"]], case["configs"]
        return {"bytes": B * (4 * L + (1 if kind == "feasible" else 2)), "flops": B * L * fk}
    if kind == "multi":
        L, B = 0.4 * 6 + 0.3 * 7 + 0.2 * 12 + 0.1 * 31, case["configs"]
        return {"bytes": B * (4 * L + 4 + 2), "flops": B * L * fk}
    if kind in ("clearance", "self"):
        L, B = (7 if kind == "clearance" else 31), case["configs"]
        return {"bytes": B * (4 * L + 8 + 4 * L), "flops": 2 * B * L * fk}
    if kind == "softmin":
        B = case["trajectories"] * case["waypoints"]
        return {"bytes": B * (28 + 28) + 8 * case["trajectories"], "flops": 2 * B * 7 * fk}
    if kind == "geom":
        B = case["queries"]
        out = 8 + 48 + 8 + 24 if case["op"] == "distance" else 1
        return {"bytes": B * (2 * 96 + out), "flops": B * 63}
    if kind == "rays":
        R = case["width"] * case["height"]
        return {"bytes": R * (24 + 4 + 4 + 8 + 24), "flops": R * 50}
    L, B = links[case["robot"]], case["problems"]
    return {"bytes": B * (2 * 4 * L + 12 + (36 if case["rotation"] else 0) + 9), "flops": 2 * B * L * fk}


# ---- results in 64 bits ----------------------------------------------------------

def _cross(a, b):
    return torch.linalg.cross(a, b, dim=-1)


def _dot(a, b):
    return (a * b).sum(-1)


def _segments(p, d, q, e):
    """Closest points of segments p + s d and q + t e, s, t in [0, 1]."""
    r = p - q
    a, c, f, b = _dot(d, d), _dot(d, r), _dot(e, r), _dot(d, e)
    ee = _dot(e, e)
    den = a * ee - b * b
    s = torch.where(den > 0, ((b * f - c * ee) / torch.where(den > 0, den, torch.ones_like(den))).clamp(0, 1),
                    torch.zeros_like(den))
    t = (b * s + f) / ee
    s = torch.where(t < 0, (-c / a).clamp(0, 1), torch.where(t > 1, ((b - c) / a).clamp(0, 1), s))
    t = t.clamp(0, 1)
    return p + s[..., None] * d, q + t[..., None] * e


def _onto_triangle(p, T):
    """Projection of p onto the plane of triangle T, and whether it is inside."""
    n = _cross(T[:, 1] - T[:, 0], T[:, 2] - T[:, 0])
    foot = p - (_dot(p - T[:, 0], n) / _dot(n, n))[:, None] * n
    inside = torch.ones(len(p), dtype=torch.bool, device=p.device)
    for k in range(3):
        inside &= _dot(_cross(T[:, (k + 1) % 3] - T[:, k], foot - T[:, k]), n) >= 0
    return foot, inside


def _crosses(T, U):
    """Whether an edge of triangle T passes through triangle U."""
    n = _cross(U[:, 1] - U[:, 0], U[:, 2] - U[:, 0])
    hit = torch.zeros(len(T), dtype=torch.bool, device=T.device)
    for k in range(3):
        a, b = T[:, k], T[:, (k + 1) % 3]
        da, db = _dot(a - U[:, 0], n), _dot(b - U[:, 0], n)
        ok = da * db <= 0
        x = a + (da / torch.where(da == db, torch.ones_like(da), da - db))[:, None] * (b - a)
        for j in range(3):
            ok &= _dot(_cross(U[:, (j + 1) % 3] - U[:, j], x - U[:, j]), n) >= 0
        hit |= ok
    return hit


def _triangles(P, Q):
    """Distance and closest points of triangle pairs [n, 3, 3]; 0 where they meet."""
    best = torch.full((len(P),), math.inf, dtype=torch.float64, device=P.device)
    cp, cq = torch.zeros_like(P[:, 0]), torch.zeros_like(P[:, 0])

    def offer(x, y, allowed=None):
        nonlocal best, cp, cq
        d = _dot(x - y, x - y)
        take = d < best if allowed is None else (d < best) & allowed
        best = torch.where(take, d, best)
        cp = torch.where(take[:, None], x, cp)
        cq = torch.where(take[:, None], y, cq)

    for i in range(3):
        for j in range(3):
            offer(*_segments(P[:, i], P[:, (i + 1) % 3] - P[:, i], Q[:, j], Q[:, (j + 1) % 3] - Q[:, j]))
    for k in range(3):
        foot, inside = _onto_triangle(P[:, k], Q)
        offer(P[:, k], foot, inside)
        foot, inside = _onto_triangle(Q[:, k], P)
        offer(foot, Q[:, k], inside)
    meet = _crosses(P, Q) | _crosses(Q, P)
    return torch.where(meet, torch.zeros_like(best), best).sqrt(), cp, cq


def _mesh_distance(A, B):
    """Distance and closest points of mesh pairs: A, B [k, a or b, 3, 3]
    world triangles.  Triangle pairs that cannot be the closest by their
    bounding spheres are left out."""
    ca, cb = A.mean(2), B.mean(2)
    ra = (A - ca[:, :, None]).norm(dim=-1).amax(-1)
    rb = (B - cb[:, :, None]).norm(dim=-1).amax(-1)
    near = torch.cdist(ca, cb)
    limit = near.flatten(1).amin(1)
    k, i, j = torch.nonzero(near - ra[:, :, None] - rb[:, None, :] <= limit[:, None, None] + 1e-9, as_tuple=True)
    d = torch.full((len(A),), math.inf, dtype=torch.float64, device=A.device)
    cp, cq = torch.zeros_like(A[:, 0, 0]), torch.zeros_like(A[:, 0, 0])
    parts = [_triangles(A[k[s:s + 4000000], i[s:s + 4000000]], B[k[s:s + 4000000], j[s:s + 4000000]])
             for s in range(0, len(k), 4000000)]
    if not parts:
        return d, cp, cq
    dd, p, q = (torch.cat(x) for x in zip(*parts))
    d = d.scatter_reduce(0, k, dd, "amin")
    first = torch.full((len(A),), len(k), dtype=torch.int64, device=A.device)
    at = torch.nonzero(dd == d[k])[:, 0]
    first = first.scatter_reduce(0, k[at], at, "amin")
    return d, p[first], q[first]


def _exact_geom(case, x, dev):
    A, B = sc.cylinder_mesh(0.05, 0.3, 32, case["rings"]), sc.icosphere_mesh((0, 0, 0), 0.1, case["subdiv"])
    tris = [torch.as_tensor(v[f], device=dev) for v, f in (A, B)]
    step = max(1, 40000000 // (len(tris[0]) * len(tris[1])))
    out = []
    for s in range(0, case["queries"], step):
        world = []
        for T, t in zip((x["Ta"], x["Tb"]), tris):
            T = torch.as_tensor(T[s:s + step], device=dev)
            world.append(torch.einsum("kij,avj->kavi", T[:, :9].reshape(-1, 3, 3), t) + T[:, None, None, 9:])
        out.append(_mesh_distance(*world))
    d, p, q = (torch.cat(v) for v in zip(*out))
    # touching surfaces and several pairs of equally near points have no
    # closest points of their own: the distance alone is compared
    return {"d": d, "cp": None, "elem": None, "dir": None}


def _exact_rays(case, x, dev):
    env = sc.sphere_field(np.random.default_rng(1001), n=case["spheres"])
    tri = torch.as_tensor(np.stack([v[f] for v, f in env.meshes]), device=dev)  # [objects, 320, 3, 3]
    centre = tri.mean((1, 2))
    radius = (tri - centre[:, None, None]).norm(dim=-1).amax((1, 2)) * (1 + 1e-9)
    S, D = (torch.as_tensor(x[k], dtype=torch.float64, device=dev) for k in ("s", "d"))
    t_best = torch.full((len(S),), math.inf, dtype=torch.float64, device=dev)
    for b in range(0, len(S), 16384):
        s, d = S[b:b + 16384], D[b:b + 16384]
        w = centre[None] - s[:, None]
        along = (w * d[:, None]).sum(-1) / _dot(d, d)[:, None]
        off = (w - along[..., None] * d[:, None]).norm(dim=-1)
        r, o = torch.nonzero(off <= radius[None], as_tuple=True)
        for c in range(0, len(r), 20000):
            rr, oo = r[c:c + 20000], o[c:c + 20000]
            T, ss, ddir = tri[oo], s[rr][:, None], d[rr][:, None]
            e1, e2 = T[:, :, 1] - T[:, :, 0], T[:, :, 2] - T[:, :, 0]
            p, ww = _cross(ddir.expand_as(e2), e2), ss - T[:, :, 0]
            det = _dot(e1, p)
            q = _cross(ww, e1)
            safe = torch.where(det == 0, torch.ones_like(det), det)
            u, v, t = _dot(ww, p) / safe, (q * ddir).sum(-1) / safe, _dot(e2, q) / safe
            hit = (det != 0) & (u >= 0) & (v >= 0) & (u + v <= 1) & (t >= 0)
            t = torch.where(hit, t, torch.full_like(t, math.inf)).amin(1)
            t_best[b:b + 16384] = t_best[b:b + 16384].scatter_reduce(0, rr, t, "amin")
    point = torch.where(torch.isfinite(t_best)[:, None], S + torch.nan_to_num(t_best, posinf=0.0)[:, None] * D,
                        torch.zeros_like(S))
    return {"obj": None, "tri": None, "t": t_best, "point": point}


def _exact_softmin(case, x, dev):
    """Signed link-sphere distances (minus the deepest link vertex's depth
    where the surfaces meet), the soft-min of those within 30 tau of the
    smallest, and its gradient by the joints' screw axes."""
    env = sc.sphere_field(np.random.default_rng(1001), n=case["spheres"])
    robot = sc.arm(7, rings=32)
    q = torch.as_tensor(x["q"], dtype=torch.float64, device=dev)[0]
    W, L = q.shape
    R, t = _fk64(robot, q)
    obj = torch.as_tensor(np.stack([v[f] for v, f in env.meshes]), device=dev)
    oc = obj.mean((1, 2))
    orad = (obj - oc[:, None, None]).norm(dim=-1).amax((1, 2))
    n = _cross(obj[:, :, 1] - obj[:, :, 0], obj[:, :, 2] - obj[:, :, 0])
    n = n / n.norm(dim=-1, keepdim=True)
    off = _dot(n, obj[:, :, 0])
    mesh_v = [torch.as_tensor(v, device=dev) for v, _ in robot.meshes]
    mesh_t = [torch.as_tensor(v[f], device=dev) for v, f in robot.meshes]

    def signed(w, l, objs):
        """(distance, point on the link, direction) of link l at waypoint w to each object."""
        T = torch.einsum("ij,avj->avi", R[w, l], mesh_t[l]) + t[w, l]
        d, p, c = _mesh_distance(T[None].expand(len(objs), -1, -1, -1), obj[objs])
        u = torch.where(d[:, None] > 0, (p - c) / d.clamp(min=1e-300)[:, None], torch.zeros_like(p))
        V = mesh_v[l] @ R[w, l].T + t[w, l]
        for k in torch.nonzero(d == 0)[:, 0].tolist():
            depth, face = (off[objs[k]][None] - V @ n[objs[k]].T).min(1)
            v = int(depth.argmax())
            if depth[v] > 0:
                d[k], p[k], u[k] = -depth[v], V[v], n[objs[k], face[v]]
        return d, p, u

    # lower bounds by bounding spheres of the link's triangles and the objects
    low = torch.empty(W, L, len(oc), dtype=torch.float64, device=dev)
    for w in range(W):
        for l in range(L):
            T = torch.einsum("ij,avj->avi", R[w, l], mesh_t[l]) + t[w, l]
            c = T.mean(1)
            r = (T - c[:, None]).norm(dim=-1).amax(-1)
            low[w, l] = (torch.cdist(c, oc) - r[:, None]).amin(0) - orad
    at = int(low.argmin())
    w, l, o = at // (L * len(oc)), at // len(oc) % L, at % len(oc)
    reach = float(signed(w, l, torch.tensor([o], device=dev))[0][0]) + 30 * TAU
    found = []
    for w in range(W):
        for l in range(L):
            objs = torch.nonzero(low[w, l] <= max(reach, 0.0) + 1e-9)[:, 0]
            for s in range(0, len(objs), 24):
                d, p, u = signed(w, l, objs[s:s + 24])
                found += [(w, l, d[k], p[k], u[k]) for k in torch.nonzero(d < reach)[:, 0].tolist()]
    d = torch.stack([f[2] for f in found])
    m = d.min()
    keep = d < m + 30 * TAU
    e = torch.where(keep, torch.exp(-(d - m) / TAU), torch.zeros_like(d))
    grad = torch.zeros(W, L, dtype=torch.float64, device=dev)
    axes = torch.as_tensor(robot.axes, device=dev)
    for weight, (w, l, _, p, u) in zip(e, found):
        axis = torch.einsum("jab,jb->ja", R[w, :l + 1], axes[:l + 1])
        grad[w, :l + 1] += weight * (_cross(axis, p - t[w, :l + 1]) @ u)
    return {"value": (m - TAU * torch.log(e.sum()))[None], "grad": (grad / e.sum())[None]}


def exact(case, seed):
    """The outputs of `run` in 64 bits.  None where verdicts are whole numbers
    (the collision queries), where no brute-force pass over the triangle pairs
    ends in seconds (clearances and larger soft-min batches), and for inverse
    kinematics, whose result is wherever its iteration stops."""
    dev = DEVICE if torch.cuda.is_available() else "cpu"
    if case["kind"] == "geom" and case["op"] == "distance" and case["queries"] <= 16384 and case["subdiv"] <= 3:
        return _exact_geom(case, _host_inputs(case, seed), dev)
    if case["kind"] == "rays":
        return _exact_rays(case, _host_inputs(case, seed), dev)
    if case["kind"] == "softmin" and case["trajectories"] == 1 and case["waypoints"] <= 32:
        return _exact_softmin(case, _host_inputs(case, seed), dev)
    return None
