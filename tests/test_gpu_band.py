"""The FP64 decision of undecided triangle pairs works on one record per warp
with its operations spread over the lanes.  Verdicts stay the oracle's where
that splits unevenly: chains of 1, 5, 6, 12 and 31 links (the chain is formed
five steps at a time), trees, prismatic and welded joints, self pairs and
environment pairs, with and without margins, for configurations (both verdicts
and feasibility) and edges.  Surfaces that touch exactly (links moved along an
axis by whole steps against boxes on a grid) make most contacts undecided in
FP32."""

import os

import numpy as np
import pytest

from klampt_gb300 import scenes as sc

pytestmark = pytest.mark.gpu
NT = os.cpu_count() or 4


def _robot(kind, margins):
    if kind == "gantry":  # prismatic x, y, z, a weld, a revolute: boxes as links
        T0 = np.tile(np.array([1, 0, 0, 0, 1, 0, 0, 0, 1, 0, 0, 0.0]), (5, 1))
        r = sc.RobotSpec("gantry", np.arange(-1, 4, dtype=np.int32), np.array([1, 1, 1, 2, 0], np.int32), T0,
                         np.array([[1, 0, 0], [0, 1, 0], [0, 0, 1], [0, 0, 1], [0, 0, 1.0]]),
                         np.full(5, -2.0), np.full(5, 2.0),
                         [sc.box_mesh((0, 0, 0.25 * k), (0.125, 0.125, 0.0625)) for k in range(5)])
    elif kind == "humanoid":
        r = sc.humanoid()
    else:
        r = sc.arm(int(kind[3:]), rings=2, segments=6)
    if margins:
        r.margins = np.full(r.num_links, 0.015)
    return r


@pytest.mark.parametrize("kind", ["arm1", "arm5", "arm6", "arm12", "gantry", "humanoid"])
@pytest.mark.parametrize("margins", [False, True])
def test_undecided_pairs_match_oracle(kind, margins):
    from klampt_gb300 import build
    build.build()
    from oracle import oracle_py
    oracle_py.build()
    from klampt_gb300.engine import World
    rng = np.random.default_rng(len(kind) + margins)
    robot = _robot(kind, margins)
    grid = [sc.box_mesh(0.25 * np.array(c), (0.125, 0.125, 0.0625)) for c in rng.integers(-4, 5, (40, 3))]
    env = sc.env_from_objects("grid", grid)
    if margins:
        env.margins = np.full(env.num_objects, 0.01)
    L = robot.num_links
    q = sc.uniform_configs(robot, 400, rng)
    if kind == "gantry":  # whole steps: faces, edges and corners meet exactly
        q[:, :3] = 0.25 * rng.integers(-6, 7, (400, 3))
        q[:, 4] = np.where(rng.random(400) < 0.5, 0.0, q[:, 4])
    else:
        q[::3] = 0.0  # straight chains: links meet the next ones' end caps
    o = oracle_py.Oracle(robot, env)
    w = World(env, [robot])
    eo, so, _ = o.check_configs(q, nthreads=NT)
    e, s = (x.cpu().numpy() for x in w.check_configs(q))
    assert np.array_equal(e, eo) and np.array_equal(s, so)
    limits = ((q >= robot.qmin) & (q <= robot.qmax)).all(1)  # (FP32 values, FP64 limits)
    assert np.array_equal(w.is_feasible(q).cpu().numpy().astype(bool), limits & ~(eo | so).astype(bool))
    qa, qb = q[:200], np.clip(q[200:], robot.qmin.astype(np.float32), robot.qmax.astype(np.float32))
    n = rng.integers(1, 30, 200).astype(np.int32)
    fo, _ = o.check_edges(qa, qb, n, nthreads=NT)
    assert np.array_equal(w.check_edges(qa, qb, n).cpu().numpy(), fo)
    if kind == "gantry":
        assert w.stats()["band_pairs"] > 100
    w.close()
