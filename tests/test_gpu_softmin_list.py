"""The soft-min's pair list: one waypoint, ragged trajectories, more waypoints
than one chunk of the list holds (8,192), objects too large for a vertex-pair
bound (a terrain of more than 4,096 triangles), objects that are never within
reach, and waypoints with more pairs than their share of the list (done by one
warp each, beside others that fit).  Against the FP64 oracle; L is summed in
FP64 on both sides (1e-12 covers the order and exp/log roundings), the
gradient is FP32 (1e-4 of its largest entry, as the other soft-min tests take
it)."""

import os

import numpy as np
import pytest

from klampt_gb300 import scenes as sc

pytestmark = pytest.mark.gpu
NT = os.cpu_count() or 4


def _boxes(rng, n, lo, hi, h_lo, h_hi):
    return sc.random_boxes(n, rng, lo, hi, h_lo, h_hi)


def _scene(name, rng):
    """(robot, environment, trajectories [T, W, L], tau)."""
    if name == "one_waypoint":
        robot = sc.arm(4, rings=4, segments=8)
        return robot, sc.env_from_objects(name, _boxes(rng, 30, -1, 1, 0.02, 0.1)), (1, 1), 0.01
    if name == "ragged":
        robot = sc.arm(6, rings=4, segments=8)
        return robot, sc.env_from_objects(name, _boxes(rng, 30, -1, 1, 0.02, 0.1)), (7, 13), 0.02
    if name == "chunks":
        robot = sc.arm(2, rings=1, segments=4)
        return robot, sc.env_from_objects(name, _boxes(rng, 3, 0.2, 0.6, 0.02, 0.05)), (613, 14), 0.01
    if name == "terrain":
        robot = sc.arm(5, rings=2, segments=8)
        H = sc.terrain_heights(60, 50, 0.04, rng)
        meshes = [sc.heightfield_mesh(60, 50, 0.04, H, (-1.2, -1.0, -1.2))] + _boxes(rng, 8, -1, 1, 0.02, 0.1)
        return robot, sc.env_from_objects(name, meshes, [1] + [0] * 8, [0] + [1] * 8), (5, 6), 0.01
    if name == "far":
        robot = sc.arm(3, rings=1, segments=6)
        meshes = _boxes(rng, 3, 3.0, 4.0, 0.02, 0.1) + _boxes(rng, 4, 40.0, 60.0, 0.02, 0.1)
        return robot, sc.env_from_objects(name, meshes), (3, 4), 0.05
    # overflow: thousands of small boxes around the arm's base
    robot = sc.arm(4, rings=1, segments=6)
    c = rng.normal(size=(6000, 3))
    c = c / np.linalg.norm(c, axis=1, keepdims=True) * rng.uniform(0.5, 0.75, (6000, 1)) + [0, 0, 0.15]
    meshes = [sc.box_mesh(x, (0.004, 0.004, 0.004)) for x in c]
    return robot, sc.env_from_objects(name, meshes), (2, 2), 0.05


@pytest.mark.parametrize("name", ["one_waypoint", "ragged", "chunks", "terrain", "far", "overflow"])
def test_softmin_list_matches_oracle(name):
    from klampt_gb300 import build
    build.build()
    from oracle import oracle_py
    oracle_py.build()
    from klampt_gb300.engine import World
    rng = np.random.default_rng(len(name))
    robot, env, (T, Wn), tau = _scene(name, rng)
    q = rng.uniform(robot.qmin, robot.qmax, (T, Wn, robot.num_links)).astype(np.float32)
    L_o, G_o = oracle_py.Oracle(robot, env).softmin(q, tau, nthreads=NT)
    w = World(env, [robot])
    L, G = (x.cpu().numpy() for x in w.softmin(q, tau))
    L2, G2 = (x.cpu().numpy() for x in w.softmin(q, tau))
    w.close()
    assert np.array_equal(L, L2) and np.array_equal(G, G2)  # no dependence on scheduling
    assert np.abs(L - L_o).max() <= 1e-12 * max(1.0, np.abs(L_o).max())
    for t in range(T):
        assert np.abs(G[t] - G_o[t]).max() <= 1e-4 * np.abs(G_o[t]).max() + 1e-7
