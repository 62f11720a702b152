"""Soft-min batches whose pairs do not all fit the pair list: which waypoints
are listed and which are done by one warp can depend on the scheduling, so both
ways give the same bits.  The two scenes are shown to be of that kind: every
trajectory alone fits the list (few pairs evaluated), the batch cannot (more
pairs certainly within reach than the list holds, 65,536; or more at one
waypoint than its 128 segments of 128 hold)."""

import os

import numpy as np
import pytest

from klampt_gb300 import scenes as sc

pytestmark = pytest.mark.gpu
FITS = 97 * 127  # a segment is closed with 97 pairs or more


def _scene(n):
    rng = np.random.default_rng(5)
    c = rng.normal(size=(n, 3))
    c = c / np.linalg.norm(c, axis=1, keepdims=True) * rng.uniform(0.1, 0.35, (n, 1)) + [0.6, 0, 0.3]
    robot = sc.arm(4, rings=1, segments=6)
    q = rng.uniform(robot.qmin, robot.qmax, (32, 1, 4)).astype(np.float32)
    return robot, sc.env_from_objects("dense", [sc.box_mesh(x, (0.004,) * 3) for x in c]), c, q


def _certain(robot, oracle, q, centres, reach):
    """Pairs of waypoint q certainly closer than `reach` (link vertex to box centre)."""
    T = oracle.fk(q.astype(np.float64))
    n = 0
    for l, (v, _) in enumerate(robot.meshes):
        w = v @ T[l, :9].reshape(3, 3).T + T[l, 9:]
        n += int((np.linalg.norm(w[:, None] - centres[None], axis=2).min(0) < reach).sum())
    return n


def _run(w, q, tau):
    w.reset_stats()
    L, G = (x.cpu().numpy() for x in w.softmin(q, tau))
    return L, G, w.stats()["dist_pairs"]


@pytest.fixture(scope="module")
def built():
    from klampt_gb300 import build
    build.build()
    from oracle import oracle_py
    oracle_py.build()


def test_list_too_small_for_the_batch(built):
    from klampt_gb300.engine import World
    from oracle.oracle_py import Oracle
    robot, env, centres, q = _scene(2500)
    o, w, tau = Oracle(robot, env), World(env, [robot]), 0.02
    alone = [_run(w, q[k:k + 1], tau) for k in range(len(q))]
    assert max(a[2] for a in alone) <= FITS
    assert sum(_certain(robot, o, q[k, 0], centres, alone[k][0][0] + 30 * tau) for k in range(len(q))) > 65536
    for _ in range(10):
        L, G, _ = _run(w, q, tau)
        assert np.array_equal(L, [a[0][0] for a in alone])
        assert np.array_equal(G, np.concatenate([a[1] for a in alone]))
    w.close()


def test_one_waypoint_too_dense(built):
    from klampt_gb300.engine import World
    from oracle.oracle_py import Oracle
    robot, env, centres, q = _scene(12500)
    o, w, tau = Oracle(robot, env), World(env, [robot]), 0.012
    alone = [_run(w, q[k:k + 1], tau) for k in range(len(q))]
    sure = [_certain(robot, o, q[k, 0], centres, alone[k][0][0] + 30 * tau) for k in range(len(q))]
    dense = int(np.argmax(sure))
    light = [k for k in range(len(q)) if alone[k][2] <= FITS][:4]
    assert sure[dense] > 128 * 128 and len(light) == 4
    for _ in range(5):
        L, G, _ = _run(w, q[light + [dense]], tau)
        for i, k in enumerate(light):
            assert L[i] == alone[k][0][0] and np.array_equal(G[i], alone[k][1][0])
    # against the oracle, with the tolerances of the other soft-min tests
    L_o, G_o = o.softmin(q[[dense]], tau, nthreads=os.cpu_count() or 4)
    assert abs(L[4] - L_o[0]) <= 1e-12 * max(1.0, abs(L_o[0]))
    assert np.abs(G[4] - G_o[0]).max() <= 1e-4 * np.abs(G_o[0]).max() + 1e-7
    w.close()


def test_counters_include_the_bounding_evaluations(built):
    """One link, one object too large for a vertex-pair bound: evaluated for
    the bound, for the minimum and for the sum."""
    from klampt_gb300.engine import World
    rng = np.random.default_rng(1)
    H = sc.terrain_heights(60, 50, 0.04, rng)
    env = sc.env_from_objects("terrain", [sc.heightfield_mesh(60, 50, 0.04, H, (-1.2, -1.0, -1.2))])
    robot = sc.arm(1, rings=2, segments=8)
    w = World(env, [robot])
    L, _, pairs = _run(w, np.zeros((1, 1, 1), np.float32), 0.01)
    w.close()
    assert np.isfinite(L).all() and pairs == 3
