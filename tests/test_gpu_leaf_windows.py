"""Leaf pairs are expanded to one triangle pair per lane in windows of 32.
Dense triangle soups make every leaf pair a job, with leaves of one to four
triangles, windows that start inside a leaf pair, lists of less than a window
and windows of 32 one-pair jobs.  Collision verdicts, distances and closest
triangles stay the FP64 oracle's, bit for bit."""

import os

import numpy as np
import pytest

from klampt_gb300 import scenes as sc

pytestmark = pytest.mark.gpu
NT = os.cpu_count() or 4


@pytest.fixture(scope="module")
def built():
    from klampt_gb300 import build
    build.build()
    from oracle import oracle_py
    oracle_py.build()


def _soup(n, rng):
    c = rng.uniform(-0.05, 0.05, (n, 1, 3))
    V = (c + rng.uniform(-0.04, 0.04, (n, 3, 3))).reshape(-1, 3)
    return V, np.arange(3 * n, dtype=np.int32).reshape(-1, 3)


def _placements(rng, n, spread):
    q = rng.normal(size=(n, 4))
    w, x, y, z = (q / np.linalg.norm(q, axis=1, keepdims=True)).T
    R = np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                  2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                  2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], 1)
    return np.ascontiguousarray(np.concatenate([R, rng.uniform(-spread, spread, (n, 3))], 1))


@pytest.mark.parametrize("na,nb", [(1, 1), (1, 3), (2, 4), (3, 3), (4, 4), (1, 33), (5, 7), (33, 65), (129, 257)])
def test_geometry_pairs(built, na, nb):
    from klampt_gb300.engine import Geometry
    from oracle.oracle_py import GeomPairOracle
    rng = np.random.default_rng(1000 * na + nb)
    A, B = _soup(na, rng), _soup(nb, rng)
    Ta, Tb = _placements(rng, 500, 0.06), _placements(rng, 500, 0.06)
    ga, gb, o = Geometry(*A), Geometry(*B), GeomPairOracle(A, B)
    for tol in (0.0, 0.01):
        assert np.array_equal(ga.collide(gb, Ta, Tb, tol=tol).cpu().numpy(), o.collide(Ta, Tb, tol=tol, nthreads=NT))
    d, _, elem, _ = (x.cpu().numpy() for x in ga.distance(gb, Ta, Tb))
    do, _, eo, _ = o.distance(Ta, Tb, nthreads=NT)
    assert np.array_equal(d, do) and np.array_equal(elem, eo)
    ga.close()
    gb.close()


@pytest.mark.parametrize("tris", [1, 3, 4, 5, 40])
def test_configurations(built, tris):
    from klampt_gb300.engine import World
    from oracle import oracle_py
    rng = np.random.default_rng(tris)
    robot = sc.arm(7, rings=3, segments=9)
    objects = []
    for _ in range(60):
        V, F = _soup(tris, rng)
        objects.append((V * 3 + rng.uniform(-0.8, 0.8, 3), F))
    env = sc.env_from_objects("soups", objects)
    w, o = World(env, [robot]), oracle_py.Oracle(robot, env)
    for B in (40, 6000):
        q = sc.uniform_configs(robot, B, rng)
        eo, so, _ = o.check_configs(q, nthreads=NT)
        e, s = (x.cpu().numpy() for x in w.check_configs(q))
        assert np.array_equal(e, eo) and np.array_equal(s, so)
    w.close()
