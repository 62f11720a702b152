"""Minimum distance after a first contact: pairs whose deepest vertex cannot
beat the contact already found are skipped.  Values and pairs stay the FP64
oracle's where that decision is tightest: the same box listed several times
(equal depths, ties to the smaller (link, object)), nested boxes, objects not
flagged convex (distance 0 at contact, never negative), and links of a few
vertices (a remainder of one warp pass)."""

import os

import numpy as np
import pytest

from klampt_gb300 import scenes as sc

pytestmark = pytest.mark.gpu
NT = os.cpu_count() or 4


@pytest.mark.parametrize("segments,rings", [(32, 8), (5, 1)])
@pytest.mark.parametrize("convex", ["all", "none", "mixed"])
def test_min_distance_of_overlapping_objects(segments, rings, convex):
    from klampt_gb300 import build
    build.build()
    from oracle import oracle_py
    oracle_py.build()
    from klampt_gb300.engine import World
    rng = np.random.default_rng(segments + len(convex))
    meshes = []
    for c in rng.uniform(-0.6, 0.6, (12, 3)):
        h = rng.uniform(0.05, 0.25, 3)
        meshes += [sc.box_mesh(c, h), sc.box_mesh(c, h), sc.box_mesh(c, h * 0.6), sc.icosphere_mesh(c, h.min(), 1)]
    order = rng.permutation(len(meshes))
    flags = {"all": np.ones(48), "none": np.zeros(48), "mixed": rng.integers(0, 2, 48)}[convex].astype(np.uint8)
    env = sc.env_from_objects("overlapping", [meshes[i] for i in order], convex=flags)
    robot = sc.arm(5, rings=rings, segments=segments)
    q = sc.uniform_configs(robot, 256, rng)
    d_o, p_o, _, g_o = oracle_py.Oracle(robot, env).min_distance(q, 0.3, nthreads=NT)
    w = World(env, [robot])
    d, p, _, g = (x.cpu().numpy() for x in w.distance(q, 0.3))
    w.close()
    assert np.array_equal(p, p_o)
    assert np.array_equal(d, d_o)
    # FP32 gradients of FP64 features: 1e-4 of the largest entry, as the other distance tests take it
    assert np.abs(g - g_o).max() <= 1e-4 * np.abs(g_o).max() + 1e-7
    assert (d_o <= 0).mean() > 0.2
