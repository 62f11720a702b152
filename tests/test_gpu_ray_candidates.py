"""A ray keeps up to four triangles for the FP64 decision; more than that are
decided on the way.  Coincident surfaces (the same mesh listed many times, faces
that share a plane), rays through shared vertices and edges, rays in a face's
plane and rays that start on a surface fill the list with ties and with
triangles FP32 cannot decide.  The nearest hit and its ties (smaller object,
then triangle) stay the FP64 oracle's, bit for bit."""

import os

import numpy as np
import pytest

from klampt_gb300 import scenes as sc

pytestmark = pytest.mark.gpu
NT = os.cpu_count() or 4


@pytest.mark.parametrize("copies", [1, 4, 5, 23])
@pytest.mark.parametrize("offset", [0.0, 1e-9, 1e-6])
def test_coincident_surfaces(copies, offset):
    from klampt_gb300 import build
    build.build()
    from oracle import oracle_py
    oracle_py.build()
    from klampt_gb300.engine import World
    rng = np.random.default_rng(copies)
    meshes = []
    for k in range(copies):
        meshes.append(sc.box_mesh((offset * k, 0, 0), (0.5, 0.25, 0.25)))
        meshes.append(sc.icosphere_mesh((0, 0, offset * k), 0.7, 1))
        meshes.append(sc.box_mesh((0, 0.5 + offset * k, 0), (0.5, 0.25, 0.25)))
    order = rng.permutation(len(meshes))
    env = sc.env_from_objects("coincident", [meshes[i] for i in order])
    robot = sc.arm(2, rings=1, segments=4)
    V = np.concatenate([m[0] for m in meshes])
    targets = [V[rng.integers(0, len(V), 300)],                                       # vertices
               0.5 * (V[rng.integers(0, len(V), 300)] + V[rng.integers(0, len(V), 300)]),  # some edge midpoints
               rng.uniform(-0.6, 0.6, (600, 3)),
               np.round(rng.uniform(-0.6, 0.6, (300, 3)) * 4) / 4]                    # in the faces' planes
    t = np.concatenate(targets)
    s = np.concatenate([rng.normal(size=(len(t) - 300, 3)) * 2, np.round(rng.normal(size=(300, 3)) * 4) / 4])
    s[::11] = V[rng.integers(0, len(V), len(s[::11]))]                                # starts on the surfaces
    s, d = s.astype(np.float32), (t - s).astype(np.float32)
    oo, to, tt, po = oracle_py.raycast(oracle_py.Oracle(robot, env), s, d, nthreads=NT)
    w = World(env, [robot])
    o, tr, tv, p = (x.cpu().numpy() for x in w.raycast(s, d))
    w.close()
    assert np.array_equal(o, oo) and np.array_equal(tr, to)
    assert np.array_equal(tv, tt) and np.array_equal(p, po)
    assert (oo >= 0).mean() > 0.5
