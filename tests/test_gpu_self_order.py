"""Self distance evaluates the pairs nearest first; value, pair, closest points
and gradient stay those of the (i, j) order: contacts of several pairs (the
first in order is reported), pairs at exactly equal distances (mirror images of
a symmetric robot), robots without self pairs in reach, cutoffs down to 1e-6, and
batches around the blocks' two warps."""

import os

import numpy as np
import pytest

from klampt_gb300 import scenes as sc

pytestmark = pytest.mark.gpu
NT = os.cpu_count() or 4


def _configs(which, robot, rng):
    n = 401
    q = sc.uniform_configs(robot, n, rng)
    if which == "folded":      # many contacts at once
        return q
    if which == "near_zero":   # few contacts, small distances
        return (q * rng.uniform(0, 0.3, (n, 1))).astype(np.float32)
    # mirror: both arms in mirrored postures, so that pairs tie
    L = robot.num_links
    h = L // 2
    q[:, h:2 * h] = q[:, :h]
    return q


@pytest.mark.parametrize("which,robot", [("folded", "humanoid"), ("near_zero", "humanoid"), ("mirror", "dual"),
                                         ("folded", "arm"), ("near_zero", "arm")])
@pytest.mark.parametrize("cutoff", [1e-6, 0.02, 2.0])
def test_self_distance_order(which, robot, cutoff):
    from klampt_gb300 import build
    build.build()
    from oracle import oracle_py
    oracle_py.build()
    from klampt_gb300.engine import World
    rng = np.random.default_rng(len(which) + len(robot))
    r = {"humanoid": sc.humanoid, "dual": lambda: sc.dual_arm(rings=4, segments=8),
         "arm": lambda: sc.arm(7, rings=4, segments=8)}[robot]()
    env = sc.env_from_objects("far", [sc.box_mesh((9, 9, 9), (0.1, 0.1, 0.1))])
    q = _configs(which, r, rng)
    d_o, p_o, cp_o, g_o = oracle_py.self_distance(oracle_py.Oracle(r, env), q, cutoff=cutoff, nthreads=NT)
    w = World(env, [r])
    for n in (1, 2, 401):
        d, p, cp, g = (x.cpu().numpy() for x in w.self_distance(q[:n], cutoff))
        assert np.array_equal(p, p_o[:n]), np.flatnonzero((p != p_o[:n]).any(1))[:5]
        assert np.array_equal(d, d_o[:n])
        nz = (d > 0) & (p[:, 0] >= 0)
        assert np.array_equal(cp[nz], cp_o[:n][nz]) and (cp[~nz] == 0).all()
        # FP32 gradients of FP64 features, as the other distance tests take them
        assert np.abs(g - g_o[:n]).max() <= 1e-4 * max(np.abs(g_o[:n]).max(), 1e-6) + 1e-7
    w.close()
