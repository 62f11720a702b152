"""Batches around the lines where the engine changes how it splits work: few
edges (their own kernel up to 512), batches with fewer items than warps (dealt
one per warp), and configuration groups of 1, 2 and 4 by the batch size (152
SMs x 2-4 blocks x 8 warps; the sizes below straddle them for every option).
Bit-exact against the FP64 oracle."""

import os

import numpy as np
import pytest

from klampt_gb300 import scenes as sc

pytestmark = pytest.mark.gpu
NT = os.cpu_count() or 4


@pytest.fixture(scope="module")
def scene():
    from klampt_gb300 import build
    build.build()
    from oracle import oracle_py
    oracle_py.build()
    from klampt_gb300.engine import World
    robots = [sc.arm(7, rings=2, segments=8), sc.arm(12, rings=1, segments=6)]
    env = sc.env_from_objects("boxes", sc.random_boxes(25, np.random.default_rng(1)))
    w = World(env, robots)
    yield robots, w, [oracle_py.Oracle(r, env) for r in robots]
    w.close()


@pytest.mark.parametrize("per_sm", [2, 3, 4])
@pytest.mark.parametrize("E,max_steps", [(1, 400), (7, 2), (60, 300), (512, 40), (513, 40), (3000, 3)])
def test_edges(scene, per_sm, E, max_steps):
    robots, w, oracles = scene
    w.set_option("blocks_per_sm", per_sm)
    rng = np.random.default_rng(E)
    qa, qb, n = sc.random_edges(robots[0], E, rng, step=0.02, min_steps=1, max_steps=max_steps)
    fo, _ = oracles[0].check_edges(qa, qb, n, nthreads=NT)
    for _ in range(3):
        assert np.array_equal(w.check_edges(qa, qb, n).cpu().numpy(), fo)
    assert (fo >= 0).any() or E < 10


@pytest.mark.parametrize("per_sm", [2, 3, 4])
@pytest.mark.parametrize("B", [1, 2, 31, 2431, 2433, 4865, 7295, 7297, 9729, 14593, 19457])
def test_configs(scene, per_sm, B):
    robots, w, oracles = scene
    w.set_option("blocks_per_sm", per_sm)
    rng = np.random.default_rng(B)
    for r in (0, 1):
        q = sc.uniform_configs(robots[r], B, rng)
        eo, so, _ = oracles[r].check_configs(q, nthreads=NT)
        e, s = (x.cpu().numpy() for x in w.check_configs(q, robot=r))
        assert np.array_equal(e, eo) and np.array_equal(s, so)
        f = w.is_feasible(q, robot=r).cpu().numpy()
        assert np.array_equal(f.astype(bool), ~(eo | so).astype(bool))
    ids = rng.integers(0, 2, B).astype(np.int32)
    q = np.zeros((B, 12), np.float32)
    eo, so = np.zeros(B, np.uint8), np.zeros(B, np.uint8)
    for r in (0, 1):
        at = np.flatnonzero(ids == r)
        qr = sc.uniform_configs(robots[r], len(at), rng)
        q[at, :robots[r].num_links] = qr
        if len(at):
            eo[at], so[at], _ = oracles[r].check_configs(qr, nthreads=NT)
    e, s = (x.cpu().numpy() for x in w.check_configs_multi(ids, q))
    assert np.array_equal(e, eo) and np.array_equal(s, so)
